"""Prompt attention of the sequence-batch engine, element by element, against softmax attention in 64 bits: prompts long enough for the
tcgen05 kernel (csrc/seq_attention_umma.cu), plain, differential and latent, and the fp32 tiles (csrc/seq_attention_f32.cu).

The layer is built so that nothing else rounds: the mixer reads the embedded row as it is, its input projection hands the row's
coordinates on as queries, keys, values and gates (one-hot weights: exact), and its output projection hands the attention's output on
into the residual stream, which the step copies out.  What is left, per element: bf16 holds 8 bits and rounds the output to
2^-8 of itself, weights enter the sum as two bf16 terms and exponentials by ex2.approx (2^-14 of the sum of weighted magnitudes bounds
both).  In fp32 exponentials and sums stay below 2^-18 of it.  The residual adds 2^-24 of the embedded row.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
VOCAB = 600


def run_layer(dtype_name, width, attn_out, fill, lens, embed):
    """Embedded rows [T, width] and the attention's output rows [T, attn_out] of one step with prompts of `lens` tokens."""
    import torch
    from kuiperllama_b200 import sequence as sq
    lib = sq.load_seq_library()
    td = torch.bfloat16 if dtype_name == "bf16" else torch.float32
    layer = (sq.Layer * 1)()
    L = layer[0]
    L.pre_mixer = sq.Norm(None, None, 2)  # the row as it is
    w_out = torch.zeros(width, attn_out, device="cuda", dtype=td)
    w_out[torch.arange(attn_out), torch.arange(attn_out)] = 1
    kept = fill(L, w_out)
    one, head = torch.ones(width, device="cuda"), torch.zeros(VOCAB, width, device="cuda", dtype=td)
    d, order = sq.Desc(), (ctypes.c_int32 * 1)(0)
    d.dtype, d.width, d.vocab, d.norm_eps = (sq.BF16 if dtype_name == "bf16" else sq.F32), width, VOCAB, 1e-30
    d.n_layers, d.layers, d.n_runs, d.run_layer = 1, layer, 1, order
    d.embed, d.final_norm, d.head = embed.data_ptr(), sq.Norm(one.data_ptr(), None, 1), head.data_ptr()
    d.max_tokens, d.max_seqs = sum(lens) + 64, len(lens)
    torch.cuda.synchronize()
    handle = ctypes.c_void_p()
    assert lib.kllm_seq_create(ctypes.byref(d), None, ctypes.byref(handle)) == 0
    lib.kllm_seq_trace_residual.argtypes = [ctypes.c_void_p, ctypes.c_void_p]
    ids = np.random.default_rng(3).integers(0, VOCAB, sum(lens)).astype(np.int32)
    A = lambda v: (ctypes.c_int32 * len(v))(*[int(x) for x in v])  # noqa: E731
    seqs = []
    for _ in lens:
        s = ctypes.c_int32()
        assert lib.kllm_seq_open(handle, ctypes.byref(s)) == 0
        seqs.append(s.value)
    rows = np.empty((sum(lens), width), np.float32)
    assert lib.kllm_seq_trace_residual(handle, rows.ctypes.data) == 0
    assert lib.kllm_seq_step(handle, len(lens), A(seqs), A(lens), A(ids), 0, None, None, None) == 0
    lib.kllm_seq_destroy(handle)
    del kept
    x = embed[torch.from_numpy(ids).long().cuda()].double()
    return x, torch.from_numpy(rows).cuda().double()[:, :attn_out] - x[:, :attn_out]


def softmax_attention(q, k, v, scale, window=0, keep=0, chunk=0, sink=None, softcap=0.0):
    """q [T, heads, d], k [T, kv, d], v [T, kv, e] of one sequence, in 64 bits: outputs and the sums of weighted magnitudes."""
    import torch
    T, rep = q.shape[0], q.shape[1] // k.shape[1]
    i = torch.arange(T, device="cuda")
    near = i[:, None] >= 0
    if window:
        near = near & (i[:, None] - i[None, :] < window)
    if chunk:
        near = near & (i[:, None] // chunk == i[None, :] // chunk)
    seen = (i[:, None] >= i[None, :]) & (near | (i[None, :] < keep))
    out, size = [], []
    for h in range(q.shape[1]):
        s = q[:, h] @ k[:, h // rep].T * scale
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        s = s.masked_fill(~seen, -torch.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].double().expand(T, 1)], 1)
        p = torch.softmax(s, 1)[:, :T]
        out.append(p @ v[:, h // rep])
        size.append(p @ v[:, h // rep].abs())
    return torch.stack(out, 1), torch.stack(size, 1)


def by_sequence(lens, parts, f):
    import torch
    at, out = 0, []
    for n in lens:
        out.append(f(*[p[at:at + n] for p in parts]))
        at += n
    return [torch.cat(x) for x in zip(*out)]


def assert_close(got, exact, size, x, rounding, spread=2.0 ** -14):
    off = (got - exact).abs()
    bound = rounding * exact.abs() + spread * size + 2.0 ** -22 * x.abs().max()
    assert (off <= bound).all(), f"{(off > bound).float().mean().item():.2e} of the elements, worst {(off / bound).max().item():.2f} of the bound"


# heads, kv_heads, dim, vdim, window, keep_first, chunk, gate, sink, softcap
PLAIN = [(4, 1, 128, 128, 0, 0, 0, 0, 0, 0), (4, 2, 64, 64, 0, 0, 0, 1, 1, 0), (2, 2, 40, 72, 0, 0, 0, 0, 0, 0),
         (8, 2, 64, 128, 130, 0, 0, 2, 0, 0), (4, 4, 128, 8, 100, 3, 0, 0, 0, 20), (4, 1, 72, 120, 0, 0, 200, 0, 1, 0)]


@pytest.mark.parametrize("case", PLAIN, ids=str)
@pytest.mark.parametrize("dtype", ["bf16", "fp32"])
def test_plain_attention(dtype, case):
    import torch
    heads, kv, dim, vdim, window, keep, chunk, gate, sink, softcap = case
    lens = [1300, 385, 1, 641] if dtype == "bf16" else [300, 65, 1, 130]
    gates = {0: 0, 1: heads, 2: heads * vdim}[gate]
    cuts = [heads * dim, kv * dim, kv * vdim, gates]
    width, td = (sum(cuts) + 7) // 8 * 8, torch.bfloat16 if dtype == "bf16" else torch.float32
    width = max(width, heads * vdim)
    g = torch.Generator(device="cuda").manual_seed(7)
    embed = torch.randn(VOCAB, width, device="cuda", generator=g).to(td)
    sinks, eye = torch.randn(heads, device="cuda", generator=g), torch.eye(width, device="cuda", dtype=td)[:sum(cuts)].contiguous()
    scale = 3 * dim ** -0.5

    def fill(L, w_out):
        L.mixer_kind, a = 1, L.attn
        a.heads, a.kv_heads, a.dim, a.vdim, a.scale, a.gate, a.window, a.keep_first, a.chunk, a.softcap = \
            heads, kv, dim, vdim, scale, gate, window, keep, chunk, softcap
        a.w_in, a.w_out = eye.data_ptr(), w_out.data_ptr()
        if sink:
            a.sink = sinks.data_ptr()
        return eye, w_out, sinks

    x, got = run_layer(dtype, width, heads * vdim, fill, lens, embed)
    q, k, v, z = x[:, :sum(cuts)].split(cuts, 1)
    T = x.shape[0]
    exact, size = by_sequence(lens, [q.reshape(T, heads, dim), k.reshape(T, kv, dim), v.reshape(T, kv, vdim)],
                              lambda *p: softmax_attention(*p, scale, window, keep, chunk, sinks if sink else None, softcap))
    if gate:
        s = torch.sigmoid(z).reshape(T, heads, -1)
        exact, size = exact * s, size * s
    assert_close(got.reshape(T, heads, vdim), exact, size, x, *((1.01 * 2.0 ** -8,) if dtype == "bf16" else (2.0 ** -20, 2.0 ** -18)))


@pytest.mark.parametrize("heads,kv,dim,vdim", [(2, 2, 64, 128), (4, 1, 64, 64)])
def test_differential_attention(heads, kv, dim, vdim):
    """Partial results of both maps, joined by a kernel that norms each head: its division by the root mean square hands every element's
    error on to the head, so bounds are taken of the largest in the head."""
    import torch
    lens, lam, gain, scale = [1300, 700], 0.3, 0.8, 3 * dim ** -0.5
    cuts = [2 * heads * dim, 2 * kv * dim, kv * vdim]
    width = max(sum(cuts), heads * vdim)
    g = torch.Generator(device="cuda").manual_seed(8)
    embed = torch.randn(VOCAB, width, device="cuda", generator=g).bfloat16()
    eye = torch.eye(width, device="cuda", dtype=torch.bfloat16)[:sum(cuts)].contiguous()

    def fill(L, w_out):
        L.mixer_kind, a = 1, L.attn
        a.heads, a.kv_heads, a.dim, a.vdim, a.scale, a.differential, a.diff_lambda, a.diff_out_scale = \
            heads, kv, dim, vdim, scale, 1, lam, gain
        a.w_in, a.w_out = eye.data_ptr(), w_out.data_ptr()
        return eye, w_out

    x, got = run_layer("bf16", width, heads * vdim, fill, lens, embed)
    q, k, v = x[:, :sum(cuts)].split(cuts, 1)
    T = x.shape[0]
    q, k, v = q.reshape(T, heads, 2, dim), k.reshape(T, kv, 2, dim), v.reshape(T, kv, vdim)
    o, size = 0.0, 0.0
    for m, sign in ((0, 1.0), (1, -lam)):
        y, s = by_sequence(lens, [q[:, :, m], k[:, :, m], v], lambda *p: softmax_attention(*p, scale))
        o, size = o + sign * y, size + abs(sign) * s
    rms = (o * o).mean(-1, keepdim=True).sqrt()
    exact = o / rms * gain
    assert_close(got.reshape(T, heads, vdim), exact, 2 * (size / rms * gain).amax(-1, keepdim=True).expand_as(exact), x, 1.01 * 2.0 ** -8)


@pytest.mark.parametrize("heads,dim,rot,vdim,window,sink", [(4, 64, 32, 64, 0, False), (2, 96, 32, 128, 300, True), (2, 40, 0, 72, 0, False)])
def test_fresh_latent_prompts(heads, dim, rot, vdim, window, sink):
    """Prompts that start their sequences: keys and values are the step's own rows, without a page table.  Latents are +-1, so their norm is
    1, and the matrices that expand them hold multiples of 1/16: keys and values are exact sums, rounded to bf16 once."""
    import torch
    lens, rank, scale = [1300, 385, 1, 129], 64, (dim + rot) ** -0.5
    cuts = [heads * (dim + rot), rank, rot]
    width = max((sum(cuts) + 7) // 8 * 8, heads * vdim)
    g = torch.Generator(device="cuda").manual_seed(9)
    embed = torch.randn(VOCAB, width, device="cuda", generator=g)
    embed[:, cuts[0]:cuts[0] + rank] = torch.randint(0, 2, (VOCAB, rank), device="cuda", generator=g).float() * 2 - 1
    embed = embed.bfloat16()
    eye = torch.eye(width, device="cuda", dtype=torch.bfloat16)[:sum(cuts)].contiguous()
    expand = (torch.randint(-8, 9, (heads * (dim + vdim), rank), device="cuda", generator=g).float() / 16).bfloat16()
    ones, sinks = torch.ones(rank, device="cuda"), torch.randn(heads, device="cuda", generator=g)

    def fill(L, w_out):
        L.mixer_kind, a = 2, L.latent
        a.heads, a.dim, a.rot_dim, a.vdim, a.q_rank, a.kv_rank, a.scale, a.window = heads, dim, rot, vdim, 0, rank, scale, window
        a.w_in, a.kv_norm_w, a.w_out = eye.data_ptr(), ones.data_ptr(), w_out.data_ptr()
        a.w_uk, a.w_uv = expand.data_ptr(), expand[heads * dim:].data_ptr()
        if sink:
            a.sink = sinks.data_ptr()
        return eye, expand, ones, w_out, sinks

    x, got = run_layer("bf16", width, heads * vdim, fill, lens, embed)
    T = x.shape[0]
    q, c, r = x[:, :sum(cuts)].split(cuts, 1)
    kv = (c @ expand.double().T).bfloat16().double()
    k = torch.cat([kv[:, :heads * dim].reshape(T, heads, dim), r[:, None].expand(T, heads, rot)], -1)
    exact, size = by_sequence(lens, [q.reshape(T, heads, dim + rot), k, kv[:, heads * dim:].reshape(T, heads, vdim)],
                              lambda *p: softmax_attention(*p, scale, window, sink=sinks if sink else None))
    assert_close(got.reshape(T, heads, vdim), exact, size, x, 1.01 * 2.0 ** -8)
