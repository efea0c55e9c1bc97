"""Blocks of tokens through routed experts: the router over rows of a block, the pair list's tiles of up to 256 rows and the grouped
tensor-core products, against the same tokens in portions, which take the per-token router and other tilings.

Tolerances: fp32 portions differ in the order of sums only (1e-4 of the largest logit); in bf16 rows round at 2^-9 behind other sums,
and a token whose experts score alike may change them: the median row is compared at 2e-2.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def logits(eng, portions):
    """Logits of every token of one sequence brought in `portions`."""
    lib, V = eng.lib, eng.shape.vocab
    seq, out = eng.open(), []
    for ids in portions:
        n = len(ids)
        buf = np.empty((n, V), np.float32)
        arr = ctypes.c_int32 * n
        rc = lib.kllm_seq_step(eng.handle, 1, (ctypes.c_int32 * 1)(seq), (ctypes.c_int32 * 1)(n), arr(*ids), n, arr(*range(n)),
                               buf.ctypes.data_as(ctypes.c_void_p), None)
        assert rc == 0
        out.append(buf)
    eng.close_seq(seq)
    return np.concatenate(out)


def shapes(experts, top):
    from kuiperllama_b200.sequence import FobolornShape, KikunexShape, VurazenShape
    return {
        "softmax": FobolornShape("f", 256, 320, 1, (0, 1, 1), 4, 2, 64, 64, experts, top, 128, 256),
        "sigmoid": KikunexShape("k", 256, 320, (("latent", "moe"),), (0, 1, 1), 4, 32, 16, 32, 64, 64, 64, 4, 32, 32, 128, experts,
                                top, 128, groups=(2, 1) if experts >= 4 else (0, 0)),
        "top": VurazenShape("v", 256, 320, (("lightning", "moe"),), (0, 1, 1), 128, 16, 16, 4, 32, 32, 4, 2, 32, 64, 2, 32, 4, 2, 32, 32,
                            16, 128, experts, top, 128, 128),
    }


@pytest.mark.parametrize("router", ["softmax", "sigmoid", "top"])
@pytest.mark.parametrize("tokens,experts,top", [(256, 8, 2), (300, 8, 3), (700, 2, 1), (513, 40, 2)])
@pytest.mark.parametrize("bf16", [False, True])
def test_block_against_portions(router, tokens, experts, top, bf16):
    from kuiperllama_b200.sequence import BF16, F32, SeqEngine
    eng = SeqEngine(shapes(experts, top)[router], BF16 if bf16 else F32, max_tokens=1024, max_seqs=2, seed=5)
    ids = [int(x) for x in np.random.default_rng(tokens).integers(0, 320, tokens)]
    whole = logits(eng, [ids])
    parts = logits(eng, [ids[i:i + 100] for i in range(0, tokens, 100)])
    eng.close()
    off = np.abs(whole - parts).max(axis=1) / np.abs(parts).max()
    assert np.isfinite(whole).all()
    if bf16:
        assert np.median(off) < 2e-2
    else:
        assert off.max() < 1e-4


@pytest.mark.parametrize("top", [1, 2])
@pytest.mark.parametrize("act,ff", [(0, 72), (0, 200), (1, 136)])
def test_every_row_of_grouped_products(act, ff, top):
    """bf16 experts of 0 to 600 rows against 64 bits, every row: tiles end after 256 rows, at partial boxes of 64 and at widths that are no
    multiple of 16.  Rows of +-1 pass the norm as they are and lie far apart for the router.  The inner activations round to 2^-8 of
    themselves (bf16 holds 8 bits), the sums to far less: an output stays within 1.01 * 2^-8 of its products' magnitudes."""
    import torch
    from kuiperllama_b200 import sequence as sq
    counts = [1, 15, 17, 63, 64, 65, 255, 256, 257, 350, 0, 600]
    E, W, per = len(counts), 256, 5
    g = torch.Generator(device="cuda").manual_seed(ff + top)
    embed = torch.randint(0, 2, (E * per, W), device="cuda", generator=g).float() * 2 - 1
    chosen = [[i % E] if top == 1 else [i % E, (i % E + 1) % E] for i in range(E * per)]
    embed[:, :E] = -1
    for i, es in enumerate(chosen):
        embed[i, es] = 1
    embed = embed.bfloat16()
    gated = act == 0
    r = lambda *d: (torch.randn(*d, device="cuda", generator=g) * d[-1] ** -0.5).bfloat16()  # noqa: E731
    gate_up, down, router = r(E, (2 if gated else 1) * ff, W), r(E, W, ff), torch.zeros(E, W, device="cuda")
    for e in range(E):
        router[e, e] = 8 + e / 8
    one, w_in, w_out = torch.ones(W, device="cuda"), r(24, W), torch.zeros(W, 8, device="cuda", dtype=torch.bfloat16)
    layer = (sq.Layer * 1)()
    L = layer[0]
    L.pre_mixer, L.pre_ff = sq.Norm(one.data_ptr(), None, 1), sq.Norm(one.data_ptr(), None, 1)
    L.mixer_kind, a = 1, L.attn  # adds nothing: its output projection is zero
    a.heads, a.kv_heads, a.dim, a.vdim, a.scale, a.w_in, a.w_out = 1, 1, 8, 8, 1.0, w_in.data_ptr(), w_out.data_ptr()
    L.ff_kind, m = 1, L.moe
    m.experts, m.top, m.ff, m.router_scale, m.act = E, top, ff, 1.0, act
    m.w_router, m.gate_up, m.down = router.data_ptr(), gate_up.data_ptr(), down.data_ptr()
    ids = [e + E * (i % per) for e, n in enumerate(counts) for i in range(n)]
    ids = [ids[i] for i in np.random.default_rng(5).permutation(len(ids))]
    T, d, order = len(ids), sq.Desc(), (ctypes.c_int32 * 1)(0)
    d.dtype, d.width, d.vocab, d.norm_eps, d.n_layers, d.layers, d.n_runs, d.run_layer = sq.BF16, W, E * per, 1e-30, 1, layer, 1, order
    d.embed, d.final_norm, d.head, d.max_tokens, d.max_seqs = embed.data_ptr(), sq.Norm(one.data_ptr(), None, 1), embed.data_ptr(), T + 64, 1
    torch.cuda.synchronize()
    lib, handle, seq = sq.load_seq_library(), ctypes.c_void_p(), ctypes.c_int32()
    lib.kllm_seq_trace_residual.argtypes = [ctypes.c_void_p, ctypes.c_void_p]
    assert lib.kllm_seq_create(ctypes.byref(d), None, ctypes.byref(handle)) == 0
    assert lib.kllm_seq_open(handle, ctypes.byref(seq)) == 0
    rows, one_i = np.empty((T, W), np.float32), ctypes.c_int32 * 1
    assert lib.kllm_seq_trace_residual(handle, rows.ctypes.data) == 0
    assert lib.kllm_seq_step(handle, 1, one_i(seq.value), one_i(T), (ctypes.c_int32 * T)(*ids), 0, None, None, None) == 0
    lib.kllm_seq_destroy(handle)
    x = embed[torch.tensor(ids, device="cuda")].double()
    got = torch.from_numpy(rows).cuda().double() - x
    exact, size = torch.zeros_like(got), torch.zeros_like(got)
    z = x @ router.double().T
    for e in range(E):
        at = torch.tensor([i for i, t in enumerate(ids) if e in chosen[t]], device="cuda", dtype=torch.long)
        if not len(at):
            continue
        pick = torch.tensor([chosen[ids[i]] for i in at.tolist()], device="cuda")
        weight = torch.softmax(z[at[:, None], pick], 1)[pick == e][:, None]
        u = x[at] @ gate_up[e].double().T
        inner = torch.nn.functional.silu(u[:, :ff]) * u[:, ff:] if gated else torch.relu(u) ** 2
        exact[at] += weight * (inner @ down[e].double().T)
        size[at] += weight * (inner.abs() @ down[e].double().abs().T)
    assert ((got - exact).abs() <= 1.01 * 2.0 ** -8 * size + 2.0 ** -20).all()
