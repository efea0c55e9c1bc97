"""-m gpu: attention of single-token steps (csrc/seq_attention_mma.cu), with prompts of an earlier step in the cache.  Up to 64 keys a
CTA finishes its rows itself, past that splits of the keys run side by side and another kernel joins them: contexts at the edges of
tiles and splits, sinks, gates and windows, against 64 bits.  The layer and the bounds are those of test_attention_exact_gpu.py."""
import ctypes

import numpy as np
import pytest

from test_attention_exact_gpu import VOCAB, assert_close, softmax_attention

pytestmark = pytest.mark.gpu
SHAPES = [(8, 2, 128, 128, 0, 0, 0), (4, 2, 64, 64, 0, 1, 1), (4, 1, 72, 120, 40, 2, 1)]  # heads, kv, dim, vdim, window, gate, sink


def last_rows(shape, lens):
    """The attention's output rows of the step that brings the last of `lens` tokens, what 64 bits give for them, bounds, embedded rows."""
    import torch
    from kuiperllama_b200 import sequence as sq
    heads, kv, dim, vdim, window, gate, sink = shape
    lib = sq.load_seq_library()
    gates = {0: 0, 1: heads, 2: heads * vdim}[gate]
    cuts = [heads * dim, kv * dim, kv * vdim, gates]
    width, scale = max((sum(cuts) + 7) // 8 * 8, heads * vdim), 3 * dim ** -0.5
    g = torch.Generator(device="cuda").manual_seed(11)
    embed = torch.randn(VOCAB, width, device="cuda", generator=g).bfloat16()
    sinks = torch.randn(heads, device="cuda", generator=g)
    eye = torch.eye(width, device="cuda", dtype=torch.bfloat16)[:sum(cuts)].contiguous()
    w_out = torch.zeros(width, heads * vdim, device="cuda", dtype=torch.bfloat16)
    w_out[torch.arange(heads * vdim), torch.arange(heads * vdim)] = 1
    one, head = torch.ones(width, device="cuda"), torch.zeros(VOCAB, width, device="cuda", dtype=torch.bfloat16)
    layer = (sq.Layer * 1)()
    L, a = layer[0], layer[0].attn
    L.pre_mixer, L.mixer_kind = sq.Norm(None, None, 2), 1
    a.heads, a.kv_heads, a.dim, a.vdim, a.scale, a.gate, a.window = heads, kv, dim, vdim, scale, gate, window
    a.w_in, a.w_out = eye.data_ptr(), w_out.data_ptr()
    if sink:
        a.sink = sinks.data_ptr()
    d, order = sq.Desc(), (ctypes.c_int32 * 1)(0)
    d.dtype, d.width, d.vocab, d.norm_eps, d.n_layers, d.layers, d.n_runs, d.run_layer = sq.BF16, width, VOCAB, 1e-30, 1, layer, 1, order
    d.embed, d.final_norm, d.head = embed.data_ptr(), sq.Norm(one.data_ptr(), None, 1), head.data_ptr()
    d.max_tokens, d.max_seqs = sum(lens) + 64, len(lens)
    torch.cuda.synchronize()
    handle = ctypes.c_void_p()
    assert lib.kllm_seq_create(ctypes.byref(d), None, ctypes.byref(handle)) == 0
    lib.kllm_seq_trace_residual.argtypes = [ctypes.c_void_p, ctypes.c_void_p]
    ids = [np.random.default_rng(n).integers(0, VOCAB, n).astype(np.int32) for n in lens]
    A = lambda v: (ctypes.c_int32 * len(v))(*[int(x) for x in v])  # noqa: E731
    seqs = []
    for _ in lens:
        s = ctypes.c_int32()
        assert lib.kllm_seq_open(handle, ctypes.byref(s)) == 0
        seqs.append(s.value)
    assert lib.kllm_seq_step(handle, len(lens), A(seqs), A([n - 1 for n in lens]), A(np.concatenate([i[:-1] for i in ids])), 0, None, None, None) == 0
    rows = np.empty((len(lens), width), np.float32)
    assert lib.kllm_seq_trace_residual(handle, rows.ctypes.data) == 0
    assert lib.kllm_seq_step(handle, len(lens), A(seqs), A([1] * len(lens)), A([i[-1] for i in ids]), 0, None, None, None) == 0
    lib.kllm_seq_destroy(handle)
    out = []
    for e, i in enumerate(ids):
        x = embed[torch.from_numpy(i).long().cuda()].double()
        q, k, v, z = x[:, :sum(cuts)].split(cuts, 1)
        T = len(i)
        exact, size = softmax_attention(q.reshape(T, heads, dim), k.reshape(T, kv, dim), v.reshape(T, kv, vdim), scale, window,
                                        sink=sinks if sink else None)
        if gate:
            s = torch.sigmoid(z).reshape(T, heads, -1)
            exact, size = exact * s, size * s
        got = torch.from_numpy(rows[e]).cuda().double()[:heads * vdim] - x[-1, :heads * vdim]
        out.append((got.reshape(heads, vdim), exact[-1], size[-1], x[-1:]))
    return out


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("lens", [[2, 32, 33, 64], [2, 32, 33, 65, 97, 128], [3, 64, 129, 161, 192], [2, 97, 192, 193]],
                         ids=["one split", "two", "four of three tiles", "four"])
def test_single_token_steps(shape, lens):
    for got, exact, size, x in last_rows(shape, lens):
        assert_close(got, exact, size, x, 1.01 * 2.0 ** -8)
