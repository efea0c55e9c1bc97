"""-m gpu: bf16 products of token blocks on persistent CTAs (umma_kernel) in each form of tile (csrc/seq_tiles.h), whose plain results
leave by TMA in blocks of 32 features x 16 tokens where rows allow it, and gated ones from registers: every element against 64 bits, and
call after call the same bits, where tiles, blocks of a tile and the matrix end in different places.

An accumulator is cut off at each of its K / 16 steps, by at most 2^-23 of what it holds, and so are the 16 products within a step:
an element is off by at most 2 * (K / 16) * 2^-23 * sum |a_k w_k|."""
import ctypes

import numpy as np
import pytest
import torch

from gpu_util import ptr, sync
from tile_forms import NARROW, PAIR, WIDE, form

pytestmark = pytest.mark.gpu


def sum_bound(K):
    return 2 * ((K + 15) // 16) * 2.0 ** -23


@pytest.mark.parametrize("T,K,N,tiles", [
    (1200, 2048, 4096, PAIR),   # the last tile's tokens end with one block of a warp's two
    (1201, 2048, 5000, PAIR),   # one token in its last block; an odd number of feature tiles, features that end inside a warp
    (769, 1032, 12800, PAIR),   # one token in the last tile; a K that is no multiple of a block
    (2305, 1024, 4099, PAIR),   # rows of the result that TMA cannot store
    (6001, 2600, 1090, PAIR),   # features of the last pair for one of its CTAs alone
    (2048, 64, 8224, WIDE),     # one block of K
    (1501, 200, 2050, WIDE),    # a K that is no multiple of a block, rows that TMA cannot store
    (900, 72, 4736, WIDE),      # 37 feature tiles: one wave of CTAs, two of pairs
    (769, 128, 2044, NARROW),   # one token in the last tile
    (1025, 200, 1090, NARROW),  # rows that TMA cannot store
])
def test_every_element_of_a_block(kllm_lib, T, K, N, tiles):
    from kuiperllama_b200 import sequence as sq
    assert form(False, T, N, (K + 63) // 64) == tiles
    lib = sq.load_seq_library()
    g = torch.Generator(device="cuda").manual_seed(T + K + N)
    a = torch.randn(T, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    want, bound = a.double() @ w.double().T, (a.double().abs() @ w.double().abs().T) * sum_bound(K)
    first = None
    for _ in range(5):
        out = torch.full((T, N), float("nan"), device="cuda")
        assert lib.kllm_seq_gemm(sq.BF16, ptr(a), ptr(w), ptr(out), T, K, N, torch.cuda.current_stream().cuda_stream) == 0
        sync()
        assert bool(((out.double() - want).abs() <= bound).all())
        assert first is None or torch.equal(out, first)
        first = out


@pytest.mark.parametrize("T,F,tiles", [
    (2037, 1200, PAIR),  # 19 feature tiles, the last one not full: the last pair has work for one CTA alone
    (1530, 1560, PAIR),  # tokens that end inside a block of the last tile
    (900, 1560, WIDE),
    (300, 1560, NARROW),
])
def test_every_element_of_a_gated_block(T, F, tiles):
    """max(gate, 0) * up, handed on through one-hot rows of the second product and the residual.  The inner value rounds to 2^-8 of itself
    at most, the residual to 2^-24 of the row."""
    from kuiperllama_b200 import sequence as sq
    W = 1600  # 25 blocks of K
    assert form(True, T, F, W // 64) == tiles
    g = torch.Generator(device="cuda").manual_seed(T + F)
    embed = torch.randn(T, W, device="cuda", generator=g).bfloat16()
    up = (torch.randn(2 * F, W, device="cuda", generator=g) * W ** -0.5).bfloat16()
    down = torch.zeros(W, F, device="cuda", dtype=torch.bfloat16)
    down[torch.arange(F), torch.arange(F)] = 1.0
    one, w_in = torch.ones(W, device="cuda"), torch.zeros(24, W, device="cuda", dtype=torch.bfloat16)
    w_out, head = torch.zeros(W, 8, device="cuda", dtype=torch.bfloat16), torch.zeros(T, W, device="cuda", dtype=torch.bfloat16)
    layer = (sq.Layer * 1)()
    L = layer[0]
    L.pre_mixer, L.pre_ff = sq.Norm(one.data_ptr(), None, 1), sq.Norm(None, None, 2)
    L.mixer_kind, a = 1, L.attn  # adds nothing
    a.heads, a.kv_heads, a.dim, a.vdim, a.scale, a.w_in, a.w_out = 1, 1, 8, 8, 1.0, w_in.data_ptr(), w_out.data_ptr()
    L.ff_kind, L.dense.ff, L.dense.act, L.dense.up, L.dense.down = 2, F, 3, up.data_ptr(), down.data_ptr()
    d, order = sq.Desc(), (ctypes.c_int32 * 1)(0)
    d.dtype, d.width, d.vocab, d.norm_eps, d.n_layers, d.layers, d.n_runs, d.run_layer = sq.BF16, W, T, 1e-5, 1, layer, 1, order
    d.embed, d.final_norm, d.head, d.max_tokens, d.max_seqs = embed.data_ptr(), sq.Norm(one.data_ptr(), None, 1), head.data_ptr(), T + 64, 1
    torch.cuda.synchronize()
    lib, handle, first = sq.load_seq_library(), ctypes.c_void_p(), None
    lib.kllm_seq_trace_residual.argtypes = [ctypes.c_void_p, ctypes.c_void_p]
    assert lib.kllm_seq_create(ctypes.byref(d), None, ctypes.byref(handle)) == 0
    x = embed.double()
    gate, value = x @ up[:F].double().T, x @ up[F:].double().T
    off_gate, off_value = (x.abs() @ up[:F].double().abs().T) * sum_bound(W), (x.abs() @ up[F:].double().abs().T) * sum_bound(W)
    exact = torch.relu(gate) * value
    bound = 1.001 * (off_gate * value.abs() + (gate.abs() + off_gate) * off_value) + 2.0 ** -8 * exact.abs() + 2.0 ** -23 * (x[:, :F].abs() + exact.abs())
    for _ in range(3):
        seq, rows = ctypes.c_int32(), np.empty((T, W), np.float32)
        assert lib.kllm_seq_open(handle, ctypes.byref(seq)) == 0
        assert lib.kllm_seq_trace_residual(handle, rows.ctypes.data) == 0
        assert lib.kllm_seq_step(handle, 1, (ctypes.c_int32 * 1)(seq.value), (ctypes.c_int32 * 1)(T), (ctypes.c_int32 * T)(*range(T)), 0,
                                 None, None, None) == 0
        assert lib.kllm_seq_close(handle, seq.value) == 0
        got = torch.from_numpy(rows).cuda().double() - x
        assert bool(((got[:, :F] - exact).abs() <= bound).all()) and bool((got[:, F:] == 0).all())
        assert first is None or torch.equal(got, first)
        first = got
    lib.kllm_seq_destroy(handle)
