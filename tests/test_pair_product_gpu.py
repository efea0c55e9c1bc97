"""-m gpu: bf16 products of token blocks on pairs of CTAs (umma_kernel, tiles of 256 x 256), whose results leave by TMA in blocks of
32 features x 16 tokens: every element against 64 bits, and call after call the same bits, where tiles, blocks of a tile and the
matrix end in different places.

An accumulator is cut off at each of its K / 16 steps, by at most 2^-23 of what it holds, and so are the 16 products within a step:
an element is off by at most 2 * (K / 16) * 2^-23 * sum |a_k w_k|."""
import pytest
import torch

from gpu_util import ptr, sync

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,K,N", [
    (1200, 2048, 2048),  # the last tile's tokens end with one block of a warp's two
    (1201, 512, 3072),   # one token in its last block
    (769, 128, 8192),    # one token in the last tile
    (2048, 64, 8224),    # a block of K, features of the last pair for one of its CTAs alone
    (1025, 200, 4100),   # a K that is no multiple of a block, features that end inside a warp
    (2049, 72, 4099),    # rows of the result that TMA cannot store
])
def test_every_element_of_a_block(kllm_lib, T, K, N):
    from kuiperllama_b200 import sequence as sq
    lib = sq.load_seq_library()
    g = torch.Generator(device="cuda").manual_seed(T + K + N)
    a = torch.randn(T, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    want, bound = a.double() @ w.double().T, (a.double().abs() @ w.double().abs().T) * (2 * (K + 15) // 16 * 2.0 ** -23)
    first = None
    for _ in range(5):
        out = torch.full((T, N), float("nan"), device="cuda")
        assert lib.kllm_seq_gemm(sq.BF16, ptr(a), ptr(w), ptr(out), T, K, N, torch.cuda.current_stream().cuda_stream) == 0
        sync()
        assert bool(((out.double() - want).abs() <= bound).all())
        assert first is None or torch.equal(out, first)
        first = out
