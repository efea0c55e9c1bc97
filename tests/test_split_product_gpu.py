"""Products of few tokens, K split over a cluster of CTAs (csrc/seq_gemm_split.cuh), against the product in 64 bits.

bf16: the operands are exact, so only the sums differ: a tcgen05 accumulator keeps about 2^-23 of its value per step and is handed
over every 8 steps of 16 elements of K, the rest is summed in fp32 -- an element's error stays below 2^-19 of the sum of the
products' magnitudes.
"""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def call(sq, lib, dtype, a, w, out):
    import torch
    rc = lib.kllm_seq_gemm(dtype, ctypes.c_void_p(a.data_ptr()), ctypes.c_void_p(w.data_ptr()), ctypes.c_void_p(out.data_ptr()),
                           a.shape[0], a.shape[1], w.shape[0], ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    torch.cuda.synchronize()


def product(T, K, N, seed, bf16=True):
    import torch
    from kuiperllama_b200 import sequence as sq
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.randn(T, K, device="cuda", generator=g)
    w = torch.randn(N, K, device="cuda", generator=g)
    if bf16:
        a, w = a.bfloat16(), w.bfloat16()
    out = torch.full((T + 1, N), 7.0, device="cuda")  # the row behind the result has to stay as it is
    call(sq, sq.load_seq_library(), sq.BF16 if bf16 else sq.F32, a, w, out)
    return a.double(), w.double(), out


@pytest.mark.parametrize("T,K,N", [
    (9, 64, 8), (16, 72, 128), (17, 136, 129), (31, 512, 300), (32, 520, 640), (33, 1032, 1000), (40, 4096, 4096),
    (63, 2048, 2047), (64, 640, 96), (65, 1024, 1024), (127, 8192, 513), (200, 296, 2100), (24, 4104, 32000)])
def test_split_product(T, K, N):
    a, w, out = product(T, K, N, T * 7 + K)
    bound = 2.0 ** -19 * (a.abs() @ w.abs().T)
    assert ((out[:T].double() - a @ w.T).abs() <= bound).all()
    assert (out[T] == 7.0).all()


def test_split_product_repeats():
    """The partial tiles are summed in rank order: the same bits every time."""
    import torch
    first = product(40, 4096, 1000, 3)[2]
    for _ in range(3):
        assert torch.equal(product(40, 4096, 1000, 3)[2], first)


@pytest.mark.parametrize("T,K,N", [
    (9, 32, 8), (16, 36, 128), (17, 100, 129), (32, 2048, 300), (33, 1028, 640), (64, 4096, 1000), (65, 288, 96),
    (128, 512, 2047), (129, 1024, 1024), (517, 1024, 513)])
def test_split_product_fp32(T, K, N):
    """fp32 operands as three bf16 parts: left out are products of small parts (2^-24 of the product at most); with the sums' 2^-20 an
    element stays within 2^-18 of the sum of the products' magnitudes."""
    a, w, out = product(T, K, N, T * 5 + K, bf16=False)
    bound = 2.0 ** -18 * (a.abs() @ w.abs().T)
    assert ((out[:T].double() - a @ w.T).abs() <= bound).all()
    assert (out[T] == 7.0).all()


@pytest.mark.parametrize("T", [12, 40, 200])
def test_split_product_fp32_keeps_infinities_and_nans(T):
    """An infinity has no parts: such rows are summed by multiply-adds, so inf stays inf and only inf * 0, inf - inf and NaN
    give NaN; the largest finite value does not become infinite."""
    import torch
    from kuiperllama_b200 import sequence as sq
    g = torch.Generator(device="cuda").manual_seed(T)
    a, w = torch.randn(T, 256, device="cuda", generator=g), torch.randn(300, 256, device="cuda", generator=g)
    a[1, 5], a[3, 200], a[7, 9], w[4, 70], w[250, 5] = float("inf"), -float("inf"), float("nan"), float("inf"), 0.0
    a[5], w[9] = 0.0, 0.0
    a[5, 3], w[9, 3] = torch.finfo(torch.float32).max, 0.5
    out = torch.empty(T, 300, device="cuda")
    call(sq, sq.load_seq_library(), sq.F32, a, w, out)
    ref = (a.double() @ w.double().T).float()
    assert torch.equal(out.isnan(), ref.isnan())
    assert torch.equal(out == float("inf"), ref == float("inf"))
    assert torch.equal(out == -float("inf"), ref == -float("inf"))
    fine = ref.isfinite()
    assert torch.allclose(out[fine], ref[fine], rtol=1e-5, atol=1e-4)


def chain(a, w):
    """The product as a chain of fp32 multiply-adds over K, each rounded once (a product of two fp32 numbers is exact in 64 bits, and
    the sum's second rounding changes nothing at these sizes)."""
    import torch
    acc = torch.zeros(a.shape[0], w.shape[0], device="cuda")
    for k in range(a.shape[1]):
        acc = (acc.double() + a[:, k, None].double() * w[None, :, k].double()).float()
    return acc


@pytest.mark.parametrize("T", [9, 40, 130])
@pytest.mark.parametrize("K", [32, 36, 64, 96, 124, 128, 288, 1024])
def test_fp32_product_is_no_further_off_than_multiply_adds(T, K):
    """(K < 128 is summed by multiply-adds; chain() rounds a few sums in a million the other way.)"""
    import torch
    from kuiperllama_b200 import sequence as sq
    off, off_chain = 0.0, 0.0
    for seed in range(3):
        g = torch.Generator(device="cuda").manual_seed(100 * seed + K)
        a, w = torch.randn(T, K, device="cuda", generator=g), torch.randn(300, K, device="cuda", generator=g)
        out = torch.empty(T, 300, device="cuda")
        call(sq, sq.load_seq_library(), sq.F32, a, w, out)
        exact = a.double() @ w.double().T
        off += (out.double() - exact).norm().item()
        off_chain += (chain(a, w).double() - exact).norm().item()
    assert off <= 1.001 * off_chain


@pytest.mark.parametrize("T,K,N", [(12, 32, 130), (40, 64, 300), (12, 128, 130), (40, 1024, 300), (130, 288, 300)])
def test_fp32_product_keeps_every_bit(T, K, N):
    """One-hot weights hand an operand on as it is; whole numbers of up to 14 bits, whose sums stay below 2^24, are exact."""
    import torch
    from kuiperllama_b200 import sequence as sq
    g = torch.Generator(device="cuda").manual_seed(T + K)
    lib, out, pick = sq.load_seq_library(), torch.empty(T, N, device="cuda"), torch.arange(N, device="cuda")
    a, w = torch.randn(T, K, device="cuda", generator=g), torch.zeros(N, K, device="cuda")
    w[pick, pick % K] = 1.0
    call(sq, lib, sq.F32, a, w, out)
    assert torch.equal(out, a[:, pick % K])
    other = torch.randn(N, K, device="cuda", generator=g)
    call(sq, lib, sq.F32, w[:T].contiguous(), other, out)  # the other side
    assert torch.equal(out, other[:, (pick % K)[:T]].T)
    many = torch.randint(-12291, 12292, (T, K), device="cuda", generator=g).float()
    few = torch.zeros(N, K, device="cuda")
    few[:, 1::8] = torch.randint(-7, 8, (N, few[:, 1::8].shape[1]), device="cuda", generator=g).float()
    call(sq, lib, sq.F32, many, few, out)
    assert torch.equal(out.double(), many.double() @ few.double().T)
    one, other = torch.zeros(T, K, device="cuda"), torch.zeros(N, K, device="cuda")
    one[:, 3], other[:, 3] = 12291.0, 12291.0 - pick  # one product, rounded once
    call(sq, lib, sq.F32, one, other, out)
    assert torch.equal(out, (one.double() @ other.double().T).float())


@pytest.mark.parametrize("scale", [1e-30, 1e-34, 1e-39])
@pytest.mark.parametrize("K", [96, 160, 1024])
def test_fp32_product_of_tiny_operands(scale, K):
    """Numbers below 2^-100, down to those without a leading bit, whose parts would leave bf16's range."""
    import torch
    from kuiperllama_b200 import sequence as sq
    g = torch.Generator(device="cuda").manual_seed(3)
    a, w = torch.randn(20, K, device="cuda", generator=g), 1e20 * torch.randn(200, K, device="cuda", generator=g)
    a[3:9] = (a[3:9].double() * scale).float()
    out = torch.empty(20, 200, device="cuda")
    call(sq, sq.load_seq_library(), sq.F32, a, w, out)
    exact = a.double() @ w.double().T
    assert ((out.double() - exact).norm(dim=1) <= 1e-6 * exact.norm(dim=1)).all()  # multiply-adds: 5.7e-7 at K = 1024


def test_gated_fp32_product_of_tiny_operands():
    """The same in a gated feed-forward, max(gate, 0) * up, whose output the step hands out through one-hot rows and the residual."""
    import numpy as np
    import torch
    from kuiperllama_b200 import sequence as sq
    T, W, F = 20, 160, 200
    g = torch.Generator(device="cuda").manual_seed(4)
    embed = torch.randn(T, W, device="cuda", generator=g)
    embed[3:9] *= 1e-32
    up = 1e15 * torch.randn(2 * F, W, device="cuda", generator=g)
    up[7], up[F + 70] = up[7] * 1e-33, up[F + 70] * 1e-33  # below 2^-100 themselves
    down = torch.zeros(W, F, device="cuda")
    down[torch.arange(W), torch.arange(W)] = 1.0
    one, w_in, w_out = torch.ones(W, device="cuda"), torch.randn(24, W, device="cuda", generator=g), torch.zeros(W, 8, device="cuda")
    head = torch.zeros(T, W, device="cuda")
    layer = (sq.Layer * 1)()
    L = layer[0]
    L.pre_mixer, L.pre_ff = sq.Norm(one.data_ptr(), None, 1), sq.Norm(None, None, 2)
    L.mixer_kind, a = 1, L.attn  # adds nothing
    a.heads, a.kv_heads, a.dim, a.vdim, a.scale, a.w_in, a.w_out = 1, 1, 8, 8, 1.0, w_in.data_ptr(), w_out.data_ptr()
    L.ff_kind, L.dense.ff, L.dense.act, L.dense.up, L.dense.down = 2, F, 3, up.data_ptr(), down.data_ptr()
    d, order = sq.Desc(), (ctypes.c_int32 * 1)(0)
    d.dtype, d.width, d.vocab, d.norm_eps, d.n_layers, d.layers, d.n_runs, d.run_layer = sq.F32, W, T, 1e-5, 1, layer, 1, order
    d.embed, d.final_norm, d.head, d.max_tokens, d.max_seqs = embed.data_ptr(), sq.Norm(one.data_ptr(), None, 1), head.data_ptr(), 64, 1
    torch.cuda.synchronize()
    lib, handle, seq, rows = sq.load_seq_library(), ctypes.c_void_p(), ctypes.c_int32(), np.empty((T, W), np.float32)
    lib.kllm_seq_trace_residual.argtypes = [ctypes.c_void_p, ctypes.c_void_p]
    assert lib.kllm_seq_create(ctypes.byref(d), None, ctypes.byref(handle)) == 0
    assert lib.kllm_seq_open(handle, ctypes.byref(seq)) == 0
    assert lib.kllm_seq_trace_residual(handle, rows.ctypes.data) == 0
    assert lib.kllm_seq_step(handle, 1, (ctypes.c_int32 * 1)(seq.value), (ctypes.c_int32 * 1)(T), (ctypes.c_int32 * T)(*range(T)), 0, None,
                             None, None) == 0
    lib.kllm_seq_destroy(handle)
    x, u = embed.double(), embed.double() @ up.double().T
    exact = x + (torch.relu(u[:, :F]) * u[:, F:])[:, :W]
    got = torch.from_numpy(rows).cuda().double()
    assert ((got - exact).abs() <= 1e-6 * (x.abs() + (embed.double().abs() @ up[:W].double().abs().T) * (embed.double().abs() @ up[F:F + W].double().abs().T))).all()
    assert ((got - exact).norm(dim=1) <= 1e-6 * exact.norm(dim=1)).all()


@pytest.mark.parametrize("T", [9, 40, 63])
@pytest.mark.parametrize("K", [64, 72, 128, 256, 376, 384, 512, 1024])
def test_bf16_product_of_few_rows_is_no_further_off_than_multiply_adds(T, K):
    import torch
    from kuiperllama_b200 import sequence as sq
    off, off_chain = 0.0, 0.0
    for seed in range(3):
        g = torch.Generator(device="cuda").manual_seed(100 * seed + K)
        a, w = torch.randn(T, K, device="cuda", generator=g).bfloat16(), torch.randn(300, K, device="cuda", generator=g).bfloat16()
        out = torch.empty(T, 300, device="cuda")
        call(sq, sq.load_seq_library(), sq.BF16, a, w, out)
        exact = a.double() @ w.double().T
        off += (out.double() - exact).norm().item()
        off_chain += (chain(a, w).double() - exact).norm().item()
    assert off <= off_chain


@pytest.mark.parametrize("T,K,N", [(129, 72, 18945), (300, 64, 8193), (1501, 520, 2050), (2048, 2048, 2561), (4000, 136, 640),
                                   (129, 520, 4737), (140, 1024, 4736), (1900, 2048, 520)])  # around half a tile per SM
def test_persistent_product(T, K, N):
    """Token blocks with a tile of 128 tokens per SM: persistent CTAs with tiles of 256 or 128 tokens, one accumulation over K (K / 16
    steps of about 2^-24 each: within 2^-19 of the products' magnitudes up to K = 2048)."""
    a, w, out = product(T, K, N, T + K)
    bound = 2.0 ** -19 * (a.abs() @ w.abs().T)
    assert ((out[:T].double() - a @ w.T).abs() <= bound).all()
    assert (out[T] == 7.0).all()


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("tokens", [2500, 2432])
def test_gated_block_against_portions(bf16, tokens):
    """A gated feed-forward on a block that fills the chip against the same tokens in portions of 100, which take split tiles.  fp32:
    other orders of sums only; bf16: rows round at 2^-9 behind other sums."""
    import ctypes as ct

    import numpy as np
    from kuiperllama_b200.sequence import BF16, F32, BifazenShape, SeqEngine
    shape = BifazenShape("b", 256, 300, (("attention", 1000),), 4, 4, 32, 16, 32, 64, 64, 4, 2, 32, 32, 96)
    eng = SeqEngine(shape, BF16 if bf16 else F32, max_tokens=4096, max_seqs=2, seed=3)
    ids = [int(x) for x in np.random.default_rng(tokens).integers(0, 300, tokens)]

    def run(portions):
        seq, rows = eng.open(), []
        for p in portions:
            n, buf = len(p), np.empty((len(p), 300), np.float32)
            arr = ct.c_int32 * n
            assert eng.lib.kllm_seq_step(eng.handle, 1, (ct.c_int32 * 1)(seq), (ct.c_int32 * 1)(n), arr(*p), n, arr(*range(n)),
                                         buf.ctypes.data_as(ct.c_void_p), None) == 0
            rows.append(buf)
        eng.close_seq(seq)
        return np.concatenate(rows)

    whole, parts = run([ids]), run([ids[i:i + 100] for i in range(0, tokens, 100)])
    eng.close()
    off = np.abs(whole - parts).max(axis=1) / np.abs(parts).max()
    assert off.max() < (4e-2 if bf16 else 1e-4)


def test_prefill_block_that_fills_the_chip():
    """460 tokens of a TinyLlama-wide model: the gated TF32 product runs on persistent CTAs; logits as close to the exact prompt path as
    tests/test_prefill_gpu.py asks of shorter prompts."""
    import numpy as np
    from dataclasses import replace
    from kuiperllama_b200 import SHAPES, Decoder, synth_weights
    shape = replace(SHAPES["tinyllama-1.1b"], layer_num=2)
    dec = Decoder(shape, synth_weights(shape, "cuda", 5))
    toks = [1] + [int(t) for t in np.random.default_rng(1).integers(2, 32000, 459)]
    dec.prompt(toks)
    exact = dec.logits()
    dec.prefill_tf32(toks)
    assert np.abs(dec.logits() - exact).max() <= 2e-2 * np.abs(exact).max()
    dec.close()
