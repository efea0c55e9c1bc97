"""-m gpu: a step of the sequence-batch engine that fails takes nothing in (csrc/seq_engine.cu).  The failing step asks for more rows of
logits than a device holds, which the allocator refuses; the same sequences then go on, with fewer tokens than the failed step brought,
and give the bits of an engine that never failed."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
VOCAB, WIDTH, HEADS, DIM = 1 << 18, 64, 2, 32


def test_sequences_go_on_after_a_step_that_failed():
    import torch
    from kuiperllama_b200 import sequence as sq
    lib = sq.load_seq_library()
    g = torch.Generator(device="cuda").manual_seed(5)
    mat = lambda n, k: (torch.randn(n, k, device="cuda", generator=g) * k ** -0.5).bfloat16()  # noqa: E731
    embed, head, w_in, w_out, one = mat(VOCAB, WIDTH), mat(VOCAB, WIDTH), mat(3 * HEADS * DIM, WIDTH), mat(WIDTH, HEADS * DIM), torch.ones(WIDTH, device="cuda")
    layer, d, order = (sq.Layer * 1)(), sq.Desc(), (ctypes.c_int32 * 1)(0)
    L, a = layer[0], layer[0].attn
    L.pre_mixer, L.mixer_kind = sq.Norm(one.data_ptr(), None, 1), 1
    a.heads, a.kv_heads, a.dim, a.vdim, a.scale, a.w_in, a.w_out = HEADS, HEADS, DIM, DIM, DIM ** -0.5, w_in.data_ptr(), w_out.data_ptr()
    d.dtype, d.width, d.vocab, d.norm_eps, d.n_layers, d.layers, d.n_runs, d.run_layer = sq.BF16, WIDTH, VOCAB, 1e-5, 1, layer, 1, order
    d.embed, d.final_norm, d.head = embed.data_ptr(), sq.Norm(one.data_ptr(), None, 1), head.data_ptr()
    d.max_tokens, d.max_seqs = 1024, 3
    torch.cuda.synchronize()
    A = lambda v: (ctypes.c_int32 * len(v))(*[int(x) for x in v])  # noqa: E731
    rng = np.random.default_rng(8)
    tokens = lambda n: rng.integers(0, VOCAB, n).astype(np.int32)  # noqa: E731

    def step(handle, seqs, counts, ids, want):
        rows = np.full((len(want), VOCAB) if len(want) < 9 else (0,), np.nan, np.float32)
        return lib.kllm_seq_step(handle, len(seqs), A(seqs), A(counts), A(ids), len(want), A(want),
                                 rows.ctypes.data if len(want) < 9 else None, None), rows

    plan = [([40, 70], tokens(110)), ([1, 1], tokens(2)), ([30, 3], tokens(33)), ([1, 1], tokens(2))]
    out = []
    for fails in (False, True):
        handle = ctypes.c_void_p()
        assert lib.kllm_seq_create(ctypes.byref(d), None, ctypes.byref(handle)) == 0

        def opened(n):
            seqs = [ctypes.c_int32() for _ in range(n)]
            assert all(lib.kllm_seq_open(handle, ctypes.byref(s)) == 0 for s in seqs)
            return [s.value for s in seqs]

        before = opened(3)  # these end: their pages and their rows of the table are used again
        assert step(handle, before, [90, 90, 90], [7] * 270, [])[0] == 0
        assert all(lib.kllm_seq_close(handle, s) == 0 for s in before)
        seqs = opened(2)
        lengths, free = [0, 0], lib.kllm_seq_free_pages(handle)
        for counts, ids in plan:
            if fails:
                rc, _ = step(handle, seqs, [150, 200], [11] * 350, [0] * VOCAB)
                assert rc != 0
                assert [lib.kllm_seq_length(handle, s) for s in seqs] == lengths
                assert lib.kllm_seq_free_pages(handle) == free
            ends = np.cumsum(counts) - 1
            rc, rows = step(handle, seqs, counts, ids, ends.tolist())
            assert rc == 0
            lengths = [n + c for n, c in zip(lengths, counts)]
            assert [lib.kllm_seq_length(handle, s) for s in seqs] == lengths
            free = lib.kllm_seq_free_pages(handle)
            out.append(rows)
        lib.kllm_seq_destroy(handle)
    for good, again in zip(out[:len(plan)], out[len(plan):]):
        assert np.isfinite(good).all() and np.array_equal(good, again)
