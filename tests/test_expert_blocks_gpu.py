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
