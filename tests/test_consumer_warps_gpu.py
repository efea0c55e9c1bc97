"""-m gpu: KLLM_CONSUMER_WARPS (csrc/megakernel.cu).  fp32 runs teams of four warps: 8 or 12, the same bits, and its own choice for any other
number.  int8 in the toleranced mode runs teams for 8 and 12 and a warp to a task for 6, 14 and 16, all within the mode's tolerance of
the exact one."""
import numpy as np
import pytest

from gpu_util import assert_bit_equal

pytestmark = pytest.mark.gpu
TOL = 1e-4  # of the toleranced mode (test_decoder_gpu.py)


@pytest.mark.parametrize("key,numerics,choices", [("small", "exact", ["6", "8", "12"]), ("small-qwen", "fast", ["8", "12"]),
                                                  ("small-int8", "exact", ["6", "8", "12", "14", "16"]),
                                                  ("small-int8", "fast", ["6", "8", "12", "14", "16"])])
def test_every_number_of_warps(kllm_lib, monkeypatch, key, numerics, choices):
    from kuiperllama_b200 import SHAPES, Decoder, synth_weights
    monkeypatch.setenv("KLLM_ENGINE", "persistent")
    monkeypatch.delenv("KLLM_CONSUMER_WARPS", raising=False)
    shape = SHAPES[key]
    w = synth_weights(shape, "cuda", 31)
    tokens = np.random.default_rng(2).integers(0, shape.vocab_size, 24).tolist()

    def logits(mode):
        dec, out = Decoder(shape, w, numerics=mode), []
        assert dec.engine == "persistent"
        for pos, token in enumerate(tokens):
            dec.step(token, pos)
            out.append(dec.logits().copy())
        dec.close()
        return np.stack(out)

    exact = logits("exact")
    for warps in choices:
        monkeypatch.setenv("KLLM_CONSUMER_WARPS", warps)
        got = logits(numerics)
        if numerics == "exact":
            assert_bit_equal(got, exact, f"{key}, {warps} warps")
        else:
            assert np.abs(got - exact).max() <= TOL
