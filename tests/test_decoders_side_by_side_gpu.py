"""-m gpu: decoders of several shapes in one process share the decode kernel; one that is created later and needs less shared memory takes
none away from an earlier one (csrc/megakernel.cu, allow_shared_memory)."""
import pytest

from gpu_util import assert_bit_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("larger,smaller,numerics", [("small", "small-qwen", "exact"), ("small-tp-int8", "small-int8", "fast"),
                                                     ("small-tp-int8", "small-int8", "exact")])
def test_an_earlier_decoder_runs_after_a_smaller_one(kllm_lib, monkeypatch, larger, smaller, numerics):
    from kuiperllama_b200 import SHAPES, Decoder, synth_weights
    monkeypatch.setenv("KLLM_ENGINE", "persistent")
    first = Decoder(SHAPES[larger], synth_weights(SHAPES[larger], "cuda", 3), numerics=numerics)
    first.generate(1, 0, 8)
    alone = first.logits().copy()
    second = Decoder(SHAPES[smaller], synth_weights(SHAPES[smaller], "cuda", 4), numerics=numerics)
    assert first.engine == second.engine == "persistent"
    second.generate(1, 0, 8)
    first.generate(1, 0, 8)
    assert_bit_equal(first.logits(), alone, f"{larger} beside {smaller}")
    first.close(), second.close()
