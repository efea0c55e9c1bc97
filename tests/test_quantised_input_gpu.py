"""-m gpu: the quantised input vector of the toleranced int8 mode (quantize_input_inplace, csrc/megakernel.cu) takes a value that is no
number for zero: a w1 row whose scales are NaN leaves a NaN among the 64 values of its group, and the logits are those of a row of zeros."""
import pytest

from gpu_util import assert_bit_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mma", [False, True])
@pytest.mark.parametrize("key", ["small-int8", "small-tp-int8"])
def test_a_value_that_is_no_number_counts_as_zero(kllm_lib, monkeypatch, key, mma):
    import torch
    from kuiperllama_b200 import SHAPES, Decoder, synth_weights
    monkeypatch.setenv("KLLM_ENGINE", "persistent")
    monkeypatch.setenv("KLLM_INT8_MMA", str(int(mma)))
    shape = SHAPES[key]
    rows = (0, 3, 70, shape.hidden_dim - 1)
    logits = []
    for value in (0.0, float("nan")):
        w = synth_weights(shape, "cuda", 31)
        per_row = w["s1"][0].reshape(shape.hidden_dim, -1)
        per_row[list(rows)] = value
        assert torch.equal(w["s1"][0].reshape(shape.hidden_dim, -1).isnan().any(1).nonzero().flatten().cpu(),
                           torch.tensor(rows if value != value else [], dtype=torch.int64))
        dec = Decoder(shape, w, numerics="fast")
        assert dec.engine == "persistent"
        for pos, token in enumerate((1, 5, 9)):
            dec.step(token, pos)
            logits.append(dec.logits().copy())
        dec.close()
    for zero, nan in zip(logits[:3], logits[3:]):
        assert_bit_equal(nan, zero, key)
