"""Gated products of token blocks on persistent CTAs (csrc/seq_gemm_umma.cuh): activations without branches, over their whole range.

One-hot weights hand a row's coordinates on as gate and up values, exactly, and the joined ones back into the residual stream (the clamped form is SwiGLU's sigmoid too).  A result is
rounded to bf16 once (2^-8 of itself with room for the exponential's 2^-21), the residual adds 2^-24 of the row."""
import numpy as np
import pytest

from test_attention_exact_gpu import VOCAB, run_layer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("act,limit,alpha", [(3, 0.0, 0.0), (4, 7.0, 1.7), (5, 0.0, 0.0)])
@pytest.mark.parametrize("lens", [[2100], [1500, 601]])
def test_activations(act, limit, alpha, lens):
    import torch
    ff, width = 510, 1024
    g = torch.Generator(device="cuda").manual_seed(act)
    embed = torch.randn(VOCAB, width, device="cuda", generator=g) * torch.exp2(torch.randint(-12, 8, (VOCAB, width), device="cuda", generator=g).float())
    embed[5, :ff] = torch.linspace(-2000, 2000, ff, device="cuda")
    embed[6, :ff] = torch.linspace(-12, 12, ff, device="cuda")
    embed = embed.bfloat16()
    one = torch.eye(width, device="cuda").bfloat16()
    up, down = one[:2 * ff].contiguous(), torch.zeros(width, ff, device="cuda").bfloat16()
    down[torch.arange(ff), torch.arange(ff)] = 1
    zero, w_in = torch.zeros(width, 128, device="cuda").bfloat16(), torch.zeros(3 * 128, width, device="cuda").bfloat16()

    def fill(L, w_out):
        L.mixer_kind, a = 1, L.attn
        a.heads, a.kv_heads, a.dim, a.vdim, a.scale, a.w_in, a.w_out = 1, 1, 128, 128, 1.0, w_in.data_ptr(), zero.data_ptr()
        from kuiperllama_b200 import sequence as sq
        L.pre_ff = sq.Norm(None, None, 2)  # the row as it is
        L.ff_kind, L.dense.ff, L.dense.act, L.dense.up, L.dense.down = 2, ff, act, up.data_ptr(), down.data_ptr()
        L.dense.act_a, L.dense.act_b = limit, alpha
        return up, down, zero, w_in

    x, got = run_layer("bf16", width, 512, fill, lens, embed)
    z, u = x[:, :ff], x[:, ff:2 * ff]
    if act == 3:
        want = z.clamp(min=0) * u
    elif act == 4:
        z = z.clamp(max=limit)
        want = z * torch.sigmoid(alpha * z) * (u.clamp(-limit, limit) + 1)
    else:
        want = torch.nn.functional.gelu(z, approximate="tanh") * u
    off = (got[:, :ff] - want).abs()
    bound = 1.01 * 2.0 ** -8 * want.abs() + 2.0 ** -23 * x[:, :ff].abs() + 2.0 ** -60 * u.abs()
    if act == 5:  # gelu far below 0: 1 + tanh in 64 bits has lost its digits there
        bound += 2.0 ** -45 * (z * u).abs()
    assert np.isfinite(got.cpu().numpy()).all()
    assert (off <= bound).all(), (off / bound).max().item()
