"""Long bf16 prompts on the tcgen05 attention (csrc/seq_attention_umma.cu) against the same prompts in steps of at most 300 tokens, which
take the mma.sync attention.

Both score in fp32 and weigh values with two bf16 terms; outputs are rounded to bf16 and pass one output projection, so logits differ by
a few bf16 roundings: 2e-2 of the largest at most, 4e-3 in the median row.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = r'''
import ctypes, sys
import numpy as np, torch
from kuiperllama_b200 import sequence as sq
lib = sq.load_seq_library()
heads, kv, dim, vdim, window, keep, chunk, gate, sink, softcap, portion = [float(x) for x in sys.argv[1].split(",")]
heads, kv, dim, vdim, window, keep, chunk, gate, sink, portion = (int(x) for x in (heads, kv, dim, vdim, window, keep, chunk, gate, sink, portion))
W, V, lens = 256, 200, [1300, 385, 1, 513]
g = torch.Generator(device="cuda").manual_seed(1)
r = lambda *d, s=1.0, t=torch.bfloat16: (torch.randn(*d, device="cuda", generator=g) * s).to(t).contiguous()
gates = {0: 0, 1: heads, 2: heads * vdim}[gate]
w_in, w_out = r(heads * dim + kv * (dim + vdim) + gates, W, s=W ** -0.5), r(W, heads * vdim, s=(heads * vdim) ** -0.5)
emb, head, fin, one, sk = r(V, W), r(V, W, s=W ** -0.5), torch.ones(W, device="cuda"), torch.ones(W, device="cuda"), r(heads, t=torch.float32)
L = (sq.Layer * 1)()
L[0].pre_mixer, L[0].mixer_kind, a = sq.Norm(one.data_ptr(), None, 1), 1, L[0].attn
a.heads, a.kv_heads, a.dim, a.vdim, a.scale, a.gate, a.window, a.keep_first, a.chunk, a.softcap = heads, kv, dim, vdim, 3 * dim ** -0.5, gate, window, keep, chunk, softcap
a.w_in, a.w_out = w_in.data_ptr(), w_out.data_ptr()
if sink: a.sink = sk.data_ptr()
d = sq.Desc()
order = (ctypes.c_int32 * 1)(0)
d.dtype, d.width, d.vocab, d.norm_eps, d.n_layers, d.layers, d.n_runs, d.run_layer = sq.BF16, W, V, 1e-5, 1, L, 1, order
d.embed, d.final_norm, d.head, d.max_tokens, d.max_seqs = emb.data_ptr(), sq.Norm(fin.data_ptr(), None, 1), head.data_ptr(), 8192, 8
torch.cuda.synchronize()
h = ctypes.c_void_p()
assert lib.kllm_seq_create(ctypes.byref(d), None, ctypes.byref(h)) == 0
rng = np.random.default_rng(2)
ids = [rng.integers(0, V, n).tolist() for n in lens]
A = lambda v: (ctypes.c_int32 * len(v))(*v)
def run(cuts):
    seqs, rows = [], [[] for _ in lens]
    for _ in lens:
        s = ctypes.c_int32(); assert lib.kllm_seq_open(h, ctypes.byref(s)) == 0; seqs.append(s.value)
    for lo, hi in zip(cuts, cuts[1:]):
        use = [(k, x[lo:hi]) for k, x in enumerate(ids) if x[lo:hi]]
        flat = [t for _, x in use for t in x]
        n = len(flat)
        buf = np.empty((n, V), np.float32)
        assert lib.kllm_seq_step(h, len(use), A([seqs[k] for k, _ in use]), A([len(x) for _, x in use]), A(flat), n, A(range(n)), buf.ctypes.data_as(ctypes.c_void_p), None) == 0
        at = 0
        for k, x in use:
            rows[k].append(buf[at:at + len(x)]); at += len(x)
    for s in seqs: assert lib.kllm_seq_close(h, s) == 0
    return np.concatenate([np.concatenate(r) for r in rows])
long = run([0, portion, max(lens)] if portion else [0, max(lens)])
short = run(list(range(0, max(lens), 300)) + [max(lens)])
lib.kllm_seq_destroy(h)
np.savez(sys.argv[2], long=long, short=short)
'''


# heads, kv_heads, dim, vdim, window, keep_first, chunk, gate, sink, softcap, first portion (0: whole prompts)
@pytest.mark.parametrize("case", ["4,1,128,128,0,0,0,0,0,0,0", "4,2,64,64,0,0,0,1,1,0,0", "2,2,40,72,0,0,0,0,0,0,0",
                                  "8,2,64,128,130,0,0,2,0,0,0", "4,4,128,8,100,3,0,0,0,20,0", "4,1,72,120,0,0,200,0,1,0,0",
                                  "4,2,128,64,300,5,0,1,0,0,300", "16,2,64,64,0,0,0,0,0,0,129"])
def test_long_prompts_against_short_steps(tmp_path, case):
    import numpy as np
    path = str(tmp_path / "out.npz")
    subprocess.run([sys.executable, "-c", SCRIPT, case, path], check=True, env=dict(os.environ, PYTHONPATH=os.getcwd()), timeout=240)
    got = np.load(path)
    off = np.abs(got["long"] - got["short"]).max(axis=1) / np.abs(got["short"]).max()
    assert np.isfinite(got["long"]).all()
    assert off.max() < 2e-2 and np.median(off) < 4e-3
