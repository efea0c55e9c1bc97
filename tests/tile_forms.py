"""csrc/seq_tiles.h, compiled as it stands for the tests."""
import ctypes
import functools
import subprocess
import tempfile
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "kuiperllama_b200" / "csrc"
NARROW, WIDE, PAIR = range(3)


@functools.cache
def _lib():
    with tempfile.TemporaryDirectory() as td:
        src, so = Path(td) / "rule.cpp", Path(td) / "rule.so"
        src.write_text('#include "seq_tiles.h"\nusing namespace kllm::seq::umma;\nextern "C" int form(int g, int t, int n, int k)'
                       "{ return tile_form(g, t, n, k); }\nextern \"C\" void waves(int g, int t, int n, int* w)"
                       "{ const TileWaves x = tile_waves(g, t, n); w[0] = x.narrow, w[1] = x.wide, w[2] = x.pair; }\n")
        subprocess.check_call(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-I", str(CSRC), str(src), "-o", str(so)])
        return ctypes.CDLL(str(so))


def form(gated, tokens, features, blocks):
    return _lib().form(int(gated), tokens, features, blocks)


def waves(gated, tokens, features):
    w = (ctypes.c_int * 3)()
    _lib().waves(int(gated), tokens, features, w)
    return tuple(w)
