"""Bounded waits that ran out reach their own engine, decoder or stream (csrc/wait_flag.h).  The host logic is compiled here against a
few stand-ins for CUDA calls; on a GPU, products are captured, also by a process whose first
product this is."""
import subprocess
import sys
import textwrap
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "kuiperllama_b200" / "csrc"

PROGRAM = r"""
#include <cassert>
#include <cstdlib>
#include <thread>
#include <vector>
#include "wait_flag.h"

static int modes = 0, allocated = 0;
static bool refuse = false;
static cudaStreamCaptureMode mode_now = cudaStreamCaptureModeGlobal;
extern "C" {
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  assert(mode_now == cudaStreamCaptureModeRelaxed);  // an allocation in another mode would end a capture
  if (refuse) return cudaErrorMemoryAllocation;
  ++allocated;
  return (*p = std::malloc(n)) ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFreeHost(void* p) { --allocated; std::free(p); return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode* m) { std::swap(*m, mode_now); ++modes; return cudaSuccess; }
}

using namespace kllm;
int main() {
  {  // owners: what one noted is not another's, and is reported once
    WaitFlag a, b;
    assert(a.take() == 0);  // nothing was ever launched
    assert(a.get() && b.get() && a.get() != b.get() && a.get() == a.get());
    *a.get() = 1;
    assert(b.take() == 0 && a.take() == 1 && a.take() == 0);
    assert(mode_now == cudaStreamCaptureModeGlobal && modes == 4);
  }
  assert(allocated == 0);
  refuse = true;
  WaitFlag none;
  assert(none.get() == nullptr && none.take() == 0);
  StreamWaitFlags s;
  assert(s.get(7) == nullptr);
  refuse = false;
  int* first = s.get(7);
  assert(first && s.get(7) == first && s.get(8) != first);
  *first = 1;
  assert(!take_wait_flag(s.get(8)) && take_wait_flag(s.get(7)) && !take_wait_flag(s.get(7)));
  // more streams than flags: the last ones share, and none of them touches an earlier one's
  for (unsigned long long id = 100; id < 100 + StreamWaitFlags::kStreams; ++id) assert(s.get(id));
  assert(s.get(5000) == s.shared() && s.get(7) != s.shared());
  *s.get(5000) = 1;
  assert(s.get(5001) == s.get(5000) && s.get(7) == first);
  assert(!take_wait_flag(s.get(7)) && !take_wait_flag(s.get(100)) && take_wait_flag(s.get(5001)));
  // every raise is taken once by exactly one of several readers
  for (int round = 0; round < 200; ++round) {
    __atomic_store_n(first, 1, __ATOMIC_RELAXED);
    int got[4] = {0, 0, 0, 0};
    std::vector<std::thread> t;
    for (int i = 0; i < 4; ++i) t.emplace_back([&, i] { got[i] = take_wait_flag(s.get(7)); });
    for (auto& x : t) x.join();
    assert(got[0] + got[1] + got[2] + got[3] == 1);
  }
  return 0;
}
"""


def test_owners_and_streams_have_their_own_flags(tmp_path):
    src = tmp_path / "flags.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "flags"
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-pthread", "-I", str(CSRC), "-I", "/usr/local/cuda/include", str(src), "-o", str(exe)])
    subprocess.check_call([str(exe)], timeout=60)


def test_no_flag_of_the_process():
    """Every launch gets its owner's flag."""
    for path in sorted(CSRC.glob("*.cu*")):
        text = path.read_text()
        assert " wait_flag()" not in text and "take_wait_error" not in text, path.name


CAPTURE = textwrap.dedent("""
    import ctypes, torch
    from kuiperllama_b200 import load_library, sequence as sq
    lib = {lib}
    bf16, T = {bf16}, {tokens}
    g = torch.Generator(device="cuda").manual_seed(1)
    a, w = (torch.randn(n, 256, device="cuda", generator=g) for n in (T, 384))
    if bf16: a, w = a.bfloat16(), w.bfloat16()
    out = torch.zeros(T, 384, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    status = lambda: {status}
    if {warm}:
        assert lib.kllm_seq_gemm(sq.F32, p(w), p(w), p(out), 2, 256, 2, None) == 0 if "seq" in "{call}" else \
            lib.kllm_gemm_tf32(p(w), p(w), p(out), 2, 256, 2, None) == 0
        torch.cuda.synchronize()
    graph, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(graph, stream=s):
        st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        rc = {call}
    assert rc == 0, rc
    graph.replay()
    torch.cuda.synchronize()
    ref = a.double() @ w.double().T
    assert ((out.double() - ref).norm() / ref.norm()).item() < 2e-3
    assert status() == 0
""")
SEQ = "lib.kllm_seq_gemm(sq.BF16 if bf16 else sq.F32, p(a), p(w), p(out), T, 256, 384, st)"
TF32 = "lib.kllm_gemm_tf32(p(a), p(w), p(out), T, 256, 384, st)"


@pytest.mark.gpu
@pytest.mark.parametrize("lib,call,bf16,tokens", [("sq.load_seq_library()", SEQ, False, 4), ("sq.load_seq_library()", SEQ, True, 4),
                                                  ("sq.load_seq_library()", SEQ, False, 40), ("sq.load_seq_library()", SEQ, True, 40),
                                                  ("load_library()", TF32, False, 40)])
@pytest.mark.parametrize("warm", [False, True])
def test_products_are_captured(lib, call, bf16, tokens, warm):
    status = "lib.kllm_product_status(st)" if "seq" in lib else "0"
    code = CAPTURE.format(lib=lib, call=call, bf16=bf16, tokens=tokens, status=status, warm=warm)
    subprocess.run([sys.executable, "-c", code], check=True, cwd=ROOT, timeout=180)
