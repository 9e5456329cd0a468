"""CPU checks of the runtime's host pieces, compiled from its headers by the
host compiler with the CUDA calls replaced by counting fakes."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "sc25-stz2_b200", "csrc")
CUDA = next((os.path.dirname(os.path.dirname(p)) for p in (shutil.which("nvcc"),) if p), "/usr/local/cuda")

pytestmark = pytest.mark.skipif(not (shutil.which("g++") and os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h"))),
                                reason="no host compiler or CUDA headers")


def run(tmp_path, main, sources=(), libs=()):
    src = tmp_path / "main.cpp"
    src.write_text(main)
    exe = tmp_path / "main"
    cmd = ["g++", "-std=c++17", "-O1", "-I", CSRC, "-I", os.path.join(ROOT, "include"), "-I", os.path.join(CUDA, "include"),
           str(src), *[os.path.join(CSRC, s) for s in sources], "-o", str(exe), *libs, "-lpthread"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
    return r.stdout


def test_an_early_return_waits_for_every_stream(tmp_path):
    """Work queued before a failure reads pinned buffers and descriptors that
    the next call writes: an early return waits for all the call's streams, a
    finished call for none of them again."""
    out = run(tmp_path, r"""
#include "runtime.h"
static std::string seen;
extern "C" cudaError_t cudaStreamSynchronize(cudaStream_t s)
{
    seen += (char)('0' + (int)(size_t)s);
    return cudaErrorUnknown;  // its status is not the caller's error
}
static int call(bool fail, bool thrown)
{
    stz::DrainOnExit drain{(cudaStream_t)1, (cudaStream_t)2, (cudaStream_t)3};
    if (thrown) throw std::bad_alloc();
    if (fail) return 1;
    drain.done = true;
    return 0;
}
int main()
{
    call(true, false);
    seen += '|';
    call(false, false);
    seen += '|';
    try { call(false, true); } catch (const std::bad_alloc&) {}
    seen += '|';
    { stz::DrainOnExit one{(cudaStream_t)4}; }
    std::printf("%s\n", seen.c_str());
}
""")
    assert out.strip() == "123||123|4"
