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


def test_a_container_job_without_memory_does_not_throw(tmp_path):
    """Frames are built and compressed on pool threads, where an exception
    ends the process: a job that gets no memory is reported instead, for
    headers and for compressed payload frames."""
    out = run(tmp_path, r"""
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include "host.h"
static std::atomic<size_t> limit{SIZE_MAX};
void* operator new[](size_t n, const std::nothrow_t&) noexcept { return n > limit ? nullptr : std::malloc(n); }
void operator delete[](void* p) noexcept { std::free(p); }
void operator delete[](void* p, size_t) noexcept { std::free(p); }
static int once(bool header, bool payload)
{
    using namespace stz;
    const int layers = 3, C = 4;
    const size_t per = 40000;  // words a layer; zeros, so each frame is worth compressing
    std::vector<uint32_t> words(layers * per, 0);
    std::vector<uint64_t> off(layers + 1);
    for (int i = 0; i <= layers; ++i) off[i] = i * per;
    std::vector<uint32_t> sub(layers * C, 0), unpred(layers, 0);
    FileHeader h{};
    h.zstd_level = 3;
    std::vector<StreamParts> parts(5);
    for (auto& p : parts) p.words = words.data(), p.chunk_word_off = off.data(), p.layers = layers, p.chunks_per_layer = 1;
    ThreadPool pool(4);
    HostArena arena;  // empty: every block is its own
    ContainerWriter w(h, parts, pool, arena);
    const uint16_t sym[2] = {1, 2};
    const uint8_t len[2] = {1, 1};
    std::vector<uint8_t> values(header ? 200000 : 8);
    limit = header || payload ? 100000 : SIZE_MAX;
    w.compress_groups(1, [&](size_t, int layer) -> size_t { return layer < 0 || payload ? 0 : SIZE_MAX; }, [](size_t) {},
                      [&](size_t s) {
                          return build_stream_header(parts[s], arena, sym, len, 2, 0, 0, values.size(), values.data(), 1,
                                                     unpred.data(), off.data(), sub.data(), layers, C);
                      });
    limit = SIZE_MAX;
    return w.out_of_memory();
}
int main() { std::printf("%d%d%d\n", once(false, false), once(true, false), once(false, true)); }
""", ["host.cpp"], ["-l:libzstd.so.1"])
    assert out.strip() == "011"


def test_threads_that_wait_for_another_do_not_use_a_core(tmp_path):
    """Seven threads wait 0.4 s for what the eighth waits for: each thing is
    waited for once, is done when wait returns, and the process uses a fraction
    of that time (polling threads would use seven times it)."""
    out = run(tmp_path, r"""
#include <cstdio>
#include <sys/resource.h>
#include "host.h"
int main()
{
    stz::SharedWaits w(2);
    std::atomic<int> calls{0}, early{0};
    std::atomic<bool> done[2] = {{false}, {false}};
    std::vector<std::thread> t;
    for (int k = 0; k < 8; ++k)
        t.emplace_back([&] {
            for (size_t i = 0; i < 2; ++i) {
                w.wait(i, [&] {
                    ++calls;
                    std::this_thread::sleep_for(std::chrono::milliseconds(200));
                    done[i] = true;
                });
                if (!done[i]) ++early;
            }
        });
    for (auto& x : t) x.join();
    rusage r;
    getrusage(RUSAGE_SELF, &r);
    const double cpu = r.ru_utime.tv_sec + r.ru_stime.tv_sec + 1e-6 * (r.ru_utime.tv_usec + r.ru_stime.tv_usec);
    std::printf("%d %d %d\n", (int)calls, (int)early, cpu < 0.2);
}
""")
    assert out.split() == ["2", "0", "1"]
