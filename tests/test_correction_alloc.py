"""Plan creation's correction factors when host memory runs out while their
threads are started: the call returns the factors or throws bad_alloc (which
the C entry points turn into TC_ERR_ALLOC); it never ends the process.  The
program below replaces operator new, for the library too, by one that fails
once, at each allocation of the call in turn."""
import os
import subprocess

from tomocam_b200 import _lib

PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <new>
#include <vector>

static std::atomic<long> left{-1};  // allocations until the failing one; < 0: none fails
void *operator new(std::size_t n) {
    if (left.load() >= 0 && left.fetch_sub(1) == 0) throw std::bad_alloc();
    void *p = std::malloc(n ? n : 1);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, std::size_t) noexcept { std::free(p); }

namespace tc {
struct EsKernel {
    int w;
    double beta;
};
std::vector<double> es_correction(int nm, int nf, const EsKernel &es);
}  // namespace tc

int main() {
    const tc::EsKernel es{13, 2.30 * 13};
    const int nm = 5815, nf = 11664;  // enough terms for every thread of the pool
    const std::vector<double> ref = tc::es_correction(nm, nf, es);
    int thrown = 0, returned = 0;
    for (long k = 0; k < 200; ++k) {
        left = k;
        try {
            const std::vector<double> c = tc::es_correction(nm, nf, es);
            const bool unused = left.load() >= 0;
            left = -1;
            if (c != ref) return 2;
            ++returned;
            if (unused) {  // fewer than k + 1 allocations: every one has failed once
                std::printf("%d thrown, %d returned\n", thrown, returned);
                return 0;
            }
        } catch (const std::bad_alloc &) {
            left = -1;
            ++thrown;
        }
    }
    return 3;
}
"""


def test_every_failed_allocation_is_reported(tmp_path):
    src, exe = tmp_path / "alloc.cpp", tmp_path / "alloc"
    src.write_text(PROGRAM)
    libdir = os.path.dirname(_lib.LIB_PATH)
    _lib.lib()
    cudart = [ln.split()[-1] for ln in open("/proc/self/maps") if "libcudart.so" in ln]
    assert cudart, "the library is linked to the CUDA runtime"
    r = subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", str(src), "-o", str(exe), "-rdynamic",
                        "-L" + libdir, "-l:" + os.path.basename(_lib.LIB_PATH), cudart[0],
                        "-Wl,--disable-new-dtags,-rpath," + libdir + ":" + os.path.dirname(cudart[0])],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
    assert "thrown" in r.stdout
