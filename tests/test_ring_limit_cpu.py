"""The rule by which the mixed form takes its bin ring: the largest radius that the host gives the
kernels (ring_limit) is the last float that the rule itself (ring_ok) accepts, for any sign and
size of its arguments and without a search that could take long; the kernels' FP32 reach is no
less than the rule's.  Host code of the header, compiled as plain C++."""
import os
import subprocess

from conftest import ROOT

SOURCE = r"""
#include "acum_internal.h"
#include <chrono>
#include <cstdio>
using namespace acum;
static float f(unsigned b) { float r; memcpy(&r, &b, 4); return r; }
int main()
{
    const double inf = INFINITY, nan = NAN;
    const double kbs[] = {1e-40, 1e-20, 1e-9, 1.0, 57.3, 3e3, 1e6, 1e20, 1e40, 0.0, -1e-9, -1.0, -3e3, -1e20, inf, -inf, nan};
    const double unit[] = {1e-30, 1e-10, 1.0, 1e10, 1e30}, mach[] = {0.0, 1e-12, 0.1, 0.9, 0.9995, 2.0};
    const double far[] = {-1.0, 0.0, 1e-3, 1.0, 30.0, 1e12, inf, nan};
    const int rings[] = {512, 1024, 2048};
    const auto t = std::chrono::steady_clock::now();
    long n = 0, bad = 0;
    for (double kb : kbs)
        for (double u : unit)
            for (double m : mach)
                for (double o : far)
                    for (int R : rings) {
                        const double a0 = 340.0 * u, vx = m * a0;
                        const float r = ring_limit(vx, 0.0, 0.0, a0, kb, o * u, R);
                        const auto ok = [&](float x) { return ring_ok(x, vx, 0.0, 0.0, a0, kb, o * u, R); };
                        unsigned bits;
                        memcpy(&bits, &r, 4);
                        ++n;
                        if (r < 0.f) {
                            bad += r != -1.f || ok(0.f);
                            continue;
                        }
                        const float next = f(bits + 1);
                        bool fine = ok(r) && !ok(next) && kb > 0.0;
                        const float k = (float)ring_reach_rate(vx, 0.0, 0.0, a0, kb);
                        for (float x : {r, r * 0.5f, r * 1e-3f, 0.f}) {
                            const double want = ring_reach_bins(x, vx, 0.0, 0.0, a0, kb);
                            const float got = ring_reach_float(x, k);
                            fine = fine && got >= want && got <= want + 0.02;
                        }
                        if (!fine) printf("kb %g unit %g mach %g far %g ring %d: %g\n", kb, u, m, o, R, r);
                        bad += !fine;
                    }
    printf("%ld %ld %.3f\n", n, bad, std::chrono::duration<double>(std::chrono::steady_clock::now() - t).count());
    return bad != 0;
}
"""


def test_ring_limit_is_the_last_radius_accepted(tmp_path):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    src, exe = tmp_path / "ring.cpp", tmp_path / "ring"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I" + os.path.join(ROOT, "acum3_periodic_gb300", "csrc"),
                    "-I" + os.path.join(ROOT, "include"), "-I" + os.path.join(cuda, "include"), str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], stdout=subprocess.PIPE, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
    n, bad, seconds = r.stdout.split()[-3:]
    # a few evaluations of the rule each: under a microsecond, where a walk over the floats takes seconds
    assert int(n) > 10000 and float(seconds) < 2.0
