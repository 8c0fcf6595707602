"""The drop-ins' record fields in pairs of floats against the FP64 arithmetic in whose place they
stand, both rounded to float and compared with extended precision: no field is further off, over
magnitudes, and with sums whose terms cancel.  Host code of the header, compiled as plain C++."""
import os
import subprocess

from conftest import ROOT

SOURCE = r"""
#include "acum_internal.h"
#include <cstdio>
#include <random>
using namespace acum;
typedef _Float128 Q;
int main()
{
    std::mt19937_64 g(1);
    const auto u = [&] { return (double)(g() >> 11) * 0x1p-53; };
    const auto pair = [](double v) { return make_float2((float)v, (float)(v - (double)(float)v)); };
    double worst[2] = {0, 0}, sum[2] = {0, 0};
    long n = 0, differ = 0;
    for (int it = 0; it < 2000000; ++it) {
        const double a0 = 300.0 + 60.0 * u(), rho = 0.5 + u();
        const double ia0 = 1.0 / a0, D1 = 1.0 / (4.0 * M_PI * a0), C = D1 * rho * a0;
        float v[3], m[3], d[3];
        const double vs = exp(12 * u() - 4), ps = exp(14 * u()), as = exp(-14 * u());
        for (int c = 0; c < 3; ++c) {
            v[c] = (float)(vs * (u() - 0.5));
            m[c] = (float)(u() - 0.5);
            d[c] = (float)(200 * (u() - 0.5));
        }
        const float P = (float)(ps * (u() - 0.5)), ds = (float)as;
        float Pd = (float)(300 * ps * (u() - 0.5));
        if (it % 4 == 1) {  // the terms of v.n and of Pd n + P nd cancel to their last places
            m[2] = (float)(-((double)v[0] * m[0] + (double)v[1] * m[1]) / v[2]);
            Pd = (float)(-(double)P * d[0] / m[0]);
        }
        if (it % 4 == 2) {  // and to some of their places
            const double e = exp(-16 * u());
            m[2] = (float)(-((double)v[0] * m[0] + (double)v[1] * m[1]) / v[2] * (1 + e));
            Pd = (float)(-(double)P * d[0] / m[0] * (1 + e));
        }
        const float2 D = mul_pair(pair(D1), make_float2(ds, 0.f));
        const auto see = [&](float2 f, double fp64, Q exact) {
            const float got = f.x + f.y, was = (float)fp64;
            const double ulp = ldexp(1.0, ilogb((double)exact) - 23);
            if (exact == 0 || ilogb((double)exact) < -125) return;
            const double e[2] = {(double)fabs((double)((Q)got - exact)) / ulp, fabs((double)((Q)was - exact)) / ulp};
            for (int k = 0; k < 2; ++k) {
                worst[k] = std::max(worst[k], e[k]);
                sum[k] += e[k] * e[k];
            }
            differ += got != was;
            ++n;
        };
        const double vn = fma((double)v[2], (double)m[2], fma((double)v[1], (double)m[1], (double)v[0] * m[0]));
        see(mul_pair(mul_pair(dot3(v, m), make_float2(ds, 0.f)), pair(C)), C * vn * ds,
            (Q)C * ((Q)v[0] * m[0] + (Q)v[1] * m[1] + (Q)v[2] * m[2]) * ds);
        see(mul_pair(pair(ia0), make_float2(v[0], 0.f)), v[0] * ia0, (Q)ia0 * v[0]);
        see(mul_pair(prod2(P, m[0]), D), D1 * ds * ((double)P * m[0]), (Q)D1 * ds * P * m[0]);
        see(mul_pair(dot2(Pd, m[0], P, d[0]), D), D1 * ds * fma((double)Pd, (double)m[0], (double)P * d[0]),
            (Q)D1 * ds * ((Q)Pd * m[0] + (Q)P * d[0]));
    }
    printf("%ld %ld %.9f %.9f %.9f %.9f\n", n, differ, worst[0], worst[1], sqrt(sum[0] / n), sqrt(sum[1] / n));
    return 0;
}
"""


def test_record_fields_in_pairs(tmp_path):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    src, exe = tmp_path / "pairs.cpp", tmp_path / "pairs"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=gnu++17", "-ffp-contract=off",
                    "-I" + os.path.join(ROOT, "acum3_periodic_gb300", "csrc"), "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(cuda, "include"), str(src), "-o", str(exe)], check=True)
    _, _, worst, worst64, rms, rms64 = subprocess.run([str(exe)], check=True, stdout=subprocess.PIPE, text=True,
                                                         timeout=300).stdout.split()
    # half an ulp of the rounding to float and 2^-43 of the field before it
    assert float(worst) < 0.5 + 2.0 ** -19
    assert float(worst) <= float(worst64) + 2.0 ** -19
    # the RMS of the two differ by what 2^-43 of a field turns: 2^-19 of the roundings, a unit each
    assert float(rms) <= float(rms64) * (1.0 + 2.0 ** -19)
