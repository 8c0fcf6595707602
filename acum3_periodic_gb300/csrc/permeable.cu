// Permeable-surface preprocessing on the GPU: preprocess_per (preprocess.cu:8-226).
//
//  per_prep_kernel   one block per element; the element's series are read from the
//                    reference's AoS arrays (variables.cu:11-42 field order, nPRham = 4
//                    as main.cu:87 sets it for permeable decks) and written back in place.
//
// The arithmetic is FP64 whatever the storage type, and follows the reference's order of
// operations with no fused multiply-adds (explicit __dmul_rn / __dadd_rn where the
// compiler would contract), so that with double storage the outputs equal the
// reference's FP64 build bit for bit, and with float storage they are those FP64 results
// rounded once.  The reference's FP32 build rounds every intermediate to float instead.
//
// Work per element: five flow series (rho, u, v, w, P) scaled, optionally filtered (two
// passes of a 3-point periodic median and a 13-tap periodic Gaussian, preprocess.cu:
// 113-137) and differentiated (periodic or end-biased central differences, preprocess.cu:
// 150-163); the normal's periodic derivative (166-168); the position scaled, its
// derivative V and V's derivative (172-180).
//
// The FP64 pipe bounds the kernel (about 16 cycles of the SM per warp instruction; with the
// filter about 21 such operations per output of a pass, 236 per element and step in all; 8192
// elements x 1440 steps in float 8.74 -> 5.5 ms; 701 x 361 in double, open and unfiltered, 99 ->
// 40 us).  So only what has to be FP64 runs there: float conversions, the median's comparisons,
// the scalings and the quotients' first products are integer operations, the quotients by 2 dTau
// then one to three (quot), and the Gaussian forms each product once per run (in integers as well
// the Gaussian's products gained nothing more: 6.8 ms with all seven, 5.6 with two, 5.7 with
// none).  All series stand in six FP64 rows of shared memory (48 bytes a step, 192 KB at 4096
// steps), so that each array's rows are read and written whole, once, and the filter's runs of
// several series fill the block's warps.
#include <cmath>

#include "acum_internal.h"
#include "ptx.h"

namespace acum {

namespace {

constexpr int kPerThreads = 256;
constexpr int kPerRows = 6;
// Threads per block and steps per filter run, by the period: short periods have few runs, so
// smaller blocks put more elements on an SM (20000 elements x 100 steps, filtered, float:
// 2.23 ms in blocks of 256, 1.24 in blocks of 64; 3000 x 60 349 -> 198 us); long ones form
// fewer products in longer runs (8192 x 1440 6.60 ms with runs of 17, 6.30 with 23; 20000 x 100
// with runs of 13 1.76, of 9 1.37).  Past the period at which a block still holds two series' long
// runs it filters one at a time either way, and short runs are the shorter ones (2000 elements x
// 3000 steps, float and double, 4.98 and 4.89 ms with runs of 23, 4.27 and 4.18 with 17; 1666 x 3600
// 4.18 and 4.19, 3.97 and 3.98; 1464 x 4096 4.00 and 3.92, 4.02 and 3.95).
constexpr int kSmallT = 160, kMediumT = 512, kShortRun = 17, kLongRun = 23, kLongT = kPerThreads / 2 * kLongRun;

template <typename S>
struct PerPtrs {
    S *X, *N, *V, *U, *PR;
};

// ---- quotients by 2 dTau

// Correctly rounded a / b from y = RN(1/b) with FMA corrections: Markstein's theorem
// (P. Markstein, IBM J. Res. Dev. 34(1), 1990; Cornea-Hasegan, Golliver & Markstein,
// ARITH-14, 1999, Theorem 1): if y = RN(1/b) and q is within 1 ulp of a/b, then
// r = a - b q is exact and RN(q + r y) = RN(a/b).  q = RN(a y) followed by one correction
// is within 1 ulp; the second correction then gives the IEEE quotient, for a/b in the
// normal range.  A zero numerator keeps its sign through the product a y.
__device__ __noinline__ double div_by(double a, double b, double y)
{
    double q = __dmul_rn(a, y);
    double r = __fma_rn(-q, b, a);
    q = __fma_rn(r, y, q);
    r = __fma_rn(-q, b, a);
    q = __fma_rn(r, y, q);
    return a == 0.0 ? __dmul_rn(a, y) : q;
}

// a / b with the reciprocal in two parts (b.y + b.yl = 1/b to 106 bits): a y + RN(a yl),
// rounded once, is within half an ulp and 2^-52 of one (N. Brisebarre, J.-M. Muller & S.
// Raina, IEEE Trans. Comp. 53(8), 2004); with float storage that is the value rounded to
// float.  Double storage adds one of Markstein's corrections, which gives the IEEE quotient;
// where y is within 2^-54 of 1/b, RN(a y) is within 1 ulp by itself and yl is not needed.
// Numerators outside 2^-900 .. 2^900 (or a step outside 2^-100 .. 2^100) take the general
// sequence, zeros stay as they are (b > 0).
enum Quot { kQuotOnce, kQuotIEEE, kQuotNear };

template <Quot Q>
__device__ __forceinline__ double quot(double a, const PerDiv& b)
{
    const unsigned h = (unsigned)__double2hiint(a) & 0x7fffffffu;
    if (h - 0x07b00000u < b.span) {
        const double q = Q == kQuotNear ? mul_d(a, b.y) : __fma_rn(a, b.y, mul_d(a, b.yl));
        return Q == kQuotOnce ? q : __fma_rn(__fma_rn(-q, b.b, a), b.y, q);
    }
    if (b.span != 0 && (h | (unsigned)__double2loint(a)) == 0) return a;
    return div_by(a, b.b, b.y);
}

// d/dtau of the series in row `src` at step t: central differences (mathfunc.cu:132-140),
// periodic, or the end-biased form (mathfunc.cu:142-159: central interior, ends from
// 3 du[1] - 3 du[2] + du[3])
template <Quot Q>
__device__ __forceinline__ double series_deriv(const double* src, int t, int T, const PerDiv& b, bool biased)
{
    if (!biased || (t > 0 && t < T - 1)) {
        const int tm = t == 0 ? T - 1 : t - 1, tp = t == T - 1 ? 0 : t + 1;
        return quot<Q>(src[tp] - src[tm], b);
    }
    const int s = t == 0 ? 1 : -1;
    const int k1 = t + s, k2 = t + 2 * s, k3 = t + 3 * s;
    const double d1 = quot<Q>(src[k1 + 1] - src[k1 - 1], b);
    const double d2 = quot<Q>(src[k2 + 1] - src[k2 - 1], b);
    const double d3 = quot<Q>(src[k3 + 1] - src[k3 - 1], b);
    return __dadd_rn(__dsub_rn(__dmul_rn(3.0, d1), __dmul_rn(3.0, d2)), d3);
}

// ---- the filter

// the reference's 3-point median (mathfunc.cu:208-341): the left or the middle value if it
// lies strictly between the others, else the right one
__device__ __forceinline__ double median3(double l, double m, double r)
{
    const long long kl = order_key(l), km = order_key(m), kr = order_key(r);
    const long long hi = max(max(kl, km), kr), lo = min(min(kl, km), kr);
    return (kl < hi && kl > lo) ? l : ((km < hi && km > lo) ? m : r);
}

// One pass of median and 13-tap Gaussian (mathfunc.cu:375-421) at the kRun steps from t0 on,
// any T >= 6.  The taps are symmetric and bit-identical in pairs (w[k] = w[12 - k]:
// gauss_taps forms both from the same (k - 6)^2), so the product w[k] Q[q] of output t is
// also the product w[12 - k] Q[q] of output t + 2k - 12: sample by sample, the seven distinct
// products are formed once and added to the outputs they belong to (7 + 42 / kRun products
// per output instead of 13), while every output adds its 13 products in the reference's
// order.  The reference starts from +0: that only matters where every product is -0, and is
// put right on the bits.  Thirteen sums and seven products are alive at one time, so the run
// fits in registers; kRun is odd, so that the lanes' windows start in different banks.
template <int kRun>
__device__ __forceinline__ void filter_run(const double* row, int t0, int T, const double* w, double (&out)[kRun])
{
    int q = t0 - 7;
    q += q < 0 ? T : 0;
    q += q < 0 ? T : 0;
    const auto next = [&]() {
        const double v = row[q];
        q = q + 1 == T ? 0 : q + 1;
        return v;
    };
    double x0 = next(), x1 = next();
#pragma unroll
    for (int j = 0; j < kRun + 12; ++j) {  // sample t0 - 6 + j
        const double x2 = next();
        const double v = median3(x0, x1, x2);
        x0 = x1;
        x1 = x2;
        double p[7];
#pragma unroll
        for (int k = 0; k < 7; ++k) p[k] = __dmul_rn(w[k], v);
#pragma unroll
        for (int s = 0; s < kRun; ++s) {
            const int k = j - s;
            if (k == 0) out[s] = p[0];
            else if (k > 0 && k <= 12) out[s] = __dadd_rn(out[s], p[k < 6 ? k : 12 - k]);
        }
    }
#pragma unroll
    for (int s = 0; s < kRun; ++s)
        if (__double_as_longlong(out[s]) == (long long)0x8000000000000000ULL) out[s] = 0.0;
}

// two passes on the five flow rows, in place: as many series at a time as the block's
// threads hold runs of
template <int kRun>
__device__ void filter_rows(double* rows, int T, const double* w)
{
    const int nruns = (T + kRun - 1) / kRun, most = blockDim.x / nruns;
    for (int pass = 0; pass < 2; ++pass)
        for (int v0 = 0; v0 < 5; v0 += most) {
            const int items = min(most, 5 - v0) * nruns;
            const int v = threadIdx.x / nruns, t0 = (threadIdx.x - v * nruns) * kRun;
            double* row = rows + (size_t)(v0 + v) * T;
            double out[kRun];
            if (threadIdx.x < items) filter_run(row, t0, T, w, out);
            __syncthreads();
            if (threadIdx.x < items) {
#pragma unroll
                for (int s = 0; s < kRun; ++s)
                    if (t0 + s < T) row[t0 + s] = out[s];
            }
            __syncthreads();
        }
}

// ---- rows of the AoS arrays

// Two neighbouring values in one access where the address is a multiple of their size (it is,
// unless an array or a surface starts at an odd element), else one by one.  The widths are
// written out, so that none depends on what the compiler knows of the alignment.
struct Two {
    double a, b;
};
__device__ __forceinline__ double load1(const float* p)
{
    float x;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(x) : "l"(p));
    return widen_d(x);
}
__device__ __forceinline__ double load1(const double* p)
{
    double x;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(x) : "l"(p));
    return x;
}
__device__ __forceinline__ Two load2(const float* p)
{
    if ((reinterpret_cast<size_t>(p) & 7) != 0) return {load1(p), load1(p + 1)};
    float x, y;
    asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(x), "=f"(y) : "l"(p));
    return {widen_d(x), widen_d(y)};
}
__device__ __forceinline__ Two load2(const double* p)
{
    if ((reinterpret_cast<size_t>(p) & 15) != 0) return {load1(p), load1(p + 1)};
    Two v;
    asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.a), "=d"(v.b) : "l"(p));
    return v;
}
__device__ __forceinline__ void store1(float* p, double x)
{
    asm volatile("st.global.f32 [%0], %1;" ::"l"(p), "f"(narrow_d(x)) : "memory");
}
__device__ __forceinline__ void store1(double* p, double x)
{
    asm volatile("st.global.f64 [%0], %1;" ::"l"(p), "d"(x) : "memory");
}
__device__ __forceinline__ void store2(float* p, double x, double y)
{
    if ((reinterpret_cast<size_t>(p) & 7) != 0) {
        store1(p, x);
        store1(p + 1, y);
        return;
    }
    asm volatile("st.global.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(narrow_d(x)), "f"(narrow_d(y)) : "memory");
}
__device__ __forceinline__ void store2(double* p, double x, double y)
{
    if ((reinterpret_cast<size_t>(p) & 15) != 0) {
        store1(p, x);
        store1(p + 1, y);
        return;
    }
    asm volatile("st.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(x), "d"(y) : "memory");
}

template <typename S, Quot Q, int R>
__global__ void __launch_bounds__(kPerThreads, R > 0 ? 3 : 5) per_prep_kernel(PerPtrs<S> p, const __grid_constant__ PerArgs a)
{
    extern __shared__ __align__(16) double rows[];  // [kPerRows][T]
    const int T = a.T;
    const PerSurf* tab = a.table ? a.table : a.surf;
    int lo = 0, hi = a.nSurf - 1;  // the last surface that starts at or before the element
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (tab[mid].first <= (int)blockIdx.x) lo = mid;
        else hi = mid - 1;
    }
    const long long at = (long long)((int)blockIdx.x - tab[lo].first) * T;
    S* X = p.X + tab[lo].ptr[0] + at * 4;    // x, y, z, ds
    S* N = p.N + tab[lo].ptr[1] + at * 6;    // n, ndot
    S* V = p.V + tab[lo].ptr[2] + at * 6;    // V, Vdot
    S* U = p.U + tab[lo].ptr[3] + at * 6;    // u, udot
    S* PR = p.PR + tab[lo].ptr[4] + at * 4;  // P, Pdot, rho, rhodot
    const bool biased = a.periodic != 1;
    double *r0 = rows, *r1 = r0 + T, *r2 = r1 + T, *r3 = r2 + T, *r4 = r3 + T, *r5 = r4 + T;

    // flow series: rho, u, v, w, P
    for (int t = threadIdx.x; t < T; t += blockDim.x) {
        const Two uv = load2(U + (size_t)t * 6);
        r0[t] = mul_d(load1(PR + (size_t)t * 4 + 2), a.rhoRef);
        r1[t] = mul_d(uv.a, a.a0);
        r2[t] = mul_d(uv.b, a.a0);
        r3[t] = mul_d(load1(U + (size_t)t * 6 + 2), a.a0);
        // left to right (preprocess.cu:66); the factor 0.5 is exact and stands with rhoRef
        r4[t] = mul_d(mul_d(mul_d(load1(PR + (size_t)t * 4), a.half_rho), a.mref2), a.a02);
    }
    __syncthreads();
    if (R > 0) filter_rows<(R > 0 ? R : 1)>(rows, T, a.gauss);
    for (int t = threadIdx.x; t < T; t += blockDim.x) {
        S *u = U + (size_t)t * 6, *pr = PR + (size_t)t * 4;
        const double d0 = series_deriv<Q>(r0, t, T, a.div, biased);
        const double d1 = series_deriv<Q>(r1, t, T, a.div, biased);
        const double d2 = series_deriv<Q>(r2, t, T, a.div, biased);
        const double d3 = series_deriv<Q>(r3, t, T, a.div, biased);
        const double d4 = series_deriv<Q>(r4, t, T, a.div, biased);
        store2(u, r1[t], r2[t]);
        store2(u + 2, r3[t], d1);
        store2(u + 4, d2, d3);
        store2(pr, r4[t], d4);
        store2(pr + 2, r0[t], d0);
    }
    __syncthreads();
    // position scaled, panel area (preprocess.cu:56: (ds CFDscale) CFDscale), normal as it is
    for (int t = threadIdx.x; t < T; t += blockDim.x) {
        S* x = X + (size_t)t * 4;
        const Two xy = load2(x), zs = load2(x + 2), n01 = load2(N + (size_t)t * 6);
        r3[t] = n01.a;
        r4[t] = n01.b;
        r5[t] = load1(N + (size_t)t * 6 + 2);
        r0[t] = mul_d(xy.a, a.cfd);
        r1[t] = mul_d(xy.b, a.cfd);
        r2[t] = mul_d(zs.a, a.cfd);
        store2(x, r0[t], r1[t]);
        store2(x + 2, r2[t], mul_d(mul_d(zs.b, a.cfd), a.cfd));
    }
    __syncthreads();
    // normal: periodic derivative of the unchanged n (preprocess.cu:166-168)
    for (int t = threadIdx.x; t < T; t += blockDim.x) {
        S* n = N + (size_t)t * 6;
        store1(n + 3, series_deriv<Q>(r3, t, T, a.div, false));
        store2(n + 4, series_deriv<Q>(r4, t, T, a.div, false), series_deriv<Q>(r5, t, T, a.div, false));
    }
    __syncthreads();
    // V = dx/dtau and Vdot = dV/dtau, both periodic (preprocess.cu:172-180)
    for (int t = threadIdx.x; t < T; t += blockDim.x) {
        r3[t] = series_deriv<Q>(r0, t, T, a.div, false);
        r4[t] = series_deriv<Q>(r1, t, T, a.div, false);
        r5[t] = series_deriv<Q>(r2, t, T, a.div, false);
    }
    __syncthreads();
    for (int t = threadIdx.x; t < T; t += blockDim.x) {
        S* v = V + (size_t)t * 6;
        store2(v, r3[t], r4[t]);
        store2(v + 2, r5[t], series_deriv<Q>(r3, t, T, a.div, false));
        store2(v + 4, series_deriv<Q>(r4, t, T, a.div, false), series_deriv<Q>(r5, t, T, a.div, false));
    }
}

template <typename S, Quot Q, int R>
cudaError_t launch_per_t(const PerPtrs<S>& p, const PerArgs& a, int threads, cudaStream_t s)
{
    const size_t smem = (size_t)a.T * kPerRows * sizeof(double);
    if (smem > 48 * 1024) {
        cudaError_t err = cudaFuncSetAttribute(per_prep_kernel<S, Q, R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)smem);
        if (err != cudaSuccess) return err;
    }
    per_prep_kernel<S, Q, R><<<a.E, threads, smem, s>>>(p, a);
    return cudaGetLastError();
}

template <typename S, Quot Q>
cudaError_t launch_per_s(void* X, void* N, void* V, void* U, void* PR, const PerArgs& a, cudaStream_t s)
{
    const PerPtrs<S> p{(S*)X, (S*)N, (S*)V, (S*)U, (S*)PR};
    const int threads = a.T <= kSmallT ? 64 : a.T <= kMediumT ? 128 : kPerThreads;
    if (a.lowpass != 1) return launch_per_t<S, Q, 0>(p, a, threads, s);
    static_assert(kSmallT <= 64 * kShortRun && kMediumT <= 128 * kShortRun && kMaxPerSteps <= kPerThreads * kShortRun,
                  "a series' runs fit in a block");
    return a.T <= kMediumT || a.T > kLongT ? launch_per_t<S, Q, kShortRun>(p, a, threads, s)
                                           : launch_per_t<S, Q, kLongRun>(p, a, threads, s);
}

// The rows of a permeable deck as read_surf leaves them (io.cu:263-293): each 12-column
// row x y z u v w P rho ds nx ny nz goes to Xham (x, y, z, ds), Nham (n), Uham (u) and
// PRham (P at 0, rho at 2); the derivative columns and Vham start at zero and are all
// written by the preprocessing.  One thread per (element, step); FP64 storage.
__global__ void per_rows_kernel(const float* __restrict__ raw, const long long* __restrict__ raw_off,
                                const int* __restrict__ e_surf, const int* __restrict__ e_local,
                                const int* __restrict__ e_count, int E, int T, double* X, double* N, double* V,
                                double* U, double* PR)
{
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)E * T) return;
    const int e = (int)(idx / T), t = (int)(idx % T);
    const int s = e_surf[e];
    const float* r = raw + raw_off[s] + ((size_t)t * e_count[s] + e_local[e]) * 12;
    const size_t k = (size_t)e * T + t;
    double* x = X + k * 4;
    double* n = N + k * 6;
    double* v = V + k * 6;
    double* u = U + k * 6;
    double* pr = PR + k * 4;
    x[0] = r[0]; x[1] = r[1]; x[2] = r[2]; x[3] = r[8];
    u[0] = r[3]; u[1] = r[4]; u[2] = r[5]; u[3] = 0.0; u[4] = 0.0; u[5] = 0.0;
    pr[0] = r[6]; pr[1] = 0.0; pr[2] = r[7]; pr[3] = 0.0;
    n[0] = r[9]; n[1] = r[10]; n[2] = r[11]; n[3] = 0.0; n[4] = 0.0; n[5] = 0.0;
    for (int c = 0; c < 6; ++c) v[c] = 0.0;
}

}  // namespace

cudaError_t launch_per_rows(const float* raw, const long long* raw_off, const int* e_surf, const int* e_local,
                            const int* e_count, int E, int T, double* const d[5], cudaStream_t s)
{
    const long long n = (long long)E * T;
    if (n <= 0) return cudaErrorInvalidValue;
    per_rows_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(raw, raw_off, e_surf, e_local, e_count, E, T, d[0],
                                                               d[1], d[2], d[3], d[4]);
    return cudaGetLastError();
}

PerDiv per_div(double b)
{
    PerDiv d;
    d.b = b;
    d.y = 1.0 / b;
    const double rest = std::fma(-b, d.y, 1.0);  // exact
    d.yl = rest * d.y;
    d.span = b >= 0x1p-100 && b <= 0x1p100 ? 0x78300000u - 0x07b00000u : 0u;
    d.near = std::fabs(rest) < 0x1p-54;
    return d;
}

cudaError_t launch_per_prep(void* X, void* N, void* V, void* U, void* PR, bool is_double, const PerArgs& a,
                            cudaStream_t s)
{
    if (a.E < 1 || a.nSurf < 1 || a.T < 4 || a.T > kMaxPerSteps) return cudaErrorInvalidValue;
    if (!is_double) return launch_per_s<float, kQuotOnce>(X, N, V, U, PR, a, s);
    return a.div.near ? launch_per_s<double, kQuotNear>(X, N, V, U, PR, a, s)
                      : launch_per_s<double, kQuotIEEE>(X, N, V, U, PR, a, s);
}

}  // namespace acum
