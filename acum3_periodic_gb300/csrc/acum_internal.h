// acum_internal.h -- declarations shared by the CUDA translation units and the C++ host
// layer of libacum.  Not part of the public ABI (include/acum.h).
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>
#include <algorithm>
#include <string>
#include <vector>

#include "../../include/acum.h"

namespace acum {

// Record layout of one element-step for the tonal kernels.
// FP64 records (the plain form and the adjoints): 5 groups of 4 reals, a lane reads its
// step with 2x128-bit loads per group; the panel weight dsD = D1 ds, D1 = 1/(4 pi a0), is
// folded into the loading vectors, and the powers of a0 into all fields, so that the integrand
// has lengths in units of a0 (one FP64 operation less each, on a pipe that bounds the kernels):
//   g0: x, y, z, ATD          (ATD   = D1 * rho0 * (V.n) * ds)
//   g1: Mx, My, Mz, M2        (M     = V / a0^2,  M2 = |V|^2 / a0^2)
//   g2: Mdx, Mdy, Mdz, 0      (Md    = Vdot / a0^2)
//   g3: Lx, Ly, Lz, Lm        (L     = dsD P n / a0^2,  Lm = L.V)
//   g4: Ldx, Ldy, Ldz, 0      (Ld    = dsD (Pdot n + P ndot) / a0^2)
// FP32 records (the mixed form): the 16 fields the integrand cannot do without, 4 groups
// of 4 floats, so that a lane reads an element pair's step with 8 128-bit loads; the
// panel weight dsD is folded into the loading vectors, and |M|^2, L.M and x.vInf are
// recomputed from the fields they are made of:
//   g0: x, y, z, ATD
//   g1: Mx, My, Mz, Ldx'      (Ld' = dsD Ldot)
//   g2: Mdx, Mdy, Mdz, Ldy'
//   g3: Lx', Ly', Lz', Ldz'   (L'  = dsD L)
// In HBM the FP64 records are tiled [element][window][group][32 steps][4]: an (element,
// 32-step window) tile is contiguous (5120 B), which is what one bulk (TMA) copy moves
// into shared memory.  The FP32 records interleave pairs of elements so that the mixed
// kernel reads the two elements' values of a field as one register pair (the operand of
// a packed FP32 instruction): [element pair][window][group][half][32 lanes][4], half 0 =
// (f0 of e, f0 of e+1, f1 of e, f1 of e+1), half 1 = the same for fields 2 and 3; an
// (element pair, window) tile is 4096 B.  Their windows overlap: window w, lane l holds
// step (31 w + l) mod T for 31 w + l = 0 .. T (lanes past T hold zeros), so lane l - 1
// of the same window holds the left end of lane l's source interval and the last window
// reaches step T, which is step 0 one period on (the periodic wrap of core.cu:173-194).
// ceil(T / 31) windows.
constexpr int kGroups = 5;    // FP64 records
constexpr int kGroups32 = 4;  // FP32 records
constexpr int kWin = 32;
constexpr int kStride32 = 31;  // steps between the FP32 records' windows
constexpr int kFields = 18;  // x,y,z,ds, n(3), ndot(3), V(3), Vdot(3), P, Pdot

__host__ __device__ __forceinline__ int nwin32(int T) { return (T + kStride32 - 1) / kStride32; }

// Mixed ring form: a bound, in observer-time bins and with a margin, on how far a
// sample's observer time lies from its step plus the observer's anchor (the retarded
// time of the origin): |t - t0| <= |x| / (a0 - |vInf|), because the travel time through a
// uniformly moving medium changes by at most 1 / (a0 - |vInf|) per unit of source
// displacement; r = the records' largest |x|, kb = oM / dPsi bins per second.
// ring_reach_rate: bins per unit of |x|, a normal float; -1 where there is no bound: flight
// that is not subsonic, or a time that does not run forwards (kb <= 0).
__host__ __device__ __forceinline__ double ring_reach_rate(double vx, double vy, double vz, double a0, double kb)
{
    const double vm = sqrt(vx * vx + vy * vy + vz * vz);
    if (!(vm < 0.999 * a0)) return -1.0;
    const double k = kb / (a0 - vm) * 1.0001;
    return k >= 0x1p-126 && k < 0x1p127 ? k : -1.0;
}
// 1e30 when r is not finite or there is no bound
__host__ __device__ __forceinline__ double ring_reach_bins(float r, double vx, double vy, double vz, double a0,
                                                           double kb)
{
    const double k = ring_reach_rate(vx, vy, vz, a0, kb);
    if (!(r <= 1.0e30f) || k < 0.0) return 1.0e30;
    return (double)r * k + 2.0;
}
// the same in FP32 for the kernels, k = (float)ring_reach_rate: a little larger for its rounding
__host__ __device__ __forceinline__ float ring_reach_float(float r, float k) { return r * k * 1.000001f + 2.01f; }
// Whether the ring kernel serves a deck: a ring of R slots holds every bin a window of 31
// intervals can reach, and the observer-time offset of every sample is bounded by the
// reach, so that the ring kernel needs no per-sample range check.  The second holds when
// the term b = alpha t0 + D0.v + (D0 - x).v of the retarded-time difference quadratic
// stays positive for every source point x and observer D0 (then its denominator b +
// sqrt(q) >= b > 0 and |dt| keeps its bound |x| / (a0 - |vInf|)): b >= sqrt(alpha)
// |D0| - |x| |vInf|, so it suffices that sqrt(alpha) min|D0| > 1.01 |x|max |vInf|; with no
// flight b = alpha t0 >= 0 and a zero b comes with a non-negative discriminant term.
// obs_rmin = the smallest observer distance from the origin (< 0: unknown).
__host__ __device__ __forceinline__ bool ring_ok(float r, double vx, double vy, double vz, double a0, double kb,
                                                 double obs_rmin, int R)
{
    const double reach = ring_reach_bins(r, vx, vy, vz, a0, kb);
    if (!(2.0 * reach + 40.0 <= (double)R)) return false;
    const double vm = sqrt(vx * vx + vy * vy + vz * vz);
    if (vm == 0.0) return true;
    return obs_rmin >= 0.0 && sqrt(a0 * a0 - vm * vm) * obs_rmin > 1.01 * (double)r * vm;
}

// The largest |x| that ring_ok accepts (it is monotone in r), -1 if none: what the kernels
// compare the records' radius with.
inline float ring_limit(double vx, double vy, double vz, double a0, double kb, double obs_rmin, int R)
{
    const auto ok = [&](unsigned bits) {
        float r;
        memcpy(&r, &bits, sizeof(r));
        return ring_ok(r, vx, vy, vz, a0, kb, obs_rmin, R);
    };
    if (!ok(0)) return -1.f;
    // the two bounds solved for r, which a few roundings separate from the last float that
    // passes; found between its neighbours, or between 0 and infinity where they do not hold it
    const double vm = sqrt(vx * vx + vy * vy + vz * vz);
    double guess = (0.5 * (R - 40) - 2.0) / ring_reach_rate(vx, vy, vz, a0, kb);
    if (vm > 0.0) guess = std::min(guess, sqrt(a0 * a0 - vm * vm) * obs_rmin / (1.01 * vm));
    const float g = (float)std::min(std::max(guess, 0.0), 1.0e30);
    unsigned at;
    memcpy(&at, &g, sizeof(at));
    unsigned lo = at > 4 ? at - 4 : 0, hi = at + 4;
    if (!ok(lo)) lo = 0;
    if (ok(hi)) hi = 0x7f800000u;
    while (hi - lo > 1) {
        const unsigned mid = lo + (hi - lo) / 2;
        if (ok(mid)) lo = mid;
        else hi = mid;
    }
    float r;
    memcpy(&r, &lo, sizeof(r));
    return r;
}

// the smallest distance from the origin of n observers given as FP32 (x, y, z) triples
inline double obs_min_distance(const float* xyz, long long n)
{
    double m = n > 0 ? 1.0e300 : -1.0;
    for (long long i = 0; i < n; ++i) {
        const double x = xyz[3 * i], y = xyz[3 * i + 1], z = xyz[3 * i + 2];
        const double d = sqrt(x * x + y * y + z * z);
        if (!(d >= m)) m = d;  // a NaN distance makes the minimum NaN (unknown)
    }
    return m;
}

#ifdef __CUDACC__
// The largest source distance from the origin |x| among the records a kernel writes, as
// the bits of a non-negative float in *word (unsigned order = float order; a NaN
// distance is above every finite one): a warp-wide maximum, then one atomic per warp.
// Every lane of the warp that is still running calls it.
__device__ __forceinline__ void note_radius(unsigned* word, float r)
{
    if (!word) return;
    const unsigned mask = __activemask();
    const unsigned m = __reduce_max_sync(mask, __float_as_uint(fabsf(r)));
    if ((threadIdx.x & 31) == (unsigned)(__ffs(mask) - 1)) atomicMax(word, m);
}
#endif

// The mixed form's anchor of an observer: the retarded time t0 from the origin and what
// follows from it (tonal.cu).  Formed once per observer by the kernels that make the records
// (about 70 FP64 operations, which every warp of the tonal kernel otherwise repeats for
// every work item: 18 us an item of 32 observers; 4165 elements, 500 steps, 203 observers 2.15
// -> 1.96 ms, a batch of 24 small decks 1.58 -> 1.42 ms).
struct alignas(16) Anchor {
    float t0, s0, kf;  // t0, alpha t0 + D0.v, frac(t0 * oM / dPsi)
    int ki;            // round(t0 * oM / dPsi) modulo T, plus toff
    float px, py, pz;  // D0 - t0 v
    float pad;
};
struct AnchorJob {
    const float* obs;  // device [O][3]
    int O, T, toff;
    double alpha, vx, vy, vz, oM, dPsi;
    Anchor* out;       // device [O]
};
// a multiple of T of at least 2^23, added to bin indices before the modulo
inline int bin_offset(int T) { return (int)(((1 << 23) + T - 1) / T * T); }
inline AnchorJob anchor_job(const float* obs, int O, int T, double a0, const double* vinf, double oM, double dPsi,
                            Anchor* out)
{
    AnchorJob j;
    j.obs = obs;
    j.O = O;
    j.T = T;
    j.toff = bin_offset(T);
    j.alpha = a0 * a0 - (vinf[0] * vinf[0] + vinf[1] * vinf[1] + vinf[2] * vinf[2]);
    j.vx = vinf[0];
    j.vy = vinf[1];
    j.vz = vinf[2];
    j.oM = oM;
    j.dPsi = dPsi;
    j.out = out;
    return j;
}

struct DeviceErr {
    unsigned int bits;
    unsigned int disc, order, nonfinite, timeout;
    // work-list counters of the persistent tonal kernel: the next item to take and the
    // blocks done; the last block of a launch sets both back to zero
    int item_next, item_done;
};

struct TonalGeom {
    int E, Epad, T, nW, O;
    double a0, rho, oM, dPsi, dTau;  // dPsi in radians
    double vinf[3];
    double obs_rmin;  // smallest observer distance from the origin (of the FP32 positions; < 0 unknown)
};

// The flight that a kernel is compiled for: none, any, or one without a y component (its
// products with vInf are left out; the results are the same).
enum Wind { kCalm, kWind, kWindXZ };
inline Wind wind_of(double vx, double vy, double vz)
{
    return vy != 0.0 ? kWind : (vx != 0.0 || vz != 0.0) ? kWindXZ : kCalm;
}

// The FP64 form's observer time in bins, u = kb (t_r + tau dTau) with kb = oM / dPsi: the bins
// per second as a value and what its rounding leaves out, and a source step in bins as 1 + eps and
// rounded.  An observer's samples take kbl times its own retarded time of the origin, from which
// theirs differ by a small part.  (With kb and kb dTau rounded and used alone, the error against
// 80-bit arithmetic was 1.0 to 2.1 times that of the observer time in radians, at 1440 steps in
// hover 6.0e-13 of the observer RMS against 2.8e-13.)
struct F64Time {
    double kb, kbl, eps, step;
};
inline F64Time f64_time(double oM, double dPsi, double dTau)
{
    F64Time t;
    t.kb = oM / dPsi;
    t.kbl = fma(-t.kb, dPsi, oM) / dPsi;
    t.eps = fma(dTau, oM, -dPsi) / dPsi;
    t.step = 1.0 + t.eps;
    return t;
}

struct TonalTile {
    int W;      // observers (warps) per block
    int SE;     // elements per pipeline stage
    int NS;     // pipeline stages
    int chunk;  // elements per work item (multiple of SE)
    int nchunk;
    int items;
    int grid;         // blocks launched (the mixed kernel strides over the items)
    int per_sm;       // mixed: blocks that run on an SM at one time
    int tile_group;   // mixed: observer tiles per group of the item order
    int flush_elems;  // mixed: elements summed in FP32 before the FP64 flush
    int opw;          // observers per warp
    bool tm;          // mixed: record stages copied into tensor memory and read from there
    int ring;         // mixed: bin slots per observer of the sliding ring (a power of 2), 0 = whole rows
    int ring_lo;      // mixed: slots of the smaller ring launched before this kernel in the same
                      // plan, which takes the records first when they fit it (0: none)
    size_t smem;
};

// preprocessing (tonal.cu)
struct PrepArgs {
    const float* raw;      // [surf][T][E_i][8] device
    int nsurf;
    const long long* raw_off;  // device: start (floats) of each surface's rows
    const int* e_surf;     // device: surface of each global element
    const int* e_local;    // device: element index within its surface
    const int* e_count;    // device: E_i per surface
    int E, Epad, T;
    double a0, rho, pscale, cfd, dTau;
    int periodic, lowpass;
    double gauss[13];
    double* rec64;         // [Epad][nW][5][32][4] or null
    float* rec32;          // pair-interleaved FP32 records or null
    unsigned* rmax;        // with rec32: the largest |x| (note_radius), or null
    double* fields;        // optional [E][T][18]
    double* cub;           // scratch [E][5]: make_periodic's cubics
    // set by launch_prep: 1 / (2 dTau), 1 / a0, 1 / (4 pi a0), rho / (4 pi), and floats
    double i2dt, ia0, D1, atd;
    float fi2dt, fi4dt2, fD1, fia0, fcfd, frho, fa0;
};
// with rec32: also the anchors of `job`
cudaError_t launch_prep(const PrepArgs& a, const AnchorJob& job, cudaStream_t s);

// Pairs of floats as unevaluated sums x + y (T. J. Dekker, Numer. Math. 18, 1971; TwoSum: D. E.
// Knuth, The Art of Computer Programming 2, 4.2.2): the product and the sum of two floats, exactly.
__host__ __device__ __forceinline__ float2 prod2(float a, float b)
{
    const float p = a * b;
    return make_float2(p, fmaf(a, b, -p));
}
__host__ __device__ __forceinline__ float2 sum2(float a, float b)
{
    const float s = a + b, t = s - a;
    return make_float2(s, (a - (s - t)) + (b - t));
}
// the product of two pairs, to about 2^-46
__host__ __device__ __forceinline__ float2 mul_pair(float2 a, float2 b)
{
    const float p = a.x * b.x;
    return make_float2(p, fmaf(a.x, b.x, -p) + fmaf(a.x, b.y, a.y * b.x));
}
// a b + c d and a.b as pairs, to about 2^-48 of the result, or 2^-70 of the largest term where the
// terms cancel: the rounding errors of the products and sums are summed with theirs in turn
__host__ __device__ __forceinline__ float2 dot2(float a, float b, float c, float d)
{
    const float2 p = prod2(a, b), q = prod2(c, d), s = sum2(p.x, q.x);
    const float2 l = sum2(p.y, q.y), m = sum2(s.y, l.x), h = sum2(s.x, m.x);
    return sum2(h.x, h.y + (l.y + m.y));
}
__host__ __device__ __forceinline__ float2 dot3(const float* a, const float* b)
{
    const float2 p = prod2(a[0], b[0]), q = prod2(a[1], b[1]), r = prod2(a[2], b[2]);
    const float2 s = sum2(p.x, q.x), t = sum2(s.x, r.x);
    const float2 l = sum2(s.y, t.y), m = sum2(p.y, q.y), n = sum2(l.x, m.x), o = sum2(n.x, r.y), h = sum2(t.x, o.x);
    return sum2(h.x, h.y + ((l.y + m.y) + (n.y + o.y)));
}

// records straight from reference-layout AoS arrays (for the drop-in entry points)
struct AosArgs {
    const void* X;  // float or double, AoS as variables.cu:54
    const void* N;
    const void* V;
    const void* PR;
    int is_double;
    int nSurf;
    const int *Ecnt, *XPtr, *NPtr, *VPtr, *PRPtr;  // device: elements and array starts per surface
    int E, Epad, T;
    double a0, rho;
    double* rec64;   // is_double
    float* rec32;    // float storage
    unsigned* rmax;  // with rec32: the largest |x| (note_radius), or null
};
// float storage: also the anchors of `job`
cudaError_t launch_aos_records(const AosArgs& a, const AnchorJob& job, cudaStream_t s);
cudaError_t launch_anchors(const AnchorJob& job, cudaStream_t s);

// What the host needs of a drop-in's device arrays before it can launch anything, in one
// small read: the elements, the flow, whether tObs is the uniform grid t * dPsi that the
// walk of core.cu:199-231 assumes (main.cu:124), the observers' smallest distance.
struct DropinFacts {
    long long E;       // sum of the counts
    double vinf[3];
    double obs_rmin;   // smallest observer distance from the origin, NaN if one is not a number
    int negative;      // a count below zero
    int uneven;        // tObs is another grid
};
cudaError_t launch_dropin_facts(bool is_double, const int* E, int nSurf, const void* vinf, const void* tobs, int T,
                                double dPsi, const void* robs, int O, DropinFacts* out, cudaStream_t s);

// permeable preprocessing (preprocess_per) in place on reference-layout AoS arrays
constexpr int kMaxPerSteps = 4096;
// a surface: its first element and where its arrays start (X, N, V, U, PR; in elements of
// the storage type)
struct alignas(32) PerSurf {
    int first;
    int ptr[5];
};
constexpr int kPerInline = 48;  // surfaces that travel with the launch
// divisor b = 2 dTau, y = RN(1/b), yl the rest of 1/b
struct PerDiv {
    double b, y, yl;
    unsigned span;  // range of the high words that the short quotient takes (0: none)
    int near;       // y is within 2^-54 of 1/b, relatively
};
PerDiv per_div(double b);
struct PerArgs {
    const PerSurf* table;  // device: the surfaces where they are more than kPerInline, else null
    int nSurf, E, T;
    PerDiv div;
    double a0, a02, rhoRef, half_rho, mref2, cfd;  // a02 = pow(a0, 2), mref2 = pow(Mref, 2)
    int periodic, lowpass;
    double gauss[13];
    PerSurf surf[kPerInline];
};
cudaError_t launch_per_prep(void* X, void* N, void* V, void* U, void* PR, bool is_double, const PerArgs& a,
                            cudaStream_t s);
// the 12-column rows of a permeable deck ([surface][step][element][12], raw_off per
// surface) into FP64 AoS arrays d = X [E][T][4], N [E][T][6], V [E][T][6], U [E][T][6],
// PR [E][T][4] (derivative columns and V zero)
cudaError_t launch_per_rows(const float* raw, const long long* raw_off, const int* e_surf, const int* e_local,
                            const int* e_count, int E, int T, double* const d[5], cudaStream_t s);

struct TonalRun {
    TonalGeom g;
    TonalTile t;          // the plan; mixed with t.ring > 0: the ring kernel, then
    TonalTile wide[2];    // the wide-ring kernels (ring > 0: planned; kRingSlotsWide) for records
                          // that reach past the rings before them, and
    TonalTile rows;       // the whole-row kernel, which runs when every ring is too short
    const unsigned* rmax; // mixed: the records' largest |x| (note_radius bits)
    const void* rec;      // rec64 or rec32
    const double* obs64;  // [O][3], FP64 form
    const Anchor* anc;    // [O], mixed form
    double* acc;          // [O][T][2] (zeroed when nchunk > 1)
    DeviceErr* err;
    int precision;
};
cudaError_t plan_tonal(TonalRun& r, int W_req, int SE_req, int items_per_sm, int num_sms, size_t smem_optin,
                       int opw_req = 0, int tm_req = 0, int rows_only = 0);
cudaError_t launch_tonal(const TonalRun& r, cudaStream_t s);

// Constants of one tonal launch (one case), as the kernels read them.
struct KParams {
    const void* rec;
    int Epad, T, nW, O;
    int nW32;               // windows of the FP32 records
    int ring;               // mixed: ring slots per observer (ring kernel), 0 = whole rows
    int ring_lo;            // mixed: slots of the smaller ring launched before (TonalTile::ring_lo)
    int dual;               // mixed: ring kernels and a whole-row kernel are all launched, and
                            // each tests the records' reach
    const unsigned* rmax;   // mixed: the records' largest |x| (note_radius bits)
    float ring_max, ring_lo_max;  // mixed: the largest |x| of records that fit `ring`, `ring_lo` (ring_limit)
    float reach_k;          // mixed: bins of reach per unit of |x| (ring_reach_rate)
    const Anchor* anc;
    const double* obs64;
    // mixed constants, as pairs (both halves equal: the operands of the packed FP32
    // instructions): -alpha, -vInf, a0, oM / dPsi.  16-byte aligned: the kernel reads
    // them two pairs at a time (measured 1.1 % slower at an 8-byte offset)
    alignas(16) float2 nalpha2;
    float2 nvx2, nvy2, nvz2, a02, kb2, alpha2;
    unsigned tmod;  // ceil(2^32 / T): bin index modulo T by multiply-high
    // FP64 constants
    F64Time time;
    double alpha, ialpha, vx, vy, vz, dPsi;
    int W, NS, chunk, nchunk, obs_tiles, flush_groups, tile_group;
    double* acc;
    DeviceErr* err;
};
void fill_kparams(const TonalRun& r, KParams& kp);  // of the plan r.t
void fill_kparams(const TonalRun& r, const TonalTile& tile, KParams& kp);

// Batched (persistent) mixed launch over many cases.  Work item = (case, observer tile,
// element range [e0, e1)); the kernel takes items in array order from *counter.
struct BatchItem {
    int c, ot, e0, e1;
};
// ring stages of the batched kernel: 4, or 2 for stages of 8 elements
constexpr int batch_stages(int SE) { return SE == 8 ? 2 : 4; }
// dynamic shared memory of the persistent kernel for W observers per block, elements per
// stage SE and rows of `rowlen` slots (the longest case's nTime for whole rows, the ring's
// slots for ring cases, whichever is larger)
size_t batch_smem(int W, int SE, int rowlen);
int batch_blocks_per_sm(int W, int SE, int opw, int rowlen);
size_t batch_static_smem(int SE, int opw);  // static shared memory to keep beside batch_smem
cudaError_t launch_tonal_batch(const KParams* d_cases, const BatchItem* d_items, int nitems, int* d_counter, int W,
                               int SE, int opw, int rowlen, int grid, cudaStream_t s);
constexpr int kRingSlots = 512;  // bin slots per observer of the mixed ring kernels (single deck and batched)
// Bin slots per observer of the wide rings, each for records that reach past the ring
// before it, in decks of more steps than its slots (whole rows of a shorter period hold no
// more bins).
constexpr int kWideTiers = 2;
constexpr int kRingSlotsWide[kWideTiers] = {1024, 2048};
static_assert(sizeof(TonalRun::wide) / sizeof(TonalTile) == kWideTiers, "one plan per wide ring");
// the ring that serves records of largest |x| r (ring_ok), for a deck of T steps: the
// first ring, else the first wide ring that does, else 0 (whole rows)
inline int ring_for(float r, double vx, double vy, double vz, double a0, double kb, double obs_rmin, int T)
{
    if (ring_ok(r, vx, vy, vz, a0, kb, obs_rmin, kRingSlots)) return kRingSlots;
    for (int k = 0; k < kWideTiers; ++k)
        if (T > kRingSlotsWide[k] && ring_ok(r, vx, vy, vz, a0, kb, obs_rmin, kRingSlotsWide[k]))
            return kRingSlotsWide[k];
    return 0;
}
// acc [O][T][2] of every case -> pA [T][O] (overwrite)
struct FinCase {
    const double* acc;
    double* pA;
    int O, T, tiles_o, tile0;
};
cudaError_t launch_finalize_batch(const FinCase* d_cases, int ncase, int total_tiles, cudaStream_t s);
// acc [O][T][2] -> pT/pL/pA [T][O]; mode 0 overwrite double, 1 accumulate double,
// 2 accumulate float (drop-in)
cudaError_t launch_finalize(const double* acc, int O, int T, void* pT, void* pL, void* pA, int mode, cudaStream_t s,
                            const DeviceErr* err = nullptr, unsigned* bits = nullptr);

// misc
void gauss_taps(double* w);

}  // namespace acum
