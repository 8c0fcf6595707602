// bpm.cu -- sm_103a kernels of the broadband (BPM) path and its C ABI entry points.
//
// The reference evaluates, for every observer x span section x source step, the BPM
// sub-models over 42 bands and log-adds the seven component levels in dB
// (bb_core.cu:449-583, core() at 591-1043).  Every component level has the form
//     L = 10 log10(D * A) (+ clip)   with  D = d(theta, phi) / r^2
// where only the directivity-over-distance factor D depends on the observer and the
// amplitude A depends on (section, step, band) alone.  The GPU path therefore splits the
// work three ways:
//
//  bb_pos_kernel / bb_prep_kernel   per (section, step), FP64: blade kinematics, chordwise
//      flow speed, table lookups, the fixed-point effective angle of attack and the
//      boundary-layer thicknesses (bb_core.cu:60-444), the chord/span/normal frame, and
//      every band-independent scalar of core() -- the branch decisions of the model are
//      taken here in FP64.
//  bb_spec_kernel    per (section, step, band), FP32: the spectral amplitudes A of the six
//      sub-model components (TBL-TE suction/pressure/separation, LBL-VS, TEB-VS, tip).
//  bb_obs_kernel     per (observer, section, step, band): D from the observer geometry
//      (once per (observer, section, step), shared by all bands through shared memory),
//      then the energies max(D*A, 1e-10) (the reference's -100 dB clip) summed over
//      sections and steps in FP32 partial sums folded into FP64; lane = observer and
//      warp = band pair, so each amplitude is read once per warp as a shared-memory
//      broadcast and one packed FP32 instruction covers both bands.
//  bb_final_kernel   the energy means over steps per (observer, band), in FP64 dB
//  bb_oaspl_kernel   the band sum (OASPL) per observer
//      (bb_core.cu:563-583).
//
// The reference's repeated dB log-adds become plain energy sums, which removes most of
// its transcendental work; the results are equal up to rounding.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <string>
#include <vector>

#include "acum_internal.h"
#include "ctx.h"
#include "ptx.h"

namespace acum {

constexpr int kMaxAoa = 64;  // tables with more AoA entries are refused
constexpr int kSc = 32;    // spectral scalars per (section, step)
constexpr int kGeo = 16;   // geometry record per (section, step)
constexpr int kAmp = 8;    // amplitudes per (section, step, band)

struct BBSurfDev {
    double span, omega, psi_off, tr[3];
    double crot[3], srot[3];  // cosines and sines of the fixed rotation
    int a1, a2;               // the first AoA entries of at least 0 and 6 degrees (0: none)
    int ccw, trip, nsect, sec0;
    long long data_off;
    int ns_t, na_t, nm_t, nr_t;
    int sect_off, aoa_off, mach_off, re_off;
    long long tab_off;
};

struct BpmState {
    int S = 0, nbb = 0, O = 0, T = 0;
    DBuf<BBSurfDev> surf;
    DBuf<int> secsurf, secloc;
    DBuf<double> geom, data, sect_t, aoa_t, mach_t, re_t, table, pos, spl, oaspl, ff;
    DBuf<double> sums, etot;
    // the reference-shaped call: its small arrays as bytes, its float arrays, the same widened
    DBuf<unsigned char> blob;
    DBuf<float> fl, seed_f, out_f;
    DBuf<double> wide;
    std::vector<unsigned char> h_blob;
    size_t bytes() const
    {
        return 8 * (geom.n + data.n + sect_t.n + mach_t.n + aoa_t.n + re_t.n + table.n + pos.n + spl.n + oaspl.n + ff.n +
                    sums.n + etot.n + wide.n) +
               4 * (geo.n + sc.n + amp.n + fl.n + seed_f.n + out_f.n) + blob.n;
    }
    DBuf<float> geo, sc, amp;
    int per_sm = 0;  // blocks of bb_obs_kernel that run on an SM at one time (0: not asked yet)
    bool uploaded = false;
};

static BpmState* state(acum_ctx* c)
{
    if (!c->bpm_state) c->bpm_state = new BpmState();
    return reinterpret_cast<BpmState*>(c->bpm_state);
}

void release_bpm_state(acum_ctx* c)
{
    if (!c->bpm_state) return;
    BpmState* s = state(c);
    s->surf.release(); s->secsurf.release(); s->secloc.release();
    s->geom.release(); s->data.release(); s->sect_t.release(); s->aoa_t.release(); s->mach_t.release();
    s->re_t.release(); s->table.release(); s->pos.release(); s->spl.release(); s->oaspl.release();
    s->blob.release(); s->fl.release(); s->seed_f.release(); s->out_f.release(); s->wide.release(); s->ff.release(); s->sums.release(); s->etot.release();
    s->geo.release(); s->sc.release(); s->amp.release();
    delete s;
    c->bpm_state = nullptr;
}

// ----------------------------------------------------------- model pieces (FP64)

// bb_utils.cu:6-88 -- spectral shape curves A_min, A_max, B_min, B_max
template <typename R>
__device__ __forceinline__ R amin_(R a)
{
    if (a < (R)0.204) return sqrt((R)67.552 - (R)886.788 * (a * a)) - (R)8.219;
    if (a > (R)0.244) return (R)-142.795 * (a * a * a) + (R)103.656 * (a * a) - (R)57.757 * a + (R)6.006;
    return (R)-32.665 * a + (R)3.981;
}
template <typename R>
__device__ __forceinline__ R amax_(R a)
{
    if (a < (R)0.13) return sqrt((R)67.552 - (R)886.788 * (a * a)) - (R)8.219;
    if (a > (R)0.321) return (R)-4.669 * (a * a * a) + (R)3.491 * (a * a) - (R)16.699 * a + (R)1.149;
    return (R)-15.901 * a + (R)1.098;
}
template <typename R>
__device__ __forceinline__ R bmin_(R b)
{
    if (b < (R)0.13) return sqrt((R)16.888 - (R)886.788 * (b * b)) - (R)4.109;
    if (b > (R)0.145) return (R)-817.810 * (b * b * b) + (R)355.21 * (b * b) - (R)135.024 * b + (R)10.619;
    return (R)-83.607 * b + (R)8.138;
}
template <typename R>
__device__ __forceinline__ R bmax_(R b)
{
    if (b < (R)0.1) return sqrt((R)16.888 - (R)886.788 * (b * b)) - (R)4.109;
    if (b > (R)0.187) return (R)-80.541 * (b * b * b) + (R)44.174 * (b * b) - (R)39.381 * b + (R)2.344;
    return (R)-31.313 * b + (R)1.854;
}
// bb_utils.cu:90-121 -- bluntness shape G5
template <typename R>
__device__ __forceinline__ R g5_(R h, R eta)
{
    R mu, m;
    if (h <= (R)0.25) mu = (R)0.1211;
    else if (h <= (R)0.62) mu = (R)-0.2175 * h + (R)0.1755;
    else if (h < (R)1.15) mu = (R)-0.0308 * h + (R)0.0596;
    else mu = (R)0.0242;
    if (h <= (R)0.02) m = 0;
    else if (h < (R)0.5) m = (R)68.724 * h - (R)1.35;
    else if (h <= (R)0.62) m = (R)308.475 * h - (R)121.23;
    else if (h <= (R)1.15) m = (R)224.811 * h - (R)69.354;
    else if (h < (R)1.2) m = (R)1583.28 * h - (R)1631.592;
    else m = (R)268.344;
    if (m < 0) m = 0;
    const R eta0 = -sqrt((m * m * (mu * mu * mu * mu)) / ((R)6.25 + m * m * mu * mu));
    const R k = (R)2.5 * sqrt((R)1.0 - (eta0 / mu) * (eta0 / mu)) - (R)2.5 - m * eta0;
    if (eta <= eta0) return m * eta + k;
    if (eta <= 0) return (R)2.5 * sqrt((R)1.0 - (eta / mu) * (eta / mu)) - (R)2.5;
    if (eta <= (R)0.03616) return sqrt((R)1.5625 - (R)1194.99 * (eta * eta)) - (R)1.25;
    return (R)-155.543 * eta + (R)4.375;
}

// entries of the axis a that x is not below (a comparison of doubles costs the FP64 pipe as
// much as a DFMA: by their order keys)
__device__ __forceinline__ int count_le(const double* a, int n, double x)
{
    int k = 0;
    if (x != x) {
        while (k < n && !(x < a[k])) ++k;
        return k;
    }
    const long long kx = order_key(x);
    while (k < n && !(kx < order_key(a[k]))) ++k;
    return k;
}

// sin and cos of x together: for |x| <= 0.8 their Taylor series (the first terms left out are
// below 2^-62 of the results), else the library's
__device__ __forceinline__ void sincos_small(double x, double* sn, double* cs)
{
    if (((unsigned)__double2hiint(x) & 0x7fffffffu) > 0x3fe99999u) {
        sincos(x, sn, cs);
        return;
    }
    const double z = x * x;
    double s = 1.0 / 355687428096000.0;  // 1 / 17!
    s = fma(s, z, -1.0 / 1307674368000.0);
    s = fma(s, z, 1.0 / 6227020800.0);
    s = fma(s, z, -1.0 / 39916800.0);
    s = fma(s, z, 1.0 / 362880.0);
    s = fma(s, z, -1.0 / 5040.0);
    s = fma(s, z, 1.0 / 120.0);
    s = fma(s, z, -1.0 / 6.0);
    *sn = fma(s * z, x, x);
    double c = -1.0 / 6402373705728000.0;  // 1 / 18!
    c = fma(c, z, 1.0 / 20922789888000.0);
    c = fma(c, z, -1.0 / 87178291200.0);
    c = fma(c, z, 1.0 / 479001600.0);
    c = fma(c, z, -1.0 / 3628800.0);
    c = fma(c, z, 1.0 / 40320.0);
    c = fma(c, z, -1.0 / 720.0);
    c = fma(c, z, 1.0 / 24.0);
    c = fma(c, z, -0.5);
    *cs = fma(c, z, 1.0);
}

struct BBDev {
    const BBSurfDev* surf;
    const int *secsurf, *secloc;
    const double *geom, *data, *sect_t, *aoa_t, *mach_t, *re_t, *table;
    double* pos;  // [S][T][6] quarter chord xyz, trailing edge xyz
    float* geo;   // [S*T][16]
    float* sc;    // [S*T][32]
    int S, T;
    double dtau, i2dtau, a0, vinf[3];
    int t_del;
};

// quarter-chord and trailing-edge positions (bb_core.cu:79-164)
__global__ void bb_pos_kernel(BBDev d)
{
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= (long long)d.S * d.T) return;
    const int gs = (int)(id / d.T), t = (int)(id % d.T);
    const BBSurfDev& su = d.surf[d.secsurf[gs]];
    const int k = d.secloc[gs], ns = su.nsect;
    const double* geo = d.geom + 4 * (size_t)su.sec0;
    const double span = su.span;
    // the y, z of section round(0.75 nsect) (bb_core.cu:88); nsect >= 3 keeps it in range
    const int i75 = min((int)round(ns * 0.75), ns - 1);
    const double c = geo[4 * k + 3] * span;
    double q[3] = {geo[4 * k] * span, geo[4 * i75 + 1] * span, geo[4 * i75 + 2] * span};
    if (su.ccw == 0) q[1] = -q[1];
    double psi = (d.dtau * t * su.omega + su.psi_off * M_PI / 180);
    if (su.ccw == 0) psi = -psi;
    const double th = d.data[su.data_off + ((size_t)t * ns + k) * 7 + 6] * M_PI / 180;
    double ct, st;
    sincos(th, &st, &ct);
    const double e[3] = {q[0], su.ccw == 1 ? q[1] - c * 0.75 * ct : q[1] + c * 0.75 * ct, q[2] - c * 0.75 * st};
    double cs, sn;
    sincos(psi, &sn, &cs);
    const double a[3] = {q[0] * cs - q[1] * sn, q[0] * sn + q[1] * cs, q[2]};
    const double b[3] = {e[0] * cs - e[1] * sn, e[0] * sn + e[1] * cs, e[2]};
    const double *C = su.crot, *S = su.srot;
    const double a1[3] = {a[0], a[1] * C[0] - a[2] * S[0], a[1] * S[0] + a[2] * C[0]};
    const double b1[3] = {b[0], b[1] * C[0] - b[2] * S[0], b[1] * S[0] + b[2] * C[0]};
    const double a2[3] = {a1[0] * C[1] + a1[2] * S[1], a1[1], -a1[0] * S[1] + a1[2] * C[1]};
    const double b2[3] = {b1[0] * C[1] + b1[2] * S[1], b1[1], -b1[0] * S[1] + b1[2] * C[1]};
    const double a3[3] = {a2[0] * C[2] - a2[1] * S[2], a2[0] * S[2] + a2[1] * C[2], a2[2]};
    const double b3[3] = {b2[0] * C[2] - b2[1] * S[2], b2[0] * S[2] + b2[1] * C[2], b2[2]};
    double* o = d.pos + ((size_t)gs * d.T + t) * 6;
    for (int i = 0; i < 3; ++i) {
        o[i] = a3[i] + su.tr[i];
        o[3 + i] = b3[i] + su.tr[i];
    }
}

// trilinear table lookup (bb_utils.cu:124-168): the corners of the (section, Mach, Re) bracket
// and their weights, the same for every column and AoA entry of an item
struct TableAt {
    const double* corner[8];
    double w[8];
    __device__ __forceinline__ double operator()(int col, int ia) const
    {
        const int o = ia * 7 + col;
        double v = w[0] * corner[0][o];
#pragma unroll
        for (int i = 1; i < 8; ++i) v = fma(w[i], corner[i][o], v);
        return v;
    }
};

__device__ __forceinline__ TableAt table_at(const BBDev& d, const BBSurfDev& su, double rr, double mach, double re)
{
    const double* axis[3] = {d.sect_t + su.sect_off, d.mach_t + su.mach_off, d.re_t + su.re_off};
    const int len[3] = {su.ns_t, su.nm_t, su.nr_t};
    const double x[3] = {rr, mach, re};
    int lo[3], hi[3];
    double w[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int k = count_le(axis[i], len[i], x[i]);
        lo[i] = max(0, k - 1);
        hi[i] = min(k, len[i] - 1);
        w[i] = lo[i] == hi[i] ? 0.5 : (x[i] - axis[i][lo[i]]) * rcp_d(axis[i][hi[i]] - axis[i][lo[i]]);
    }
    TableAt t;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int s = i & 1 ? hi[0] : lo[0], m = i & 2 ? hi[1] : lo[1], r = i & 4 ? hi[2] : lo[2];
        t.corner[i] = d.table + su.tab_off + (((size_t)s * su.nm_t + m) * su.nr_t + r) * su.na_t * 7;
        t.w[i] = (i & 1 ? w[0] : 1.0 - w[0]) * ((i & 2 ? w[1] : 1.0 - w[1]) * (i & 4 ? w[2] : 1.0 - w[2]));
    }
    return t;
}

// everything per (section, step) that does not depend on the observer or the band.  Bound by
// the FP64 pipe (a small deck by its latency): the table's bracket and weights are formed
// once, cl only at the AoA entries that are used, sines and cosines by sincos_small, powers
// of ten by exp10, quotients by rcp_d, and conversions and comparisons by integers (200
// sections of 720 steps 690 -> 230 us, 42 sections of 180 steps 123 -> 51 us).
__global__ void __launch_bounds__(32) bb_prep_kernel(BBDev d)
{
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= (long long)d.S * d.T) return;
    const int gs = (int)(id / d.T), t = (int)(id % d.T);
    const BBSurfDev& su = d.surf[d.secsurf[gs]];
    const int k = d.secloc[gs], ns = su.nsect, T = d.T;
    const double* geo = d.geom + 4 * (size_t)su.sec0;
    const double span = su.span;
    const double c = geo[4 * k + 3] * span;
    const double nu = 0.0000181206 / 1.22500;
    auto P = [&](int sec, int tt) { return d.pos + (((size_t)(su.sec0 + sec)) * T + tt) * 6; };
    const int tm = t == 0 ? T - 1 : t - 1, tp = t == T - 1 ? 0 : t + 1;
    const double* x0 = P(k, t);
    const double* xt = x0 + 3;
    // chordwise flow speed, Mach and Re (bb_core.cu:166-206); tr[0] = the chord's direction
    double v[3], tr[3][3], n;
    for (int i = 0; i < 3; ++i) v[i] = d.vinf[i] - (P(k, tp)[i] - P(k, tm)[i]) * d.i2dtau;
    for (int i = 0; i < 3; ++i) tr[0][i] = xt[i] - x0[i];
    n = rcp_d(sqrt_d(tr[0][0] * tr[0][0] + tr[0][1] * tr[0][1] + tr[0][2] * tr[0][2]));
    for (int i = 0; i < 3; ++i) tr[0][i] *= n;
    const double um = v[0] * tr[0][0] + v[1] * tr[0][1] + v[2] * tr[0][2];
    const double mach = fabs(um / d.a0);
    const double re = fabs(um * c / nu);
    // table brackets and cl(alpha) (bb_core.cu:208-250)
    const TableAt tab = table_at(d, su, geo[4 * k], mach, re);
    const double* aoa = d.aoa_t + su.aoa_off;
    const int na = su.na_t;
    int a3 = 0;
    for (int i = 0; i < na; ++i) {
        const double cl = tab(0, i);
        const int h = __double2hiint(cl);
        // cl > 0
        if ((h > 0 || (h == 0 && __double2loint(cl) != 0)) && (h < 0x7ff00000 || (h == 0x7ff00000 && __double2loint(cl) == 0))) {
            a3 = i;
            break;
        }
    }
    // indices clamped to the table so a malformed table cannot read outside it
    int a1 = max(su.a1, 1);
    a3 = max(a3, 1);
    const double cl1 = tab(0, a1), cl3 = tab(0, a3), cl3m = tab(0, a3 - 1);
    const double icla = (aoa[su.a2] - aoa[a1]) * rcp_d(tab(0, su.a2) - cl1);
    double w = (0 - aoa[a1 - 1]) * rcp_d(aoa[a1] - aoa[a1 - 1]);
    const double cl0 = tab(0, a1 - 1) * (1 - w) + cl1 * w;
    w = (0 - cl3m) * rcp_d(cl3 - cl3m);
    const double al0 = aoa[a3 - 1] * (1 - w) + aoa[a3] * w;
    // effective angle of attack by fixed point (bb_core.cu:291-321)
    const double* row = d.data + su.data_off + ((size_t)t * ns + k) * 7;
    const double cn = row[4], ct = row[5];
    double ae = 0.0;
    for (int it = 0; it <= 50; ++it) {
        double sn, cs;
        sincos_small(ae * (M_PI / 180), &sn, &cs);
        const double ae1 = (cn * cs - ct * sn - cl0) * icla;
        const double err = fabs(ae1 - ae);
        ae = ae1;
        // until err <= 1e-3 (bits 0x3f50624dd2f1a9fc), or not a number
        const long long e = __double_as_longlong(err);
        if (e <= 0x3f50624dd2f1a9fcLL || e > 0x7ff0000000000000LL) break;
    }
    const double alpha = fabs(ae - al0);
    // boundary-layer thicknesses (bb_core.cu:353-438)
    const double lr = log10(re);
    double bl[4];
    if (d.t_del == 0) {
        for (int i = 0; i < 4; ++i) bl[i] = row[i];
    } else if (d.t_del == 1) {
        for (int i = 0; i < na; ++i)
            if (aoa[i] >= ae) { a1 = i; break; }
        a1 = max(a1, 1);
        const double wa = (ae - aoa[a1 - 1]) * rcp_d(aoa[a1] - aoa[a1 - 1]);
        for (int i = 0; i < 4; ++i) bl[i] = c * (tab(i + 3, a1 - 1) * (1 - wa) + tab(i + 3, a1) * wa);
    } else {
        const double d0 = c * exp10(1.6569 - 0.9045 * lr + 0.0596 * (lr * lr));
        const double ds0 = c * exp10(3.0187 - 1.5397 * lr + 0.1059 * (lr * lr));
        bl[1] = d0 * exp10(-0.04175 * alpha + 0.00106 * (alpha * alpha));
        bl[3] = ds0 * exp10(-0.0432 * alpha + 0.00113 * (alpha * alpha));
        const bool low = alpha <= 7.5, high = alpha > 12.5;
        bl[0] = d0 * (low ? 1.0 : high ? 12.0 : 0.0303) * exp10((low ? 0.03114 : high ? 0.0258 : 0.2336) * alpha);
        bl[2] = ds0 * (low ? 1.0 : high ? 52.42 : 0.0162) * exp10((low ? 0.0679 : high ? 0.0258 : 0.3066) * alpha);
    }
    // chord/span/normal frame of the section (bb_core.cu:473-513)
    const int km = k == ns - 1 ? k - 1 : k, kp = k == ns - 1 ? k : k + 1;
    for (int i = 0; i < 3; ++i) tr[1][i] = P(kp, t)[i] - P(km, t)[i];
    n = rcp_d(sqrt_d(tr[1][0] * tr[1][0] + tr[1][1] * tr[1][1] + tr[1][2] * tr[1][2]));
    for (int i = 0; i < 3; ++i) tr[1][i] *= n;
    const double turn = su.ccw == 1 ? 1.0 : -1.0;  // clockwise: span x chord
    tr[2][0] = turn * (tr[0][1] * tr[1][2] - tr[0][2] * tr[1][1]);
    tr[2][1] = turn * (tr[0][2] * tr[1][0] - tr[0][0] * tr[1][2]);
    tr[2][2] = turn * (tr[0][0] * tr[1][1] - tr[0][1] * tr[1][0]);
    n = sqrt_d(tr[2][0] * tr[2][0] + tr[2][1] * tr[2][1] + tr[2][2] * tr[2][2]);
    // the clockwise branch divides by the square root of the norm (bb_core.cu:510-512)
    n = rcp_d(su.ccw == 1 ? n : sqrt_d(n));
    for (int i = 0; i < 3; ++i) tr[2][i] *= n;
    double ls;
    if (k == 0) ls = (geo[4 * (k + 1)] - geo[4 * k]) / 2.0 * span;
    else if (k == ns - 1) ls = (geo[4 * k] - geo[4 * (k - 1)]) / 2.0 * span;
    else ls = (geo[4 * (k + 1)] - geo[4 * (k - 1)]) / 2.0 * span;

    // band-independent scalars of core() (bb_core.cu:599-1039)
    double del_s = bl[0], del_p = bl[1], dis_s = bl[2], dis_p = bl[3];
    if (del_s < 0.0) del_s = 1.0e-10;
    if (del_p < 0.0) del_p = 1.0e-10;
    if (dis_p < 0.0) dis_p = 1.0e-10;
    if (dis_s < 0.0) dis_s = 1.0e-10;
    const double u = fabs(um), M = mach, rc = re, mc = 0.6 * mach;
    const double rdp = u * dis_p / nu;
    const double st1 = 0.02 * exp10(-0.6 * log10(M));
    double st2;
    if (alpha < 1.33) st2 = st1;
    else if (alpha > 12.5) st2 = st1 * 4.72;
    else st2 = st1 * exp10(0.0054 * ((alpha - 1.33) * (alpha - 1.33)));
    double a0r;
    if (rc < 9.52e4) a0r = 0.57;
    else if (rc > 8.57e5) a0r = 1.13;
    else a0r = (-9.57e-13) * ((rc - 8.57e5) * (rc - 8.57e5)) + 1.13;
    const double ar = (-20.0 - amin_(a0r)) / (amax_(a0r) - amin_(a0r));
    double b0r;
    if (rc < 9.52e4) b0r = 0.3;
    else if (rc > 8.57e5) b0r = 0.56;
    else b0r = (-4.48e-13) * ((rc - 8.57e5) * (rc - 8.57e5)) + 0.56;
    const double brr = (-20.0 - bmin_(b0r)) / (bmax_(b0r) - bmin_(b0r));
    double k1;
    if (rc < 2.47e5) k1 = -4.31 * lr + 156.3;
    else if (rc > 8.0e5) k1 = 128.5;
    else k1 = -9.0 * lr + 181.6;
    const double dk1 = rdp <= 5000 ? alpha * (1.43 * log10(rdp) - 5.29) : 0.0;
    const double gam = 27.094 * M + 3.31, gam0 = 23.43 * M + 4.651, bet = 72.65 * M + 10.74, bet0 = -34.19 * M - 13.82;
    double k2;
    if (alpha < gam0 - gam) k2 = k1 - 1000.0;
    else if (alpha > gam0 + gam) k2 = k1 - 12.0;
    else {
        const double bg = bet * rcp_d(gam);
        k2 = k1 + sqrt_d(bet * bet - bg * bg * ((alpha - gam0) * (alpha - gam0))) + bet0;
    }
    const bool stall = (alpha >= gam0 || alpha > 12.5);
    double ars = 0.0, k2s = 0.0;
    if (stall) {
        const double rcn = 3.0 * rc;
        double a0n;
        if (rcn < 9.52e4) a0n = 0.57;
        else if (rcn > 8.57e5) a0n = 1.13;
        else a0n = -9.57e-13 * ((rcn - 8.57e5) * (rcn - 8.57e5)) + 1.13;
        double k1n;
        if (rcn < 2.47e5) k1n = -4.31 * log10(rcn) + 156.3;
        else if (rcn > 8e5) k1n = 128.5;
        else k1n = -9.0 * log10(rcn) + 181.6;
        if (alpha < gam0 - gam) k2s = k1n - 1000.0;
        else if (alpha > gam0 + gam) k2s = k1n - 12.0;
        else k2s = k1n + sqrt(bet * bet - ((bet / gam) * (bet / gam)) * ((alpha - gam0) * (alpha - gam0))) + bet0;
        ars = (-20.0 - amin_(a0n)) / (amax_(a0n) - amin_(a0n));
    }
    const double m5 = (M * M) * (M * M) * M;
    // LBL-VS (bb_core.cu:863-915)
    double stpk = 1.0, g23 = 0.0;
    const int trip0 = su.trip == 0;
    if (trip0) {
        double stl;
        if (rc < 1.3e5) stl = 0.18;
        else if (rc > 1.3e5 && rc <= 4e5) stl = 0.001756 * exp10(0.3931 * lr);
        else stl = 0.28;
        stpk = exp10(-0.04 * alpha) * stl;
        const double rc0 = exp10(alpha <= 3.0 ? 0.215 * alpha + 4.978 : 0.120 * alpha + 5.263);
        const double dd = rc * rcp_d(rc0), ld = log10(dd);
        double g2;
        if (dd <= 0.3237) g2 = 77.852 * ld + 15.328;
        else if (dd <= 0.5689) g2 = 65.188 * ld + 9.125;
        else if (dd <= 1.7579) g2 = -114.052 * (ld * ld);
        else if (dd <= 3.0889) g2 = -65.188 * ld + 9.125;
        else g2 = -77.852 * ld + 15.328;
        g23 = g2 + (171.04 - 3.03 * alpha);
    }
    // TEB-VS, h = 0.5 mm, psi = 14 deg (bb_core.cu:917-971)
    const double h = 0.0005, psiv = 14.0;
    const double dh_ = (dis_s + dis_p) / 2.0 / h, hd = rcp_d(dh_);
    const double aterm = 0.212 - 0.0045 * psiv;
    const double stpeak =
        hd >= 0.2 ? aterm / (1.0 + 0.235 * dh_ - 0.0132 * (dh_ * dh_)) : 0.1 * hd + 0.095 - 0.00243 * psiv;
    const double g4 = hd <= 5.0 ? 17.5 * log10(hd) + 157.5 - 1.114 * psiv : 169.7 - 1.114 * psiv;
    const double hdp = 6.724 * (hd * hd) - 4.019 * hd + 1.107;
    // tip vortex on the last section (bb_core.cu:975-1039)
    const int tip = k == ns - 1;
    double tl = 1.0, umm = 1.0, gtip = 0.0;
    if (tip) {
        const double ar0[6] = {2.0, 2.67, 4.0, 6.0, 12.0, 24.0};
        const double rat0[6] = {0.54, 0.62, 0.71, 0.79, 0.89, 0.95};
        const double AR = span / c;
        double rat;
        if (AR < ar0[0]) rat = rat0[0];
        else if (AR > ar0[5]) rat = rat0[5];
        else {
            int kk = 0;
            while (kk < 5 && !(AR < ar0[kk])) kk++;
            kk = max(kk, 1);
            rat = rat0[kk - 1] * (ar0[kk] - AR) / (ar0[kk] - ar0[kk - 1]) +
                  rat0[kk] * (AR - ar0[kk - 1]) / (ar0[kk] - ar0[kk - 1]);
        }
        const double at = alpha * rat;
        tl = fabs(at) <= 2.0 ? (0.023 + 0.0169 * at) * c : (0.0378 + 0.0095 * at) * c;
        const double mm = (1.0 + 0.036 * at) * M;
        umm = mm * d.a0;
        gtip = M * M * (mm * mm * mm) * (tl * tl);
    }

    float4* g = reinterpret_cast<float4*>(d.geo + id * kGeo);
    const auto f = [](double y) { return narrow_d(y); };
    const float Mf = f(M), mcf = f(mc), st = stall ? 1.f : 0.f;
    g[0] = make_float4(f(xt[0]), f(xt[1]), f(xt[2]), f(tr[0][0]));
    g[1] = make_float4(f(tr[0][1]), f(tr[0][2]), f(tr[1][0]), f(tr[1][1]));
    g[2] = make_float4(f(tr[1][2]), f(tr[2][0]), f(tr[2][1]), f(tr[2][2]));
    g[3] = make_float4(Mf, mcf, st, 0.f);
    float4* q = reinterpret_cast<float4*>(d.sc + id * kSc);
    q[0] = make_float4(f(u), Mf, mcf, f(dis_s));
    q[1] = make_float4(f(dis_p), f(del_p), f(ls), f(st1));
    q[2] = make_float4(f(st2), f(ar), f(brr), f(k1 - 3.0));
    q[3] = make_float4(f(dk1), f(k2), st, f(ars));
    q[4] = make_float4(f(k2s), (float)trip0, f(stpk), f(g23));
    q[5] = make_float4(f(hd), f(stpeak), f(g4), f(hdp));
    q[6] = make_float4((float)tip, f(tl), f(umm), f(gtip));
    q[7] = make_float4(f(dis_p * m5 * ls), f(dis_s * m5 * ls), f(del_p * m5 * ls), f(m5 * sqrt_d(M) * h * ls));
}

// spectral amplitudes per (section, step, band), FP32 (bb_core.cu:637-1039)
__global__ void bb_spec_kernel(const float* __restrict__ sc, const double* __restrict__ ff, float* __restrict__ amp,
                               long long nst)
{
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= nst * kBands) return;
    const long long st = id / kBands;
    const int fb = (int)(id % kBands);
    const float* q = sc + st * kSc;
    const float f = (float)ff[fb];
    const float u = q[0];
    const float sts = f * q[3] / u, stp = f * q[4] / u;
    // TBL-TE pressure and suction sides
    const float as = fabsf(log10f(sts / q[7])), ap = fabsf(log10f(stp / q[7]));
    const float aas = amin_(as) + q[9] * (amax_(as) - amin_(as));
    const float aap = amin_(ap) + q[9] * (amax_(ap) - amin_(ap));
    const float Ap = q[28] * exp10f((aap + q[11] + q[12]) * 0.1f);
    const float As = q[29] * exp10f((aas + q[11]) * 0.1f);
    // separation (angle-of-attack) contribution
    float Aa;
    const float b = fabsf(log10f(sts / q[8]));
    if (q[14] != 0.f) Aa = q[29] * exp10f((amin_(b) + q[15] * (amax_(b) - amin_(b)) + q[16]) * 0.1f);
    else Aa = q[29] * exp10f((bmin_(b) + q[10] * (bmax_(b) - bmin_(b)) + q[13]) * 0.1f);
    // LBL-VS
    float Al = 0.f;
    if (q[17] != 0.f) {
        const float e = (f * q[5] / u) / q[18], le = log10f(e);
        float g1;
        if (e <= 0.5974f) g1 = 39.8f * le - 11.12f;
        else if (e <= 0.8545f) g1 = 98.409f * le + 2.0f;
        else if (e <= 1.17f) g1 = -5.076f + sqrtf(2.484f - 506.25f * (le * le));
        else if (e <= 1.674f) g1 = -98.409f * le + 2.0f;
        else g1 = -39.80f * le - 11.12f;
        Al = q[30] * exp10f((g1 + q[19]) * 0.1f);
    }
    // TEB-VS
    const float eta = log10f((f * 0.0005f / u) / q[21]);
    const float g514 = g5_(q[20], eta), g50 = g5_(q[23], eta);
    float g5 = g50 + 0.0714f * 14.0f * (g514 - g50);
    if (g5 > 0.f) g5 = 0.f;
    const float f4 = g5_(0.25f, eta);
    if (g5 > f4) g5 = f4;
    const float At = q[31] * exp10f((q[22] + g5) * 0.1f);
    // tip vortex
    float Av = 0.f;
    if (q[24] != 0.f) {
        const float lg = log10f(f * q[25] / q[26]) + 0.3f;
        Av = exp10f((126.0f - 30.5f * (lg * lg)) * 0.1f);
    }
    // band pairs interleaved: [item][band / 2][field][band % 2] (the operand pairs of the
    // packed contraction in bb_obs_kernel)
    float* o = amp + st * (kBands * kAmp) + (size_t)(fb >> 1) * (2 * kAmp) + (fb & 1);
    const float v[kAmp] = {Ap, As, Aa, Al, At, Av, q[27], 0.f};
#pragma unroll
    for (int c = 0; c < kAmp; ++c) o[2 * c] = v[c];
}

// Observer contraction.  Block = 64 observers (lane l serves observers l and l + 32) x
// 21 warps, one per pair of bands.  Per tile of kTI (section, step) items, the amplitudes
// of all 42 bands (contiguous in `amp`, 1344 B per item, band pairs interleaved) and the
// items' geometry records arrive in shared memory by one bulk copy into a ring of three
// buffers (two tiles ahead of the one consumed); the directivity factors D of the block's
// observers are computed into shared memory one tile ahead (double-buffered, each stored
// twice, as the operand pair of a packed instruction), in the same phase as the current
// tile's sums, so that one block barrier per tile separates the phases; each lane adds,
// for its two observers and its warp's two bands, the clipped energies of every item in
// packed FP32 (one f32x2 operation covers both bands).  The amplitude reads are warp-uniform (shared-
// memory broadcasts), the D reads conflict-free.  FP32 partial sums over at most 1024
// items are folded into FP64 sums private to the block's (observer tile, item range):
// part[split][band][component][observer], reduced over the splits by bb_final_kernel.
// Bound by the FMA and ALU pipes (per item and 64 observers a warp issues 36 products, maxima
// and sums beside 6 loads and the D of its share): items in groups of eight, which keep the
// loads ahead and one address (200 sections x 720 steps x 1024 observers 4.08 -> 3.92 ms).
constexpr int kObsPerLane = 2;
constexpr int kObsBlock = 32 * kObsPerLane;  // 64
constexpr int kPairWarps = kBands / 2;       // 21
constexpr int kBpmThreads = 32 * kPairWarps; // 672
constexpr int kTI = 32;                      // items per tile
constexpr int kFoldTiles = 32;               // 1024 items per FP32 partial
constexpr int kAmpItemBytes = kBands * kAmp * 4;  // 1344
constexpr int kGeoItemBytes = kGeo * 4;           // 64
static_assert(kBands % 2 == 0, "band pairs");
static_assert(kAmpItemBytes % 16 == 0 && kGeoItemBytes % 16 == 0, "bulk copy granularity");

// dynamic shared memory of bb_obs_kernel: kObsRing x (amplitude tile + geometry tile), 2 D
// tiles (float4 (Dh, Dh, Dl, Dl) per item and observer), the block's observers, kObsRing
// mbarriers
constexpr int kObsRing = 3;
constexpr size_t kObsSmemA = (size_t)kTI * kAmpItemBytes;
constexpr size_t kObsSmemG = (size_t)kTI * kGeoItemBytes;
constexpr size_t kObsSmemBuf = kObsSmemA + kObsSmemG;
constexpr size_t kObsSmemD = (size_t)kTI * kObsBlock * sizeof(float4);
constexpr size_t kObsSmem =
    kObsRing * kObsSmemBuf + 2 * kObsSmemD + kObsBlock * 3 * sizeof(float) + kObsRing * sizeof(uint64_t);

__device__ __forceinline__ float2 bb_directivity(const float* geo, const float* obs, int o, float vx, float vy,
                                                 float vz, float aa, float iaMv)
{
    const float4* g = reinterpret_cast<const float4*>(geo);
    const float4 g0 = g[0], g1 = g[1], g2 = g[2], g3 = g[3];
    float rx = obs[3 * o] - g0.x, ry = obs[3 * o + 1] - g0.y, rz = obs[3 * o + 2] - g0.z;
    // convected emission time (bb_core.cu:515-520)
    const float bb = rx * vx + ry * vy + rz * vz;
    const float cc = rx * rx + ry * ry + rz * rz;
    const float tau = (-bb + sqrtf(bb * bb + aa * cc)) * iaMv;
    rx -= vx * tau;
    ry -= vy * tau;
    rz -= vz * tau;
    const float r2 = rx * rx + ry * ry + rz * rz;
    // frame rows: chord (g0.w, g1.x, g1.y), span (g1.z, g1.w, g2.x), normal (g2.y, g2.z, g2.w)
    const float p0 = rx * g0.w + ry * g1.x + rz * g1.y;
    const float p1 = rx * g1.z + ry * g1.w + rz * g2.x;
    const float p2 = rx * g2.y + ry * g2.z + rz * g2.w;
    const float cx = fabsf(p0) * rsqrtf(r2);                // cos(theta)
    const float cy = fabsf(p1) * rsqrtf(p1 * p1 + p2 * p2);  // cos(phi)
    // sin^2(theta/2), sin^2(theta), sin^2(phi) without the acos; a zero angle is replaced
    // by 1e-10 as the reference does (bb_core.cu:525-530)
    const float sh2 = cx >= 1.f ? 2.5e-21f : 0.5f * (1.f - cx);
    const float sth2 = cx >= 1.f ? 1e-20f : (1.f - cx) * (1.f + cx);
    const float sp2 = cy >= 1.f ? 1e-20f : (1.f - cy) * (1.f + cy);
    // directivities d_h, d_l (bb_core.cu:620-624) over r^2
    const float M = g3.x, Mc = g3.y;
    const float q1 = 1.f + M * cx, q2 = 1.f + (M - Mc) * cx;
    const float Dh = __fdividef(2.f * sh2 * sp2, q1 * q2 * q2 * r2);
    const float Dl = __fdividef(sth2 * sp2, q1 * q1 * q1 * q1 * r2);
    return make_float2(Dh, g3.z != 0.f ? Dl : Dh);
}

__device__ __forceinline__ float2 clip2(float2 v, float lo) { return make_float2(fmaxf(v.x, lo), fmaxf(v.y, lo)); }

__global__ void __launch_bounds__(kBpmThreads, 1) bb_obs_kernel(const float* __restrict__ geo,
                                                                const float* __restrict__ amp,
                                                                const float* __restrict__ obs, int O, long long nst,
                                                                long long per_split, float vx, float vy, float vz,
                                                                float a0, int aa_mode, double* __restrict__ part,
                                                                DeviceErr* err)
{
    extern __shared__ __align__(128) unsigned char sm[];
    float4* sD0 = reinterpret_cast<float4*>(sm + kObsRing * kObsSmemBuf);  // 2 x [kTI][kObsBlock]
    float* sObs = reinterpret_cast<float*>(sm + kObsRing * kObsSmemBuf + 2 * kObsSmemD);
    uint64_t* bars =
        reinterpret_cast<uint64_t*>(sm + kObsRing * kObsSmemBuf + 2 * kObsSmemD + kObsBlock * 3 * sizeof(float));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;  // warp = band pair
    const int o0 = blockIdx.x * kObsBlock;
    const long long st_begin = (long long)blockIdx.y * per_split;
    const long long st_end = min(nst, st_begin + per_split);
    const int ntiles = st_end > st_begin ? (int)((st_end - st_begin + kTI - 1) / kTI) : 0;
    const float aMv = a0 * a0 - (vx * vx + vy * vy + vz * vz);
    const float aa = aa_mode == 1 ? 0.f : aMv;
    const float iaMv = 1.0f / aMv;
    double* mine = part + (size_t)blockIdx.y * kBands * 6 * O;  // [band][component][observer]

    for (int i = threadIdx.x; i < kObsBlock * 3; i += blockDim.x) {
        const int o = o0 + i / 3;
        sObs[i] = o < O ? obs[3 * o0 + i] : 0.f;
    }
    if (threadIdx.x == 0) {
        for (int b = 0; b < kObsRing; ++b) mbar_init(&bars[b], 1);
        mbar_fence_init();
    }
    __syncthreads();
    // tile j -> buffer j % kObsRing (phase j / kObsRing of its barrier): amplitudes, then
    // the geometry of its items
    auto tile_n = [&](int j) { return (int)min((long long)kTI, st_end - (st_begin + (long long)j * kTI)); };
    auto buf_of = [&](int j) { return sm + (size_t)(j % kObsRing) * kObsSmemBuf; };
    auto issue = [&](int j) {
        const long long t0 = st_begin + (long long)j * kTI;
        const int n = tile_n(j);
        unsigned char* buf = buf_of(j);
        mbar_expect_tx(&bars[j % kObsRing], (uint32_t)(n * (kAmpItemBytes + kGeoItemBytes)));
        bulk_g2s(buf, amp + t0 * kBands * kAmp, (uint32_t)(n * kAmpItemBytes), &bars[j % kObsRing]);
        bulk_g2s(buf + kObsSmemA, geo + t0 * kGeo, (uint32_t)(n * kGeoItemBytes), &bars[j % kObsRing]);
    };
    auto wait_tile = [&](int j) {
        return mbar_wait_bounded(&bars[j % kObsRing], (uint32_t)((j / kObsRing) & 1));
    };
    // D of every (item, observer) of tile j (bb_core.cu:515-530, 620-624) into D buffer j & 1
    auto directivity = [&](int j) {
        const int n = tile_n(j);
        const float* sG = reinterpret_cast<const float*>(buf_of(j) + kObsSmemA);
        float4* sD = sD0 + (size_t)(j & 1) * kTI * kObsBlock;
#pragma unroll 1
        for (int pidx = threadIdx.x; pidx < kTI * kObsBlock; pidx += blockDim.x) {
            const int it = pidx / kObsBlock, ol = pidx % kObsBlock;
            float2 D = make_float2(0.f, 0.f);
            if (it < n && o0 + ol < O) D = bb_directivity(sG + it * kGeo, sObs, ol, vx, vy, vz, aa, iaMv);
            sD[it * kObsBlock + ol] = make_float4(D.x, D.x, D.y, D.y);
        }
    };
    int issued = 0;
    if (threadIdx.x == 0)
        for (; issued < kObsRing && issued < ntiles; ++issued) issue(issued);

    float2 acc[kObsPerLane][6];  // (band 2 warp, band 2 warp + 1)
#pragma unroll
    for (int q = 0; q < kObsPerLane; ++q)
#pragma unroll
        for (int c = 0; c < 6; ++c) acc[q][c] = make_float2(0.f, 0.f);
    auto fold = [&]() {
#pragma unroll
        for (int q = 0; q < kObsPerLane; ++q) {
            const int o = o0 + q * 32 + lane;
            if (o < O) {
                // addresses formed here, not hoisted out of the item loop
                size_t stride = (size_t)O;
                asm volatile("" : "+l"(stride));
                double* p0 = mine + (size_t)(2 * warp) * 6 * stride + o;  // band 2 warp
                double* p1 = p0 + 6 * stride;                             // band 2 warp + 1
#pragma unroll
                for (int c = 0; c < 6; ++c) {
                    p0[c * stride] += (double)acc[q][c].x;
                    p1[c * stride] += (double)acc[q][c].y;
                }
            }
#pragma unroll
            for (int c = 0; c < 6; ++c) acc[q][c] = make_float2(0.f, 0.f);
        }
    };
    int aborted_at = -1;
    if (ntiles > 0) {
        const bool ok = wait_tile(0);
        if (ok) directivity(0);
        if (__syncthreads_or(!ok)) aborted_at = 0;
    }
    int tiles = 0;
    for (int j = 0; j < ntiles && aborted_at < 0; ++j) {
        // the next tile's D, in the same phase as this tile's sums
        bool ok = true;
        if (j + 1 < ntiles) {
            ok = wait_tile(j + 1);
            if (ok) directivity(j + 1);
        }
        const int n = tile_n(j);
        const float4* sA = reinterpret_cast<const float4*>(buf_of(j));
        const float4* sD = sD0 + (size_t)(j & 1) * kTI * kObsBlock;
#pragma unroll 8
        for (int it = 0; it < n; ++it) {
            // the warp's band pair: fields (Ap, As), (Aa, Al), (At, Av), (gtip, -) of both bands
            const float4* a = sA + (it * kPairWarps + warp) * 4;
            const float4 a0v = a[0], a1v = a[1], a2v = a[2], a3v = a[3];
            const float2 Ap = make_float2(a0v.x, a0v.y), As = make_float2(a0v.z, a0v.w);
            const float2 Aa = make_float2(a1v.x, a1v.y), Al = make_float2(a1v.z, a1v.w);
            const float2 At = make_float2(a2v.x, a2v.y), Av = make_float2(a2v.z, a2v.w);
            const float2 Ag = make_float2(a3v.x, a3v.y);
            const bool tip = Av.x != 0.f || Av.y != 0.f;
#pragma unroll
            for (int q = 0; q < kObsPerLane; ++q) {
                const float4 D = sD[it * kObsBlock + q * 32 + lane];
                const float2 Dh = make_float2(D.x, D.y), Dl = make_float2(D.z, D.w);
                acc[q][0] = add2(acc[q][0], clip2(mul2(Dh, Ap), 1e-10f));  // TBL-TE pressure side
                acc[q][1] = add2(acc[q][1], clip2(mul2(Dh, As), 1e-10f));  // TBL-TE suction side
                acc[q][2] = add2(acc[q][2], clip2(mul2(Dl, Aa), 1e-10f));  // separation
                acc[q][3] = fma2(Dh, Al, acc[q][3]);                       // LBL-VS
                acc[q][4] = fma2(Dh, At, acc[q][4]);                       // TEB-VS
                if (tip) acc[q][5] = fma2(Av, clip2(mul2(Dh, Ag), 2.2204460492503131e-16f), acc[q][5]);  // tip
            }
        }
        // every thread is done with tile j's buffer and D tile, and tile j + 1's D is
        // complete: refill the buffer with tile j + kObsRing
        if (__syncthreads_or(!ok)) {
            aborted_at = j + 1;
            break;
        }
        if (threadIdx.x == 0 && j + kObsRing < ntiles) issue(issued++);
        if (++tiles == kFoldTiles) {
            fold();
            tiles = 0;
        }
    }
    if (aborted_at >= 0) {
        // wait (bounded) for the copies still in flight (tiles aborted_at .. issued - 1,
        // counted by thread 0, which issues them) before the block exits
        if (threadIdx.x == 0) {
            flag(err, ACUM_DEVERR_TIMEOUT, &err->timeout);
            for (int j = aborted_at; j < issued; ++j) (void)wait_tile(j);
        }
        __syncthreads();
        return;
    }
    fold();
}

// Energy mean over steps and band sum in dB (bb_core.cu:563-583); the component sums
// of the clipped energies become the seven levels.  Components of `sums`: TBL pressure,
// suction, separation, LBL, TEB, tip; of BBspl: total, separation, suction, pressure,
// LBL, TEB, tip.
//
// A block holds 32 observers of one band, a warp per component sum (over the splits) and then
// a warp per level; the band's total energy goes to bb_oaspl_kernel as it is.  Large decks
// are bound by the FP64 pipe (a logarithm and a power of ten a level, 113 -> 43 us at 1024
// observers), small ones by the splits' loads, which six warps share (116 -> 28 us at 18).
__global__ void __launch_bounds__(32 * 7) bb_final_kernel(const double* __restrict__ part, int nsplit, int O, int T,
                                                          const float* __restrict__ seed_spl,
                                                          double* __restrict__ spl, float* __restrict__ spl_f,
                                                          double* __restrict__ etot)
{
    __shared__ double s[6][32];
    const int c = threadIdx.y, f = blockIdx.y, o = blockIdx.x * 32 + threadIdx.x;
    if (c < 6 && o < O) {
        const double* p = part + ((size_t)f * 6 + c) * O + o;
        const size_t stride = (size_t)kBands * 6 * O;
        double v = 0.0;
#pragma unroll 8
        for (int k = 0; k < nsplit; ++k) v += p[k * stride];
        s[c][threadIdx.x] = v;
    }
    __syncthreads();
    if (o >= O) return;
    const int x = threadIdx.x;
    // levels in the order total, separation, suction, pressure, LBL, TEB, tip
    const int level = c == 6 ? 0 : (c < 3 ? 3 - c : c + 1);
    const double comp = c == 6 ? s[0][x] + s[1][x] + s[2][x] + s[3][x] + s[4][x] + s[5][x] : s[c][x];
    const size_t i = ((size_t)o * kBands + f) * 7 + level;
    // the -100 dB seed of every (observer, step, band, component) contributes T * 1e-10
    const double seed = seed_spl ? exp10((double)seed_spl[i] * 0.1) : 1e-10;
    const double e = (seed + T * 1e-10 + comp) / (double)T;
    const double db = 10.0 * log10(e);
    if (spl) spl[i] = db;
    if (spl_f) spl_f[i] = (float)db;
    if (c == 6) etot[(size_t)o * kBands + f] = e;
}

// a warp per observer: the OASPL from the bands' total energies (from their levels, a thread
// an observer: 163 us at 1024 observers; now 7)
__global__ void __launch_bounds__(128) bb_oaspl_kernel(int O, const float* __restrict__ seed_oas,
                                                       const double* __restrict__ etot, double* __restrict__ oaspl,
                                                       float* __restrict__ oaspl_f)
{
    const int o = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (o >= O) return;  // warp-uniform
    double v = etot[(size_t)o * kBands + lane] + (lane + 32 < kBands ? etot[(size_t)o * kBands + lane + 32] : 0.0);
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    if (lane != 0) return;
    const double db = 10.0 * log10((seed_oas ? exp10((double)seed_oas[o] * 0.1) : 1e-10) + v);
    if (oaspl) oaspl[o] = db;
    if (oaspl_f) oaspl_f[o] = (float)db;
}

// floats as doubles
__global__ void bb_widen_kernel(const float* __restrict__ in, long long n, double* __restrict__ out)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] = widen_d(in[i]);
}

// ---------------------------------------------------------------- host side

// The surfaces' descriptions with their starts in the concatenated arrays.
struct BBLayout {
    std::vector<BBSurfDev> surf;
    std::vector<int> secsurf, secloc;
    int sec = 0, so = 0, ao = 0, mo = 0, ro = 0;
    long long dofs = 0, tofs = 0;

    // d: span ... nsect and the table's sizes set by the caller; rot in degrees
    template <typename A>
    int add(acum_ctx* ctx, BBSurfDev d, int T, const double* rot, const A* aoa)
    {
        if (d.na_t > kMaxAoa) return fail(ctx, ACUM_ERR_UNSUPPORTED, "broadband tables with more than 64 AoA entries");
        if (d.nsect < 3) return fail(ctx, ACUM_ERR_INVALID, "a broadband surface needs at least 3 sections");
        for (int c = 0; c < 3; ++c) {
            d.crot[c] = cos(rot[c] * M_PI / 180);
            d.srot[c] = sin(rot[c] * M_PI / 180);
        }
        d.a1 = d.a2 = 0;
        for (int k = d.na_t - 1; k >= 0; --k) {
            if (aoa[k] >= 0.0) d.a1 = k;
            if (aoa[k] >= 6.0) d.a2 = k;
        }
        d.sec0 = sec;
        d.data_off = dofs;
        d.sect_off = so;
        d.aoa_off = ao;
        d.mach_off = mo;
        d.re_off = ro;
        d.tab_off = tofs;
        for (int k = 0; k < d.nsect; ++k) {
            secsurf.push_back((int)surf.size());
            secloc.push_back(k);
        }
        surf.push_back(d);
        sec += d.nsect;
        dofs += (long long)T * d.nsect * 7;
        so += d.ns_t;
        ao += d.na_t;
        mo += d.nm_t;
        ro += d.nr_t;
        tofs += (long long)d.ns_t * d.nm_t * d.nr_t * d.na_t * 7;
        return ACUM_OK;
    }
};

static int bpm_upload(acum_ctx* ctx)
{
    BpmState* s = state(ctx);
    const BBDeck& bb = ctx->bb;
    const int nbb = bb.nsurf;
    BBLayout lay;
    for (int i = 0; i < nbb; ++i) {
        BBSurfDev d;
        memset(&d, 0, sizeof(d));
        d.span = bb.span[i];
        d.omega = bb.omega[i];
        d.psi_off = bb.psi_offset[i];
        for (int c = 0; c < 3; ++c) d.tr[c] = bb.translate[3 * i + c];
        d.ccw = bb.ccw[i];
        d.trip = bb.trip[i];
        d.nsect = bb.nsect[i];
        d.ns_t = bb.ns_t[i];
        d.na_t = bb.na_t[i];
        d.nm_t = bb.nm_t[i];
        d.nr_t = bb.nr_t[i];
        int rc = lay.add(ctx, d, ctx->T, &bb.rotate[3 * i], bb.aoa_t.data() + lay.ao);
        if (rc) return rc;
    }
    const std::vector<BBSurfDev>& sd = lay.surf;
    const std::vector<int>&secsurf = lay.secsurf, &secloc = lay.secloc;
    const int sec = lay.sec;
    s->S = sec;
    s->nbb = nbb;
    s->T = ctx->T;
    auto up = [&](DBuf<double>& b, const std::vector<double>& v) -> cudaError_t {
        cudaError_t e = b.ensure(std::max<size_t>(v.size(), 1));
        if (e != cudaSuccess) return e;
        return cudaMemcpy(b.p, v.data(), v.size() * 8, cudaMemcpyHostToDevice);
    };
    cudaError_t e;
    if ((e = s->surf.ensure(nbb)) != cudaSuccess) return cuda_fail(ctx, e, "bpm alloc");
    if ((e = cudaMemcpy(s->surf.p, sd.data(), nbb * sizeof(BBSurfDev), cudaMemcpyHostToDevice)) != cudaSuccess)
        return cuda_fail(ctx, e, "bpm upload");
    if ((e = s->secsurf.ensure(sec)) != cudaSuccess || (e = s->secloc.ensure(sec)) != cudaSuccess)
        return cuda_fail(ctx, e, "bpm alloc");
    cudaMemcpy(s->secsurf.p, secsurf.data(), sec * 4, cudaMemcpyHostToDevice);
    cudaMemcpy(s->secloc.p, secloc.data(), sec * 4, cudaMemcpyHostToDevice);
    if ((e = up(s->geom, bb.geom)) != cudaSuccess || (e = up(s->data, bb.data)) != cudaSuccess ||
        (e = up(s->sect_t, bb.sect_t)) != cudaSuccess || (e = up(s->aoa_t, bb.aoa_t)) != cudaSuccess ||
        (e = up(s->mach_t, bb.mach_t)) != cudaSuccess || (e = up(s->re_t, bb.re_t)) != cudaSuccess ||
        (e = up(s->table, bb.table)) != cudaSuccess)
        return cuda_fail(ctx, e, "bpm upload");
    s->uploaded = true;
    ctx->bb_dirty = false;
    return ACUM_OK;
}

// The kernels of the broadband path on the device arrays of `d` (whose scratch arrays are set
// here).  Seeds (dB) may be null (-100 dB); outputs as doubles or floats (null: left out).
static int bpm_enqueue(acum_ctx* ctx, BBDev& d, int aa_mode, const float* seed_spl, const float* seed_oas, double* spl,
                       double* oas, float* spl_f, float* oas_f)
{
    BpmState* s = state(ctx);
    const int O = ctx->nobs, T = ctx->T;
    const long long nst = (long long)s->S * T;
    cudaStream_t st = ctx->stream;
    cudaError_t e;
    if ((e = s->pos.ensure((size_t)nst * 6)) != cudaSuccess || (e = s->geo.ensure((size_t)nst * kGeo)) != cudaSuccess ||
        (e = s->sc.ensure((size_t)nst * kSc)) != cudaSuccess ||
        (e = s->amp.ensure((size_t)nst * kBands * kAmp)) != cudaSuccess ||
        (e = s->etot.ensure((size_t)O * kBands)) != cudaSuccess)
        return cuda_fail(ctx, e, "bpm alloc");
    if (!s->ff.p) {
        if ((e = s->ff.ensure(kBands)) != cudaSuccess ||
            (e = cudaMemcpy(s->ff.p, kBandHz, kBands * 8, cudaMemcpyHostToDevice)) != cudaSuccess) {
            s->ff.release();
            return cuda_fail(ctx, e, "bpm upload");
        }
    }
    d.pos = s->pos.p;
    d.geo = s->geo.p;
    d.sc = s->sc.p;
    d.S = s->S;
    d.T = T;
    d.dtau = ctx->der.dTau;
    d.i2dtau = 1.0 / (2 * ctx->der.dTau);
    d.a0 = ctx->in.a0;
    for (int c = 0; c < 3; ++c) d.vinf[c] = ctx->der.vinf[c];
    const int nb = (int)((nst + 127) / 128);
    cudaEventRecord(ctx->ev[EV_BPM0], st);
    bb_pos_kernel<<<nb, 128, 0, st>>>(d);
    bb_prep_kernel<<<(unsigned)((nst + 31) / 32), 32, 0, st>>>(d);
    bb_spec_kernel<<<(int)((nst * kBands + 255) / 256), 256, 0, st>>>(s->sc.p, s->ff.p, s->amp.p, nst);
    // item ranges: the number of splits (up to 8 waves of resident blocks) with the
    // smallest wave-quantisation loss; a split costs its blocks' start and its share of
    // bb_final_kernel, 0.4 % (at 1 % the case above ran 16 x 9 blocks on 152 SMs, 3.92 ms, now
    // 16 x 19 in two full waves, 3.68 ms)
    const int oblocks = (O + kObsBlock - 1) / kObsBlock;
    static bool configured = false;
    if (!configured) {
        if ((e = cudaFuncSetAttribute(bb_obs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kObsSmem)) !=
            cudaSuccess)
            return cuda_fail(ctx, e, "bpm configure");
        configured = true;
    }
    if (s->per_sm == 0 && (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&s->per_sm, bb_obs_kernel, kBpmThreads,
                                                                         kObsSmem) != cudaSuccess ||
                           s->per_sm < 1)) {
        (void)cudaGetLastError();
        s->per_sm = 1;
    }
    const int slots = s->per_sm * ctx->num_sms;
    int split = 1;
    double best = 1e30;
    const int maxs = (int)std::max<long long>(1, std::min<long long>((8 * slots + oblocks - 1) / oblocks,
                                                                      (nst + kTI - 1) / kTI));
    for (int k = 1; k <= maxs; ++k) {
        const double waves = (double)oblocks * k / slots;
        const double cost = std::ceil(waves) / waves + 0.004 * k;
        if (cost < best) {
            best = cost;
            split = k;
        }
    }
    const long long per_split = ((nst + split - 1) / split + kTI - 1) / kTI * kTI;
    split = (int)((nst + per_split - 1) / per_split);
    if ((e = s->sums.ensure((size_t)split * kBands * 6 * O)) != cudaSuccess) return cuda_fail(ctx, e, "bpm alloc");
    cudaMemsetAsync(s->sums.p, 0, (size_t)split * kBands * 6 * O * 8, st);
    dim3 grid(oblocks, split);
    cudaEventRecord(ctx->ev[EV_BOBS0], st);
    bb_obs_kernel<<<grid, kBpmThreads, kObsSmem, st>>>(s->geo.p, s->amp.p, ctx->d_obs32.p, O, nst, per_split,
                                                       (float)d.vinf[0], (float)d.vinf[1], (float)d.vinf[2],
                                                       (float)d.a0, aa_mode, s->sums.p, ctx->d_err.p);
    cudaEventRecord(ctx->ev[EV_BOBS1], st);
    bb_final_kernel<<<dim3((O + 31) / 32, kBands), dim3(32, 7), 0, st>>>(s->sums.p, split, O, T, seed_spl, spl, spl_f,
                                                                         s->etot.p);
    bb_oaspl_kernel<<<(O + 3) / 4, 128, 0, st>>>(O, seed_oas, s->etot.p, oas, oas_f);
    cudaEventRecord(ctx->ev[EV_BPM1], st);
    ctx->launches += 6;
    ctx->bpm_timed = true;
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(ctx, e, "bpm launch");
    return ACUM_OK;
}

// waits for the run and reports a device timeout
static int bpm_finish(acum_ctx* ctx)
{
    cudaError_t e;
    if ((e = cudaStreamSynchronize(ctx->stream)) != cudaSuccess) return cuda_fail(ctx, e, "bpm run");
    DeviceErr h;
    if ((e = cudaMemcpy(&h, ctx->d_err.p, sizeof(h), cudaMemcpyDeviceToHost)) != cudaSuccess)
        return cuda_fail(ctx, e, "bpm error word");
    if (h.bits & ACUM_DEVERR_TIMEOUT) {
        cudaMemset(ctx->d_err.p, 0, sizeof(DeviceErr));
        return fail(ctx, ACUM_ERR_TIMEOUT, "a bounded shared-memory pipeline wait ran out; results are incomplete");
    }
    return ACUM_OK;
}

// Runs the broadband path on the context's deck from -100 dB.
static int bpm_run(acum_ctx* ctx, int aa_mode, double* spl_h, double* oas_h)
{
    if (!ctx->have_deck || !ctx->have_bb) return fail(ctx, ACUM_ERR_STATE, "no broadband deck");
    if (aa_mode != 0 && aa_mode != 1) return fail(ctx, ACUM_ERR_INVALID, "aa_mode must be 0 or 1");
    DeviceGuard g(ctx->device);
    BpmState* s = state(ctx);
    if (ctx->bb_dirty || !s->uploaded) {
        int rc = bpm_upload(ctx);
        if (rc) return rc;
    }
    const int O = ctx->nobs;
    cudaError_t e;
    if ((e = s->spl.ensure((size_t)O * kBands * 7)) != cudaSuccess || (e = s->oaspl.ensure(O)) != cudaSuccess)
        return cuda_fail(ctx, e, "bpm alloc");
    BBDev d;
    d.surf = s->surf.p;
    d.secsurf = s->secsurf.p;
    d.secloc = s->secloc.p;
    d.geom = s->geom.p;
    d.data = s->data.p;
    d.sect_t = s->sect_t.p;
    d.aoa_t = s->aoa_t.p;
    d.mach_t = s->mach_t.p;
    d.re_t = s->re_t.p;
    d.table = s->table.p;
    d.t_del = ctx->bb.t_del;
    int rc = bpm_enqueue(ctx, d, aa_mode, nullptr, nullptr, s->spl.p, s->oaspl.p, nullptr, nullptr);
    if (rc) return rc;
    ctx->h_spl.resize((size_t)O * kBands * 7);
    ctx->h_oaspl.resize(O);
    cudaMemcpyAsync(ctx->h_spl.data(), s->spl.p, ctx->h_spl.size() * 8, cudaMemcpyDeviceToHost, ctx->stream);
    cudaMemcpyAsync(ctx->h_oaspl.data(), s->oaspl.p, O * 8, cudaMemcpyDeviceToHost, ctx->stream);
    rc = bpm_finish(ctx);
    if (rc) return rc;
    if (spl_h) memcpy(spl_h, ctx->h_spl.data(), ctx->h_spl.size() * 8);
    if (oas_h) memcpy(oas_h, ctx->h_oaspl.data(), O * 8);
    ctx->have_bpm = true;
    return ACUM_OK;
}

// findBBnoise on the workspaces of `c`: the float arrays go to the device as they are and are
// widened there, the levels come back as floats.
constexpr size_t kKeepBytes = 512ull << 20;

static int bb_noise(acum_ctx* c, BpmState* s, int n, int nObs, int nTime, float dTau, const float* span,
                    const float* omega, const int* ccw, const float* psi_offset, const int* trip, const float* rotate,
                    const float* translate, const int* xsPtr, const int* dsPtr, const int* nsect, const float* xyzcR,
                    const float* bbdata, const int* nsect_t, const int* nmach_t, const int* naoa_t, const int* nre_t,
                    const int* aPtr, const int* mPtr, const int* rPtr, const int* sPtr, const int* dPtr,
                    const float* sect_t, const float* mach_t, const float* aoa_t, const float* re_t,
                    const float* bbdata_t, int t_del, const float* vInf, const float* rObs, float a0, float* BBspl,
                    float* BBoaspl)
{
    c->begin_run();
    c->T = nTime;
    c->nobs = nObs;
    c->in.a0 = a0;
    c->der.dTau = dTau;
    for (int i = 0; i < 3; ++i) c->der.vinf[i] = vInf[i];
    BBLayout lay;
    for (int i = 0; i < n; ++i) {
        BBSurfDev d;
        memset(&d, 0, sizeof(d));
        d.span = span[i];
        d.omega = omega[i];
        d.psi_off = psi_offset[i];
        double rot[3];
        for (int k = 0; k < 3; ++k) {
            rot[k] = rotate[3 * i + k];
            d.tr[k] = translate[3 * i + k];
        }
        d.ccw = ccw[i];
        d.trip = trip[i];
        d.nsect = nsect[i];
        d.ns_t = nsect_t[i];
        d.na_t = naoa_t[i];
        d.nm_t = nmach_t[i];
        d.nr_t = nre_t[i];
        int rc = lay.add(c, d, nTime, rot, aoa_t + aPtr[i]);
        if (rc) return rc;
    }
    s->S = lay.sec;
    s->nbb = n;
    s->T = nTime;
    s->uploaded = false;  // the context's own deck, if it had one, is not what the state holds
    // one block of bytes: the descriptions, the section tables, then the small float arrays
    // (geometry, the tables' axes, the tables); the section data follow on the device
    const size_t surf_b = lay.surf.size() * sizeof(BBSurfDev), sec_b = (size_t)lay.sec * 4;
    const size_t o_geom = 0, o_sect = o_geom + 4 * (size_t)lay.sec, o_aoa = o_sect + lay.so, o_mach = o_aoa + lay.ao,
                 o_re = o_mach + lay.mo, o_tab = o_re + lay.ro, o_data = o_tab + (size_t)lay.tofs,
                 nfl = o_data + (size_t)lay.dofs;
    const size_t fl_off = surf_b + 2 * sec_b;
    s->h_blob.resize(fl_off + o_data * 4);
    unsigned char* h = s->h_blob.data();
    memcpy(h, lay.surf.data(), surf_b);
    memcpy(h + surf_b, lay.secsurf.data(), sec_b);
    memcpy(h + surf_b + sec_b, lay.secloc.data(), sec_b);
    float* f = reinterpret_cast<float*>(h + fl_off);
    const auto put = [](float*& p, const float* src, size_t k) {
        memcpy(p, src, k * 4);
        p += k;
    };
    for (int i = 0; i < n; ++i) put(f, xyzcR + xsPtr[i], 4 * (size_t)nsect[i]);
    for (int i = 0; i < n; ++i) put(f, sect_t + sPtr[i], nsect_t[i]);
    for (int i = 0; i < n; ++i) put(f, aoa_t + aPtr[i], naoa_t[i]);
    for (int i = 0; i < n; ++i) put(f, mach_t + mPtr[i], nmach_t[i]);
    for (int i = 0; i < n; ++i) put(f, re_t + rPtr[i], nre_t[i]);
    for (int i = 0; i < n; ++i)
        put(f, bbdata_t + dPtr[i], (size_t)nsect_t[i] * naoa_t[i] * nmach_t[i] * nre_t[i] * 7);
    cudaStream_t st = c->stream;
    const size_t nspl = (size_t)nObs * kBands * 7;
    cudaError_t e;
    if ((e = s->blob.ensure(fl_off)) != cudaSuccess || (e = s->fl.ensure(nfl)) != cudaSuccess ||
        (e = s->wide.ensure(nfl)) != cudaSuccess || (e = s->seed_f.ensure(nspl + nObs)) != cudaSuccess ||
        (e = s->out_f.ensure(nspl + nObs)) != cudaSuccess || (e = c->d_obs32.ensure(3 * (size_t)nObs)) != cudaSuccess)
        return cuda_fail(c, e, "bpm alloc");
    const auto in = [&](void* dst, const void* src, size_t bytes) {
        if (e == cudaSuccess) e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
    };
    in(s->blob.p, h, fl_off);
    in(s->fl.p, h + fl_off, o_data * 4);
    for (int i = 0; i < n;) {  // (cn, cc arrive already divided); neighbouring arrays in one copy
        size_t k = 0;
        const int i0 = i;
        do k += (size_t)nTime * nsect[i++] * 7;
        while (i < n && (size_t)dsPtr[i] == dsPtr[i0] + k);
        in(s->fl.p + o_data + (size_t)lay.surf[i0].data_off, bbdata + dsPtr[i0], k * 4);
    }
    in(c->d_obs32.p, rObs, 3 * (size_t)nObs * 4);
    in(s->seed_f.p, BBspl, nspl * 4);
    in(s->seed_f.p + nspl, BBoaspl, (size_t)nObs * 4);
    if (e != cudaSuccess) return cuda_fail(c, e, "bpm upload");
    bb_widen_kernel<<<(unsigned)std::min<size_t>((nfl + 255) / 256, 4096), 256, 0, st>>>(s->fl.p, (long long)nfl,
                                                                                       s->wide.p);
    BBDev d;
    d.surf = reinterpret_cast<const BBSurfDev*>(s->blob.p);
    d.secsurf = reinterpret_cast<const int*>(s->blob.p + surf_b);
    d.secloc = reinterpret_cast<const int*>(s->blob.p + surf_b + sec_b);
    d.geom = s->wide.p + o_geom;
    d.sect_t = s->wide.p + o_sect;
    d.aoa_t = s->wide.p + o_aoa;
    d.mach_t = s->wide.p + o_mach;
    d.re_t = s->wide.p + o_re;
    d.table = s->wide.p + o_tab;
    d.data = s->wide.p + o_data;
    d.t_del = t_del;
    int rc = bpm_enqueue(c, d, 0, s->seed_f.p, s->seed_f.p + nspl, nullptr, nullptr, s->out_f.p, s->out_f.p + nspl);
    if (rc == ACUM_OK) rc = bpm_finish(c);
    if (rc) return rc;
    if ((e = cudaMemcpy(BBspl, s->out_f.p, nspl * 4, cudaMemcpyDeviceToHost)) != cudaSuccess ||
        (e = cudaMemcpy(BBoaspl, s->out_f.p + nspl, (size_t)nObs * 4, cudaMemcpyDeviceToHost)) != cudaSuccess)
        return cuda_fail(c, e, "bpm results");
    return ACUM_OK;
}

}  // namespace acum

using namespace acum;

extern "C" int acum_set_bb(acum_ctx* ctx, const acum_bb_desc* b)
{
    acum::NvtxRange nvtx_range_("acum_set_bb");
    if (!ctx || !b) return fail(ctx, ACUM_ERR_INVALID, "acum_set_bb: null argument");
    if (!ctx->have_deck) return fail(ctx, ACUM_ERR_STATE, "acum_set_bb: set the tonal deck first");
    if (b->nsurf <= 0 || b->nsurf > ctx->nsurf)
        return fail(ctx, ACUM_ERR_INVALID,
                    "Number of surfaces considered for broadband noise cannot be higher than the available surfaces");
    BBDeck bb;
    const int n = b->nsurf, T = ctx->T;
    bb.nsurf = n;
    bb.t_del = b->t_del;
    bb.span.assign(b->span, b->span + n);
    bb.omega.assign(b->omega, b->omega + n);
    bb.psi_offset.assign(b->psi_offset, b->psi_offset + n);
    bb.rotate.assign(b->rotate, b->rotate + 3 * n);
    bb.translate.assign(b->translate, b->translate + 3 * n);
    bb.ccw.assign(b->ccw, b->ccw + n);
    bb.trip.assign(b->trip, b->trip + n);
    bb.nsect.assign(b->nsect, b->nsect + n);
    size_t ns = 0, nt = 0, na = 0, nm = 0, nr = 0, ntab = 0;
    for (int i = 0; i < n; ++i) {
        if (b->nsect[i] < 3) return fail(ctx, ACUM_ERR_INVALID, "a broadband surface needs at least 3 sections");
        ns += b->nsect[i];
        nt += b->ns_t[i];
        na += b->na_t[i];
        nm += b->nm_t[i];
        nr += b->nr_t[i];
        ntab += (size_t)b->ns_t[i] * b->na_t[i] * b->nm_t[i] * b->nr_t[i] * 7;
    }
    bb.geom.assign(b->geom, b->geom + 4 * ns);
    bb.data.assign(b->data, b->data + (size_t)T * ns * 7);
    // cn, cc divided by (r/R)^2 for rotating surfaces, as read_BB_inputs does (io.cu:509-512)
    size_t so = 0, dof = 0;
    for (int i = 0; i < n; ++i) {
        if ((float)bb.omega[i] != 0.0f)
            for (int t = 0; t < T; ++t)
                for (int k = 0; k < b->nsect[i]; ++k) {
                    const double rr = bb.geom[4 * (so + k)];
                    bb.data[dof + ((size_t)t * b->nsect[i] + k) * 7 + 4] /= rr * rr;
                    bb.data[dof + ((size_t)t * b->nsect[i] + k) * 7 + 5] /= rr * rr;
                }
        so += b->nsect[i];
        dof += (size_t)T * b->nsect[i] * 7;
    }
    bb.ns_t.assign(b->ns_t, b->ns_t + n);
    bb.na_t.assign(b->na_t, b->na_t + n);
    bb.nm_t.assign(b->nm_t, b->nm_t + n);
    bb.nr_t.assign(b->nr_t, b->nr_t + n);
    bb.sect_t.assign(b->sect_t, b->sect_t + nt);
    bb.aoa_t.assign(b->aoa_t, b->aoa_t + na);
    bb.mach_t.assign(b->mach_t, b->mach_t + nm);
    bb.re_t.assign(b->re_t, b->re_t + nr);
    bb.table.assign(b->table, b->table + ntab);
    ctx->bb = std::move(bb);
    ctx->have_bb = true;
    ctx->bb_dirty = true;
    return ACUM_OK;
}

extern "C" int acum_bpm(acum_ctx* ctx, int aa_mode, double* BBspl, double* BBoaspl)
{
    acum::NvtxRange nvtx_range_("acum_bpm");
    if (!ctx) return ACUM_ERR_INVALID;
    ctx->begin_run();
    return bpm_run(ctx, aa_mode, BBspl, BBoaspl);
}

extern "C" int acum_find_bb_noise(int nSurf_BB, int nObs, int nTime, float dTau, const float* span, const float* omega,
                                  const int* ccw, const float* psi_offset, const int* trip, const float* rotate,
                                  const float* translate, const int* xsPtr, const int* dsPtr, const int* nsect,
                                  const float* xyzcR, const float* bbdata, const int* nsect_t, const int* nmach_t,
                                  const int* naoa_t, const int* nre_t, const int* aPtr, const int* mPtr,
                                  const int* rPtr, const int* sPtr, const int* dPtr, const float* sect_t,
                                  const float* mach_t, const float* aoa_t, const float* re_t, const float* bbdata_t,
                                  int t_del, const float* vInf, const float* rObs, const float* tObs, int nf2,
                                  const float* ff, float a0, float* BBspl, float* BBoaspl)
{
    acum::NvtxRange nvtx_range_("acum_find_bb_noise");
    (void)tObs;
    if (nSurf_BB <= 0 || nObs <= 0 || nTime < 6 || !span || !omega || !ccw || !psi_offset || !trip || !rotate ||
        !translate || !xsPtr || !dsPtr || !nsect || !xyzcR || !bbdata || !nsect_t || !nmach_t || !naoa_t || !nre_t ||
        !aPtr || !mPtr || !rPtr || !sPtr || !dPtr || !sect_t || !mach_t || !aoa_t || !re_t || !bbdata_t || !vInf ||
        !rObs || !ff || !BBspl || !BBoaspl)
        return fail(nullptr, ACUM_ERR_INVALID, "findBBnoise: bad argument");
    if (nf2 != kBands) return fail(nullptr, ACUM_ERR_UNSUPPORTED, "findBBnoise: the band table must have 42 bands");
    for (int i = 0; i < kBands; ++i)
        if (fabs((double)ff[i] - kBandHz[i]) > 1e-6 * kBandHz[i])
            return fail(nullptr, ACUM_ERR_UNSUPPORTED, "findBBnoise: the band table must be the 1/3-octave table");
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_fail(nullptr, e, "cudaGetDevice");
    Dropin* dr = dropin_for(dev, kDropinBroadband);
    if (!dr) return fail(nullptr, ACUM_ERR_CUDA, "findBBnoise: cannot create a context");
    DropinLock lock(dr);
    acum_ctx* c = dr->c;
    DeviceGuard g(dev);
    BpmState* s = state(c);
    InFlight flight(c->stream);
    const int rc = bb_noise(c, s, nSurf_BB, nObs, nTime, dTau, span, omega, ccw, psi_offset, trip, rotate, translate,
                            xsPtr, dsPtr, nsect, xyzcR, bbdata, nsect_t, nmach_t, naoa_t, nre_t, aPtr, mPtr, rPtr, sPtr,
                            dPtr, sect_t, mach_t, aoa_t, re_t, bbdata_t, t_del, vInf, rObs, a0, BBspl, BBoaspl);
    if (rc == ACUM_OK) flight.on = false;  // it has waited
    else flight.wait();
    // the workspaces stay for the next call unless they are large
    if (s->bytes() > kKeepBytes) release_bpm_state(c);
    return rc;
}
