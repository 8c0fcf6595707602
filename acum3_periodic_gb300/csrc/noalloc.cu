// noalloc.cu -- acum_find_pressure_time_history_noalloc: the reference-shaped tonal
// drop-in for callers that must not allocate device memory.
//
// Who needs it: a solver or plugin host that has handed all device memory to its own pool
// allocator and forbids its components to allocate outside it (a cudaMalloc there fails
// for lack of memory or escapes the host's accounting), and a latency-bound loop that
// cannot afford cudaMalloc/cudaFree, which synchronise the whole device and so stall the
// loop's other streams.  Such a caller still owns and passes its inputs and outputs; what
// the computation needs besides them (the tiled per-step records, the FP64 bin sums and
// the device error word) lives here in one fixed array of device memory that every GPU
// loading this library reserves until process exit.
//
// Limits and behaviour:
//  * the scratch array is kNoAllocBytes = 128 MiB per device, and 4 MiB for the anchors of
//    the observers of one pass; a call whose records
//    (64 bytes per element and record slot: elements rounded up to 8, ceil(nTime / 31)
//    windows of 32 slots) plus FP64 bin sums (16 bytes per observer-step) exceed it is
//    rejected with ACUM_ERR_INVALID and a message that gives both sizes; at most
//    kMaxSurfaces surfaces;
//  * it accepts the inputs the allocating drop-in accepts (nTime >= 4, tObs[t] = t * dPsi
//    within the same tolerance) and refuses the others with the same status;
//  * the first call on a device looks up the array's device address (cudaGetSymbolAddress)
//    with that device current; make that first call before any stream capture;
//  * every call that launched anything synchronises `stream` before it returns, whatever it
//    returns: the summary of E, vInf, tObs and the observers and, after the kernels, the device
//    error word go to variables of the call itself;
//  * every call reuses the same array and leaves its contents behind; the call clears
//    what must start at zero itself, and two calls whose GPU work overlaps (different
//    streams or threads without ordering) race on the array -- serialise them;
//  * no cudaMalloc/cudaFree, no host heap allocation.
#include <cuda_runtime.h>
#include <stdio.h>
#include <math.h>
#include <string.h>

#include <mutex>

#include "acum_internal.h"
#include "ctx.h"

namespace acum {

constexpr size_t kNoAllocBytes = 128ull << 20;
// the observers' anchors, after the 128 MiB: more observers go in passes of this many
constexpr int kAnchorsMax = 131072;
constexpr int kMaxSurfaces = 256;
constexpr int kMaxDevices = 64;

// the scratch: tiled records first, then the [obs][step][2] FP64 bin sums
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes + kAnchorsMax * sizeof(Anchor)];

static std::mutex g_na_mu;
static void* g_na_ptr[kMaxDevices];
// the last message of this thread (no lock, no heap)
static thread_local char g_na_msg[256];

}  // namespace acum

using namespace acum;

extern "C" const char* acum_noalloc_last_error(void) { return g_na_msg; }

extern "C" int acum_find_pressure_time_history_noalloc(const float* rObs, const float* tObs, float* pT, float* pL,
                                                       float* pA, const float* Xham, const float* Nham,
                                                       const float* Vham, const float* PRham, int nSurf,
                                                       const int* XPtr, const int* NPtr, const int* VPtr,
                                                       const int* PRPtr, const int* E, int nObs, int nTime,
                                                       float dPsi, float dTau, float a0, float rhoRef,
                                                       const float* vInf, float oM, void* stream)
{
    acum::NvtxRange nvtx_range_("acum_find_pressure_time_history_noalloc");
    auto bad = [](int code, const char* m) {
        snprintf(g_na_msg, sizeof g_na_msg, "%s", m);
        return code;
    };
    if (!rObs || !tObs || !pT || !pL || !pA || !Xham || !Nham || !Vham || !PRham || !XPtr || !NPtr || !VPtr ||
        !PRPtr || !E || !vInf)
        return bad(ACUM_ERR_INVALID, "findPressureTimeHistory_noalloc: null argument");
    if (nSurf <= 0 || nSurf > kMaxSurfaces || nObs <= 0 || nTime < 4)
        return bad(ACUM_ERR_INVALID, "findPressureTimeHistory_noalloc: sizes (1..256 surfaces, nTime >= 4)");
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices)
        return bad(ACUM_ERR_CUDA, "findPressureTimeHistory_noalloc: no current device");
    void* scratch = nullptr;
    {
        // set-up once per device, with that device current
        std::lock_guard<std::mutex> lk(g_na_mu);
        if (!g_na_ptr[dev]) {
            cudaError_t e = cudaGetSymbolAddress(&g_na_ptr[dev], g_noalloc_scratch);
            if (e != cudaSuccess) {
                g_na_ptr[dev] = nullptr;
                snprintf(g_na_msg, sizeof g_na_msg, "cudaGetSymbolAddress: %s", cudaGetErrorString(e));
                return ACUM_ERR_CUDA;
            }
        }
        scratch = g_na_ptr[dev];
    }
    cudaStream_t st = (cudaStream_t)stream;
    (void)cudaGetLastError();  // an earlier call's failure is not this one's
    // what the host needs of the device arrays in one read (through the start of the scratch);
    // the kernel bins on the uniform grid main.cu:124 builds: another tObs is refused, with the
    // tolerance of the allocating drop-in
    // (where the device reads and writes the host's own memory, straight into this frame)
    int host_memory = 0;
    cudaDeviceGetAttribute(&host_memory, cudaDevAttrPageableMemoryAccess, dev);
    DropinFacts facts;
    DeviceErr h;
    InFlight flight(st);  // nothing below returns with the device still writing to the two
    DropinFacts* const to = host_memory ? &facts : (DropinFacts*)scratch;
    if (launch_dropin_facts(false, E, nSurf, vInf, tObs, nTime, dPsi, rObs, nObs, to, st) != cudaSuccess ||
        (!host_memory &&
         cudaMemcpyAsync(&facts, scratch, sizeof(facts), cudaMemcpyDeviceToHost, st) != cudaSuccess) ||
        flight.wait() != cudaSuccess)
        return bad(ACUM_ERR_CUDA, "findPressureTimeHistory_noalloc: reading E/vInf/tObs/rObs failed");
    if (facts.uneven) return bad(ACUM_ERR_UNSUPPORTED, "findPressureTimeHistory_noalloc: tObs must be t*dPsi");
    if (facts.negative) return bad(ACUM_ERR_INVALID, "findPressureTimeHistory_noalloc: negative element count");
    const long long Et = facts.E;
    if (Et <= 0) return bad(ACUM_ERR_INVALID, "findPressureTimeHistory_noalloc: no elements");
    const double obs_rmin = facts.obs_rmin;
    const int nW = (nTime + kWin - 1) / kWin, nW32 = nwin32(nTime);
    const long long Epad = (Et + 7) / 8 * 8;
    const size_t rec_bytes = (size_t)Epad * nW32 * kGroups32 * kWin * 4 * sizeof(float);
    const size_t acc_off = (rec_bytes + 255) / 256 * 256;
    const size_t acc_bytes = (size_t)nObs * nTime * 2 * sizeof(double);
    if (acc_off + acc_bytes > kNoAllocBytes) {
        snprintf(g_na_msg, sizeof g_na_msg,
                 "findPressureTimeHistory_noalloc: needs %zu bytes of scratch (records %zu + sums %zu), the "
                 "maximum is %zu",
                 acc_off + acc_bytes, rec_bytes, acc_bytes, kNoAllocBytes);
        return ACUM_ERR_INVALID;
    }
    float* rec = reinterpret_cast<float*>(scratch);
    double* acc = reinterpret_cast<double*>(reinterpret_cast<unsigned char*>(scratch) + acc_off);
    // the device error word and the records' largest |x| live in the scratch too (after
    // the sums)
    const size_t err_off = (acc_off + acc_bytes + 255) / 256 * 256;
    const size_t err_bytes = (sizeof(DeviceErr) + 15) / 16 * 16 + 16;
    if (err_off + err_bytes > kNoAllocBytes)
        return bad(ACUM_ERR_INVALID, "findPressureTimeHistory_noalloc: no room for the error word");
    DeviceErr* derr = reinterpret_cast<DeviceErr*>(reinterpret_cast<unsigned char*>(scratch) + err_off);
    unsigned* rmax = reinterpret_cast<unsigned*>(reinterpret_cast<unsigned char*>(derr) + err_bytes - 16);
    int sms = 0, optin = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    TonalRun r;
    memset(&r, 0, sizeof(r));
    r.g.E = (int)Et;
    r.g.Epad = (int)Epad;
    r.g.T = nTime;
    r.g.nW = nW;
    const int pass = nObs < kAnchorsMax ? nObs : kAnchorsMax;
    r.g.O = pass;
    r.g.a0 = a0;
    r.g.rho = rhoRef;
    r.g.oM = oM;
    r.g.dPsi = dPsi;
    r.g.dTau = dTau;
    const double* vi = facts.vinf;
    for (int q = 0; q < 3; ++q) r.g.vinf[q] = vi[q];
    r.g.obs_rmin = obs_rmin;
    r.precision = ACUM_MIXED;
    r.rmax = rmax;
    if (plan_tonal(r, 0, 0, 0, sms, (size_t)optin) != cudaSuccess)
        return bad(ACUM_ERR_UNSUPPORTED, "findPressureTimeHistory_noalloc: no tile shape fits this nTime");
    // the array keeps the previous call's contents: clear the sums, the error word and the
    // radius, which lie behind one another (the records kernel writes every slot)
    flight.on = true;
    if (cudaMemsetAsync(acc, 0, err_off - acc_off + err_bytes, st) != cudaSuccess)
        return bad(ACUM_ERR_CUDA, "findPressureTimeHistory_noalloc: clearing scratch failed");
    AosArgs a;
    memset(&a, 0, sizeof(a));
    a.X = Xham;
    a.N = Nham;
    a.V = Vham;
    a.PR = PRham;
    a.nSurf = nSurf;
    a.Ecnt = E;
    a.XPtr = XPtr;
    a.NPtr = NPtr;
    a.VPtr = VPtr;
    a.PRPtr = PRPtr;
    a.E = (int)Et;
    a.Epad = (int)Epad;
    a.T = nTime;
    a.a0 = a0;
    a.rho = rhoRef;
    a.rec32 = rec;
    a.rmax = rmax;
    Anchor* anc = reinterpret_cast<Anchor*>(reinterpret_cast<unsigned char*>(scratch) + kNoAllocBytes);
    if (launch_aos_records(a, anchor_job(rObs, pass, nTime, a0, vi, oM, dPsi, anc), st) != cudaSuccess)
        return bad(ACUM_ERR_CUDA, "findPressureTimeHistory_noalloc: launch of the records kernel failed");
    r.rec = rec;
    r.anc = anc;
    r.acc = acc;
    r.err = derr;
    cudaError_t le = launch_tonal(r, st);
    for (int o0 = pass; o0 < nObs && le == cudaSuccess; o0 += pass) {
        const int n = nObs - o0 < pass ? nObs - o0 : pass;
        le = launch_anchors(anchor_job(rObs + 3 * (size_t)o0, n, nTime, a0, vi, oM, dPsi, anc), st);
        r.g.O = n;
        r.acc = acc + (size_t)o0 * nTime * 2;
        if (le == cudaSuccess) le = plan_tonal(r, 0, 0, 0, sms, (size_t)optin);
        if (le == cudaSuccess) le = launch_tonal(r, st);
    }
    if (le != cudaSuccess || launch_finalize(acc, nObs, nTime, pT, pL, pA, 2, st, r.err,
                                             host_memory ? (unsigned*)&h.bits : nullptr) != cudaSuccess)
        return bad(ACUM_ERR_CUDA, "findPressureTimeHistory_noalloc: launch failed");
    if ((!host_memory && cudaMemcpyAsync(&h, r.err, sizeof(h), cudaMemcpyDeviceToHost, st) != cudaSuccess) ||
        flight.wait() != cudaSuccess)
        return bad(ACUM_ERR_CUDA, "findPressureTimeHistory_noalloc: kernel failed");
    if (h.bits & ACUM_DEVERR_TIMEOUT) return bad(ACUM_ERR_TIMEOUT, "a bounded shared-memory pipeline wait ran out");
    return ACUM_OK;
}
