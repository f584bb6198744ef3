// Filament stretching + bending energies of one network that already sits in
// caller-owned device memory, computed without allocating anything.
//
// This is the FP64 filament-energy kernel (FilamentStretchingHarmonic.cpp:185-275
// and FilamentBendingCosine.cpp:199-345, paths relative to medyan-5.4.0/src)
// in a stateless form: the per-block partial sums and the completion ticket
// live in a fixed file-scope device array instead of context buffers, so the
// call makes no cudaMalloc/cudaFree (which can synchronize the whole device)
// and needs no context.
//
// Scratch layout (kStaticScratchBytes):
//   [0, 256)                      completion ticket (one unsigned int); must be
//                                 zero when the kernel starts: the entry point
//                                 clears it on the caller's stream before each
//                                 launch and the last block leaves it at zero
//   [256, 256 + 16 * kStaticGrid) per-block (stretching, bending) partial sums
// Calls that overlap in time (different streams or host threads, same
// device) share this scratch and race; the caller orders them.
#include <cuda_runtime.h>

#include <mutex>
#include <algorithm>
#include <string>

#include "mech_device.cuh"
#include "mech_internal.cuh"

namespace mech {

constexpr int kStaticBlock = 256;
// Two blocks on each SM: four warps on a sub-partition keep its FP64 pipe busy,
// and more of them only shorten the shares (1M cylinders with 1, 2, 3, 4, 8
// blocks: 84.8, 75.8, 77.9, 80.7, 88.2 us).
constexpr int kStaticGrid = 2 * 152;
// A limit of the interface, named for the scratch of a slot per 256 cylinders that
// it once was: the shares of a fixed grid need no more for more cylinders.
constexpr long long kStaticMaxCylinders = 2097152;
constexpr size_t kStaticScratchBytes = 256 + 16 * (size_t)kStaticGrid;   // 5,120 bytes
constexpr int kStaticMaxDevices = 64;

static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

// Filament of cylinder c: the largest f with fcs[f] <= c (fcs ascending).  All
// lanes of a warp search together, 32 ranges a step: 20,000 filaments take three
// dependent loads.
__device__ __forceinline__ int filament_of(const int32_t* __restrict__ fcs, int nfil, int c) {
    int lo = 0, hi = nfil;   // fcs[lo] <= c < fcs[hi]
    while (hi - lo > 1) {
        const int step = (hi - lo + 31) >> 5, probe = lo + ((int)(threadIdx.x & 31) + 1) * step;
        const bool le = probe < hi && __ldg(fcs + probe) <= c;
        lo += step * __popc(__ballot_sync(0xffffffffu, le));
        hi = min(hi, lo + step);
    }
    return lo;
}

// the same for one lane's cylinder
__device__ __forceinline__ int filament_of_lane(const int32_t* __restrict__ fcs, int nfil, int c) {
    int lo = 0, hi = nfil;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(fcs + mid) <= c) lo = mid;
        else hi = mid;
    }
    return lo;
}

// A cylinder per lane: its stretching term and, unless it is the first cylinder
// of its filament, the bending term of the triple it closes (constants of the
// second cylinder).  Beads are filament-contiguous, so cylinder c of filament f
// joins beads c + f and c + f + 1.  Bound by the FP64 pipe, so a cylinder's
// vector and length are formed once and passed on to the next lane for the
// triple, and every warp walks an equal share of the 32-cylinder chunks, a
// contiguous one: the cylinder before it is formed once per share, the terms are
// summed in the lanes and the trees run once, and no barrier holds a warp back.
// The filament is searched for once per share, then followed: the next starts
// are read together and marked in a word.
// 1M cylinders: 75.8 us (a chunk per warp, with barriers between the steps: 93.6).
__global__ void __launch_bounds__(kStaticBlock)
k_fil_energy_static(const double* __restrict__ x, const int32_t* __restrict__ fcs, int nfil, int ncyl,
                    const double* __restrict__ ks, const double* __restrict__ l0, const double* __restrict__ kb,
                    const double* __restrict__ t0, unsigned char* scratch, double* out) {
    static_assert(kStaticBlock == kBlock, "block_sums");
    __shared__ double sh[2 * kBlock / 32];
    __shared__ int s_last;
    constexpr unsigned kAll = 0xffffffffu;
    unsigned int* ticket = reinterpret_cast<unsigned int*>(scratch);
    double2* part = reinterpret_cast<double2*>(scratch + 256);
    const int lane = threadIdx.x & 31;
    const long long chunks = ((long long)ncyl + 31) >> 5, warp = blockIdx.x * (kStaticBlock / 32) + (threadIdx.x >> 5),
                    warps = (long long)gridDim.x * (kStaticBlock / 32);
    int k = (int)(chunks * warp / warps);
    const int k1 = (int)(chunks * (warp + 1) / warps);
    double e[2] = {0.0, 0.0}, rp[3] = {0, 0, 0}, Lp = 0.0;   // rp, Lp: the cylinder before the chunk
    int fp = -1;                                             // and its filament
    if (k > 0 && k < k1) {
        fp = filament_of(fcs, nfil, 32 * k - 1);
        const double* p = x + 3 * ((size_t)(32 * k - 1) + (size_t)fp);
#pragma unroll
        for (int q = 0; q < 3; ++q) rp[q] = p[3 + q] - p[q];
        Lp = sqrt(rp[0] * rp[0] + rp[1] * rp[1] + rp[2] * rp[2]);
    }
    for (; k < k1; ++k) {
        const int c0 = 32 * k, c = c0 + lane, g = fp + 1 + lane;
        const int s = g < nfil ? __ldg(fcs + g) - c0 : 32;   // the next filaments' first cylinders, ascending from 0
        const unsigned starts = __reduce_or_sync(kAll, s < 32 ? 1u << s : 0u);
        // a start equal to the next one read, or (32 starts in the chunk) to the one behind them
        const int before = __shfl_up_sync(kAll, s, 1);
        const bool twice = s < 32 && ((lane > 0 && s == before) || (lane == 31 && __ldg(fcs + g + 1) - c0 == s));
        const bool valid = c < ncyl;
        int f;
        bool first;
        if (!__any_sync(kAll, twice)) {
            f = fp + __popc(starts & (kAll >> (31 - lane)));
            first = starts >> lane & 1;
            fp += __popc(starts);
        } else {   // filaments without cylinders among them
            f = filament_of_lane(fcs, nfil, min(c, ncyl - 1));
            first = __ldg(fcs + f) == c;
            fp = __shfl_sync(kAll, f, 31);
        }
        double r[3] = {0, 0, 0}, L = 0.0;
        if (valid) {
            const double* p = x + 3 * ((size_t)c + (size_t)f);
#pragma unroll
            for (int q = 0; q < 3; ++q) r[q] = p[3 + q] - p[q];
            L = sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
            const double dl = L - l0[c];
            e[0] += 0.5 * ks[c] * dl * dl;
        }
        double r1[3], L1 = __shfl_up_sync(kAll, L, 1);
#pragma unroll
        for (int q = 0; q < 3; ++q) r1[q] = __shfl_up_sync(kAll, r[q], 1);
        if (lane == 0) {
            L1 = Lp;
#pragma unroll
            for (int q = 0; q < 3; ++q) r1[q] = rp[q];
        }
        if (valid && !first)
            e[1] += bend_energy_lengths(r1[0] * r[0] + r1[1] * r[1] + r1[2] * r[2], L1, L, kb[c], t0[c]);
        Lp = __shfl_sync(kAll, L, 31);
#pragma unroll
        for (int q = 0; q < 3; ++q) rp[q] = __shfl_sync(kAll, r[q], 31);
    }
    const double a = block_sums<2>(e, sh);
    const double b = __shfl_sync(kAll, a, 1);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = make_double2(a, b);
        __threadfence();
        s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    // last block: slots in a fixed order (thread t takes t, t + 256, ...), then the block tree
    __threadfence();
    double t[2] = {0.0, 0.0};
    for (int q = threadIdx.x; q < (int)gridDim.x; q += blockDim.x) {
        const double2 v = __ldcg(part + q);
        t[0] += v.x;
        t[1] += v.y;
    }
    const double sum = block_sums<2>(t, sh);
    if (threadIdx.x < 2) out[threadIdx.x] = sum;
    if (threadIdx.x == 0) *ticket = 0u;
}

// The scratch address belongs to the module loaded into one CUDA context: a
// context that is destroyed and re-created (cudaDeviceReset, a primary
// context released by every user) reloads the module and the array can move.
// So the address is cached per (device, current context) and looked up again
// whenever the current context of that device changes.  The context handle
// comes from the driver's cuCtxGetCurrent, reached through the runtime's
// entry-point query so that the library needs no link against libcuda.
using CtxGetCurrentFn = int (*)(void**);   // CUresult cuCtxGetCurrent(CUcontext*)

static std::mutex g_static_mu;
static void* g_static_ptr[kStaticMaxDevices];
static void* g_static_ctx[kStaticMaxDevices];
static CtxGetCurrentFn g_ctx_get_current = nullptr;
static bool g_ctx_query_done = false;

static void* current_context() {
    if (!g_ctx_query_done) {
        g_ctx_query_done = true;
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &fn, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            g_ctx_get_current = reinterpret_cast<CtxGetCurrentFn>(fn);
        else
            cudaGetLastError();
    }
    void* ctx = nullptr;
    if (!g_ctx_get_current || g_ctx_get_current(&ctx) != 0) return nullptr;
    return ctx;
}

// Device address of the scratch array in the current context of device
// `dev` (which must be current), looked up at the first call in that context.
static int static_scratch(int dev, unsigned char** out) {
    if (dev < 0 || dev >= kStaticMaxDevices) return set_error_text(MECH_ERR_ARG, "device ordinal out of range");
    std::lock_guard<std::mutex> lk(g_static_mu);
    void* ctx = current_context();
    if (!g_static_ptr[dev] || !ctx || ctx != g_static_ctx[dev]) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_static_scratch);
        if (e != cudaSuccess || !p)
            return set_error_text(MECH_ERR_CUDA, std::string("cudaGetSymbolAddress(scratch): ") + cudaGetErrorString(e));
        g_static_ptr[dev] = p;
        g_static_ctx[dev] = current_context();   // the lookup itself makes the primary context current
    }
    *out = static_cast<unsigned char*>(g_static_ptr[dev]);
    return MECH_OK;
}

}  // namespace mech

extern "C" int32_t mech_filament_energy_device(int32_t n_filaments, int32_t n_cylinders, const int32_t* fil_cyl_start,
                                               const double* coord, const double* k_stretch, const double* eq_length,
                                               const double* k_bend, const double* eq_theta, double* energies,
                                               void* stream) {
    using namespace mech;
    if (n_filaments < 1 || n_cylinders < 0 || !fil_cyl_start || !coord || !k_stretch || !eq_length || !k_bend ||
        !eq_theta || !energies)
        return set_error_text(MECH_ERR_ARG, "mech_filament_energy_device: null pointer or bad count");
    const long long blocks = ((long long)n_cylinders + kStaticBlock - 1) / kStaticBlock;
    if (n_cylinders > kStaticMaxCylinders)
        return set_error_text(MECH_ERR_CAPACITY,
                              "mech_filament_energy_device: n_cylinders " + std::to_string(n_cylinders) +
                                  " exceeds the fixed scratch limit of " + std::to_string(kStaticMaxCylinders) +
                                  " cylinders");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        return set_error_text(MECH_ERR_NO_DEVICE, "no CUDA device visible");
    }
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return set_error_text(MECH_ERR_CUDA, std::string("cudaGetDevice: ") + cudaGetErrorString(e));
    unsigned char* scratch = nullptr;
    int rc = static_scratch(dev, &scratch);
    if (rc != MECH_OK) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (n_cylinders == 0) {
        e = cudaMemsetAsync(energies, 0, 2 * sizeof(double), s);
        if (e != cudaSuccess) return set_error_text(MECH_ERR_CUDA, std::string("cudaMemsetAsync: ") + cudaGetErrorString(e));
        return MECH_OK;
    }
    e = cudaMemsetAsync(scratch, 0, sizeof(unsigned int), s);
    if (e != cudaSuccess) return set_error_text(MECH_ERR_CUDA, std::string("cudaMemsetAsync: ") + cudaGetErrorString(e));
    const unsigned grid = (unsigned)std::min<long long>(blocks, kStaticGrid);
    k_fil_energy_static<<<grid, kStaticBlock, 0, s>>>(coord, fil_cyl_start, n_filaments, n_cylinders,
                                                                  k_stretch, eq_length, k_bend, eq_theta, scratch,
                                                                  energies);
    e = cudaGetLastError();
    if (e != cudaSuccess) return set_error_text(MECH_ERR_CUDA, std::string("k_fil_energy_static: ") + cudaGetErrorString(e));
    return MECH_OK;
}
