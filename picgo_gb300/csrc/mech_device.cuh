// Device helpers shared by the kernel translation units: deterministic block
// reductions, the per-replica finalizers of the CG state machine, and the
// per-interaction force-field math of the filament, linker/motor and boundary
// potentials.
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stddef.h>

#include "mech_internal.cuh"

static_assert(offsetof(mech::CGState, active) == 4 && offsetof(mech::CGState, fbuf) == 12 &&
                  offsetof(mech::CGState, dbuf) == 16 && offsetof(mech::CGState, dual) == 28 &&
                  offsetof(mech::CGState, lambda) == 32 && offsetof(mech::CGState, beta) == 40,
              "lane_state reads the head of CGState as three vectors");

namespace mech {

constexpr int kBlock = 256;
constexpr int kDualSearches = 4;         // see CGState::dual
constexpr double kLambdaTol = 1e-8;      // CGMethod::LAMBDATOL (CGMethod.hpp:98)
constexpr double kLambdaReduce = 0.5;    // CGMethod::LAMBDAREDUCE
constexpr double kBacktrackSlope = 0.4;  // CGMethod::BACKTRACKSLOPE

// ---------------------------------------------------------------------------
// Block reductions with a fixed combination tree (results do not depend on
// scheduling).  All threads of a kBlock block must call them.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}

// Sum over the block; valid in thread 0.
__device__ __forceinline__ double block_sum(double v, double* sh /* >= 32 */) {
    v = warp_sum(v);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) sh[w] = v;
    __syncthreads();
    double r = 0.0;
    if (w == 0) {
        r = (l < (blockDim.x >> 5)) ? sh[l] : 0.0;
        r = warp_sum(r);
    }
    return r;
}
__device__ __forceinline__ double block_max(double v, double* sh) {
    v = warp_max(v);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) sh[w] = v;
    __syncthreads();
    double r = 0.0;
    if (w == 0) {
        r = (l < (blockDim.x >> 5)) ? sh[l] : 0.0;
        r = warp_max(r);
    }
    return r;
}

// Sums of N values (a power of two) over each warp and then the block: the
// first steps of the trees halve the number of values a lane carries, so N
// trees take N + 3 additions (N = 4: 6) where one after another they take 5 N.
// Thread t < N gets value t.  A value's tree has the shape of block_sum's
// whatever its place among the N: same bits, and a tile's sums do not depend on
// the tiles it shares a block with.  `sh` holds N * kBlock / 32 doubles.
template <int N>
__device__ __forceinline__ double block_sums(double (&v)[N], double* sh) {
    const int l = threadIdx.x & 31, w = threadIdx.x >> 5;
    int idx = 0, o = 16;
#pragma unroll
    for (int h = N / 2; h >= 1; h >>= 1, o >>= 1) {
        const bool up = (l & o) != 0;
#pragma unroll
        for (int k = 0; k < h; ++k) {
            const double keep = up ? v[k + h] : v[k], send = up ? v[k] : v[k + h];
            v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
        if (up) idx += h;
    }
#pragma unroll
    for (; o >= 1; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    __syncthreads();
    if ((l & (32 / N - 1)) == 0) sh[w * N + idx] = v[0];
    __syncthreads();
    double a[kBlock / 32] = {};
    if (threadIdx.x < N) {
#pragma unroll
        for (int k = 0; k < kBlock / 32; ++k) a[k] = sh[k * N + threadIdx.x];
#pragma unroll
        for (int h = kBlock / 64; h >= 1; h >>= 1)
#pragma unroll
            for (int k = 0; k < h; ++k) a[k] += a[k + h];
    }
    return a[0];
}
// the same for maxima of N unsigned values
template <int N>
__device__ __forceinline__ unsigned long long block_maxima(unsigned long long (&v)[N], unsigned long long* sh) {
    const int l = threadIdx.x & 31, w = threadIdx.x >> 5;
    int idx = 0, o = 16;
#pragma unroll
    for (int h = N / 2; h >= 1; h >>= 1, o >>= 1) {
        const bool up = (l & o) != 0;
#pragma unroll
        for (int k = 0; k < h; ++k) {
            const unsigned long long keep = up ? v[k + h] : v[k], send = up ? v[k] : v[k + h];
            v[k] = max(keep, __shfl_xor_sync(0xffffffffu, send, o));
        }
        if (up) idx += h;
    }
#pragma unroll
    for (; o >= 1; o >>= 1) v[0] = max(v[0], __shfl_xor_sync(0xffffffffu, v[0], o));
    __syncthreads();
    if ((l & (32 / N - 1)) == 0) sh[w * N + idx] = v[0];
    __syncthreads();
    unsigned long long a = 0;
    if (threadIdx.x < N)
        for (int k = 0; k < kBlock / 32; ++k) a = max(a, sh[k * N + threadIdx.x]);
    return a;
}

// Maximum of part[i * stride + off] for i in [b, e), whole block; result in thread 0.
__device__ __forceinline__ double max_slots(const double* part, int stride, int off, int b, int e, double* sh) {
    double acc = 0.0;
    for (int i = b + threadIdx.x; i < e; i += blockDim.x) acc = fmax(acc, __ldcg(part + (size_t)i * stride + off));
    return block_max(acc, sh);
}

// Ticket: returns true in every thread of the block that finished replica r's
// last tile of this kernel.  Must be called by all threads after the block's
// partials are written.
__device__ __forceinline__ bool last_tile(int* ticket, int r, int ntiles, int* sh_flag) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        const int t = atomicAdd(ticket + r, 1);
        *sh_flag = (t == ntiles - 1);
        if (*sh_flag) ticket[r] = 0;
    }
    __syncthreads();
    const bool last = *sh_flag != 0;
    if (last) __threadfence();
    return last;
}

// ---------------------------------------------------------------------------
// CG state machine pieces (CGMethod.hpp:826-1743), run by one thread.
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool call_limit(const CGState& S) {
    return (S.energyCallLimit != 0 && S.numEnergyCall > S.energyCallLimit) ||
           (S.forceCallLimit != 0 && S.numForceCall > S.forceCallLimit);
}
__device__ __forceinline__ bool converged(const CGState& S) {
    return S.maxF < S.gradTol || S.energyRelChange < S.energyRelTol;
}

// lambda = 0 after a line search (CGMethod.hpp:1337-1367): stop with
// errorLineSearch, enter safe mode, or (already in safe mode) hand MController's
// recovery move to the host.  Applied where the line search fails, so no launch
// of its own has to look for failed replicas.
__device__ __forceinline__ void dispatch_failed(CGState& S) {
    if (!S.tryToRecover) {
        S.errorFlags |= 1u;
        S.status = MECH_ERR_LINESEARCH;
        S.phase = PH_DONE;
    } else if (!S.safeMode) {
        S.safeMode = 1;
        S.numSafeMode++;
        S.phase = PH_RESET;
    } else {
        S.safeMode = 0;
        S.numRecover++;
        S.phase = PH_RECOVER;
    }
}

__device__ __forceinline__ void begin_iteration(CGState& S);
// d = F (resetCGParams, CGMethod.hpp:963-972), as long as the step logic asks
// for it: a search that cannot begin asks once more, in safe mode.
__device__ __forceinline__ void settle(CGState& S) {
    for (int k = 0; k < 2 && S.phase == PH_RESET; ++k) {
        S.dIsF = 1;
        S.dPending = 0;
        S.slope = S.FdotF;
        S.lastFdotF = S.FdotF;
        begin_iteration(S);
    }
}

// Loop head and the start of backtrackingLineSearch (CGMethod.hpp:238-296, :1279-1320).
// The energy at the current coordinates is the cached E0: it is the accepted
// trial's energy, bit for bit, because the trial coordinates x + lambda d are
// the coordinates the move produces.
__device__ __forceinline__ void begin_iteration(CGState& S) {
    if (call_limit(S) || converged(S)) {
        S.phase = PH_DONE;
        return;
    }
    S.numIter++;
    if (S.maxF == 0.0) {     // "return zero if no forces": lambda 0, no energy call
        S.lambda = 0.0;
        S.phase = PH_FAILED;
        dispatch_failed(S);
        return;
    }
    S.lambda = fmin(S.lambdaMax, S.maxDist / S.maxF);
    S.numEnergyCall++;       // the reference evaluates E0 here
    const double armijo = S.safeMode ? 0.0 : kBacktrackSlope;
    S.reducedSlope = armijo * S.slope;
    if (S.searchTrials > 1) S.dual = kDualSearches;
    else if (S.dual > 0) --S.dual;
    S.searchTrials = 0;
    S.phase = PH_LS_TRIAL;
}

// One backtracking step after the trial energy E (CGMethod.hpp:296-361);
// `trial_buf` is the position buffer holding that trial's coordinates.
__device__ __forceinline__ void line_search_step(CGState& S, double E, int trial_buf) {
    S.numEnergyCall++;
    S.numTrials++;
    S.searchTrials++;
    double lambda = S.lambda;
    double Elam = E;
    const double ideal = -S.reducedSlope * lambda;
    bool done = false;
    if (lambda < 0 || ideal > 0) {
        done = true;
        lambda = 0.0;
    }
    const double change = Elam - S.E0;
    if (change <= ideal) done = true;
    else lambda *= kLambdaReduce;
    if (lambda <= 0.0 || lambda <= kLambdaTol) {
        done = true;
        lambda = 0.0;
        Elam = S.E0;
    }
    S.lambda = lambda;
    if (!done) {                       // next trial at the halved lambda
        S.dual = kDualSearches;
        return;
    }
    S.totalEnergy = Elam;
    if (lambda == 0.0) {
        S.phase = PH_FAILED;
        dispatch_failed(S);
        return;
    }
    S.newEnergy = Elam;
    S.E0 = Elam;                       // energy at the moved coordinates
    S.xbuf = trial_buf;                // the trial buffer becomes current
    S.phase = PH_FORCE;
}

// ---------------------------------------------------------------------------
// Bead positions.  FP64 engine: three doubles per bead.  Mixed engine: each
// component is an unevaluated sum hi + lo of two floats (about 48 significant
// bits), so positions, trial moves and difference vectors need no FP64
// arithmetic, which runs at 1/57 of the FP32 rate on this GPU.  Both formats
// take 24 bytes per bead.
// ---------------------------------------------------------------------------
template <typename Real> struct Pos;
template <> struct Pos<double> { double x[3]; };
template <> struct Pos<float> { float h[3], l[3]; };

__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
    s = a + b;
    const float bb = s - a;
    e = (a - (s - bb)) + (b - bb);
}
__device__ __forceinline__ void fast_two_sum(float a, float b, float& s, float& e) {
    s = a + b;
    e = b - (s - a);
}

__device__ __forceinline__ Pos<double> load_pos(const double* X, int b) {
    Pos<double> p;
    const double* q = X + 3 * (size_t)b;
    p.x[0] = q[0]; p.x[1] = q[1]; p.x[2] = q[2];
    return p;
}
__device__ __forceinline__ Pos<float> load_pos(const float* X, int b) {
    Pos<float> p;
    const float2* q = reinterpret_cast<const float2*>(X + 6 * (size_t)b);
    const float2 a = q[0], c = q[1], e = q[2];
    p.h[0] = a.x; p.h[1] = a.y; p.h[2] = c.x; p.l[0] = c.y; p.l[1] = e.x; p.l[2] = e.y;
    return p;
}
__device__ __forceinline__ void store_pos(double* X, int b, const Pos<double>& p) {
    double* q = X + 3 * (size_t)b;
    q[0] = p.x[0]; q[1] = p.x[1]; q[2] = p.x[2];
}
__device__ __forceinline__ void store_pos(float* X, int b, const Pos<float>& p) {
    float2* q = reinterpret_cast<float2*>(X + 6 * (size_t)b);
    q[0] = make_float2(p.h[0], p.h[1]);
    q[1] = make_float2(p.h[2], p.l[0]);
    q[2] = make_float2(p.l[1], p.l[2]);
}

// The search direction as a line-search pass reads it (CGState::dPending): the
// vector at `d`, or F + beta d (CGMethod.hpp:1553-1556) when `F` is set, rounded
// alike in every kernel.
template <typename Real>
struct Direction {
    const Real* d;
    const Real* F;
    Real* out;      // where the filament kernel stores a new direction
    Real beta;
};
// What an evaluation kernel needs of a replica's state, read by every thread
// for itself (three broadcast loads issued together, no barrier).
template <typename Real>
struct LaneState {
    bool go;         // selected by the launch (replica_selected)
    int xb, fb, dbuf, dIsF, dPending, dual;
    double lambda;
    Real lam, beta;
};
template <typename Real>
__device__ __forceinline__ LaneState<Real> lane_state(const DevNet<Real>& n, int r, int want) {
    const int4* q = reinterpret_cast<const int4*>(n.st + r);
    const int4 a = q[0], b = q[1];
    const double2 c = reinterpret_cast<const double2*>(q)[2];
    LaneState<Real> s;
    s.go = want < 0 ? a.y != 0 : a.x == want;
    s.xb = a.z;
    s.fb = a.w;
    s.dbuf = b.x;
    s.dIsF = b.y;
    s.dPending = b.z;
    s.dual = b.w;
    s.lambda = c.x;
    s.lam = (Real)c.x;
    s.beta = (Real)c.y;
    return s;
}
template <typename Real>
__device__ __forceinline__ Direction<Real> direction_of(const DevNet<Real>& n, const LaneState<Real>& S) {
    Direction<Real> D;
    const int fd = S.dPending ? S.fb ^ 1 : S.fb;   // the forces that are the direction
    D.d = S.dIsF ? n.f[fd] : n.d[S.dbuf];
    D.F = S.dPending ? n.f[S.fb] : nullptr;
    D.out = n.d[S.dbuf ^ 1];
    D.beta = S.beta;
    return D;
}
__device__ __forceinline__ float new_direction(float F, float beta, float d) { return fmaf(beta, d, F); }
__device__ __forceinline__ double new_direction(double F, double beta, double d) { return fma(beta, d, F); }
template <typename Real>
__device__ __forceinline__ void direction_at(const Direction<Real>& D, int b, Real v[3]) {
    const Real* d = D.d + 3 * (size_t)b;
    v[0] = d[0]; v[1] = d[1]; v[2] = d[2];
    if (D.F) {
        const Real* F = D.F + 3 * (size_t)b;
#pragma unroll
        for (int k = 0; k < 3; ++k) v[k] = new_direction(F[k], D.beta, v[k]);
    }
}

// x + lambda d (CGMethod.cpp:43-46).  Every kernel that needs the trial
// position uses these, so the materialized trial coordinates and the ones
// formed on the fly are identical.  Mixed engine: the step rounded to single
// precision.
__device__ __forceinline__ Pos<double> moved(const Pos<double>& p, const double d[3], double lam) {
    Pos<double> o;
#pragma unroll
    for (int k = 0; k < 3; ++k) o.x[k] = fma(lam, d[k], p.x[k]);
    return o;
}
__device__ __forceinline__ Pos<float> moved(const Pos<float>& p, const float d[3], float lf) {
    Pos<float> o;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        float s, e, lo;
        two_sum(p.h[k], __fmul_rn(lf, d[k]), s, e);
        lo = __fadd_rn(p.l[k], e);
        fast_two_sum(s, lo, o.h[k], o.l[k]);
    }
    return o;
}

// bead b at x (trial = false) or x + lambda d
template <typename Real>
__device__ __forceinline__ Pos<Real> bead_at(const Real* X, const Direction<Real>& D, int b, bool trial, Real lam) {
    const Pos<Real> p = load_pos(X, b);
    if (!trial) return p;
    Real d[3];
    direction_at(D, b, d);
    return moved(p, d, lam);
}

// compensated single-precision accumulator
struct FF {
    float h = 0.f, l = 0.f;
    __device__ __forceinline__ void add(float v) {
        float s, e;
        two_sum(h, v, s, e);
        const float lo = __fadd_rn(l, e);
        fast_two_sum(s, lo, h, l);
    }
};
// Sums of N compensated pairs (a power of two, at most 32) over a warp: the trees
// packed as in block_sums, N pair additions (and a few) where N trees take 5 N.
// Every lane gets the sum, in a[0], of the pair whose number is returned: lane
// 32 k / N that of one of the N.  No double arithmetic: a warp's FP64 instruction
// holds its sub-partition's FP64 pipe for ~78 cycles on this part, so a per-tile
// double tree costs more than the tile's loads.
__device__ __forceinline__ void add_pairs(FF& a, float h, float l) {
    float t, te;
    two_sum(a.h, h, t, te);
    te = __fadd_rn(te, __fadd_rn(a.l, l));
    fast_two_sum(t, te, a.h, a.l);
}
template <int N>
__device__ __forceinline__ int warp_pair_sums(FF (&a)[N]) {
    const int l = threadIdx.x & 31;
    int idx = 0, o = 16;
#pragma unroll
    for (int h = N / 2; h >= 1; h >>= 1, o >>= 1) {
        const bool up = (l & o) != 0;
#pragma unroll
        for (int k = 0; k < h; ++k) {
            FF keep = up ? a[k + h] : a[k];
            const FF send = up ? a[k] : a[k + h];
            add_pairs(keep, __shfl_xor_sync(0xffffffffu, send.h, o), __shfl_xor_sync(0xffffffffu, send.l, o));
            a[k] = keep;
        }
        if (up) idx += h;
    }
#pragma unroll
    for (; o >= 1; o >>= 1)
        add_pairs(a[0], __shfl_xor_sync(0xffffffffu, a[0].h, o), __shfl_xor_sync(0xffffffffu, a[0].l, o));
    return idx;
}
// The same over the block: lane t < N of warp 0 gets pair t.  `sh` holds
// 2 N kBlock / 32 floats.
template <int N>
__device__ __forceinline__ FF block_pair_sums(FF (&a)[N], float* sh) {
    const int l = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int idx = warp_pair_sums<N>(a);
    if ((l & (32 / N - 1)) == 0) {
        sh[2 * (w * N + idx)] = a[0].h;
        sh[2 * (w * N + idx) + 1] = a[0].l;
    }
    __syncthreads();
    FF r[kBlock / 32];
    if (threadIdx.x < N) {
#pragma unroll
        for (int k = 0; k < kBlock / 32; ++k) {
            r[k].h = sh[2 * (k * N + threadIdx.x)];
            r[k].l = sh[2 * (k * N + threadIdx.x) + 1];
        }
#pragma unroll
        for (int h = kBlock / 64; h >= 1; h >>= 1)
#pragma unroll
            for (int k = 0; k < h; ++k) add_pairs(r[k], r[k + h].h, r[k + h].l);
    }
    return r[0];
}

// Mixed-engine partial slots: a compensated (hi, lo) float pair stored in the
// 8 bytes of a double slot, so partial sums never pass through FP64.
__device__ __forceinline__ void store_pair(double* slot, float h, float l) {
    *reinterpret_cast<float2*>(slot) = make_float2(h, l);
}
__device__ __forceinline__ float2 load_pair(const double* slot) { return __ldcg(reinterpret_cast<const float2*>(slot)); }
__device__ __forceinline__ void add_pair(FF& acc, float2 v) {
    acc.add(v.x);
    acc.add(v.y);
}

// a - b as Real
__device__ __forceinline__ void pdiff(const Pos<double>& a, const Pos<double>& b, double r[3]) {
    r[0] = a.x[0] - b.x[0]; r[1] = a.x[1] - b.x[1]; r[2] = a.x[2] - b.x[2];
}
__device__ __forceinline__ void pdiff(const Pos<float>& a, const Pos<float>& b, float r[3]) {
#pragma unroll
    for (int k = 0; k < 3; ++k) r[k] = __fadd_rn(__fsub_rn(a.h[k], b.h[k]), __fsub_rn(a.l[k], b.l[k]));
}
__device__ __forceinline__ void to_double(const Pos<double>& p, double o[3]) { o[0] = p.x[0]; o[1] = p.x[1]; o[2] = p.x[2]; }
__device__ __forceinline__ void to_double(const Pos<float>& p, double o[3]) {
#pragma unroll
    for (int k = 0; k < 3; ++k) o[k] = (double)p.h[k] + (double)p.l[k];   // exact
}
__device__ __forceinline__ Pos<float> split(const double x[3]) {
    Pos<float> p;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        p.h[k] = (float)x[k];
        p.l[k] = (float)(x[k] - (double)p.h[k]);
    }
    return p;
}

// ---------------------------------------------------------------------------
// Maximum of per-thread values of the engine's precision, in thread 0.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double block_max_r(double v, double* sh) { return block_max(v, sh); }
__device__ __forceinline__ double block_max_r(float v, double* sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_down_sync(0xffffffffu, v, o));
    const int wi = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) sh[wi] = (double)v;
    __syncthreads();
    double r = 0.0;
    if (wi == 0) {
        r = (l < (blockDim.x >> 5)) ? sh[l] : 0.0;
        r = warp_max(r);
    }
    return r;
}

// areEqual(theta0, 0) (utility.h:75-78), in the engine's precision
__device__ __forceinline__ bool near_zero_theta(double t) { return fabs(t - 0.0) < 1e-6; }
__device__ __forceinline__ bool near_zero_theta(float t) { return fabsf(t) < 1e-6f; }

// the four filament constants of a bead slot in one vector load
__device__ __forceinline__ void load_par(const float* P, int j, float& ks, float& l0, float& kb, float& t0) {
    const float4 v = reinterpret_cast<const float4*>(P)[j];
    ks = v.x; l0 = v.y; kb = v.z; t0 = v.w;
}
__device__ __forceinline__ void load_par(const double* P, int j, double& ks, double& l0, double& kb, double& t0) {
    const double2 a = reinterpret_cast<const double2*>(P)[2 * (size_t)j];
    const double2 b = reinterpret_cast<const double2*>(P)[2 * (size_t)j + 1];
    ks = a.x; l0 = a.y; kb = b.x; t0 = b.y;
}

// Comparisons of doubles on their bits, off the FP64 pipe.
__device__ __forceinline__ unsigned long long abs_bits(double x) {
    return (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffULL;
}
// areEqual(theta0, 0) on bits: the order of finite magnitudes is that of their
// bits, and a NaN lies above every threshold
__device__ __forceinline__ bool theta_is_zero(double t) {
    return abs_bits(t) < (unsigned long long)__double_as_longlong(1e-6);
}
// x clamped to [-1, 1], a NaN kept
__device__ __forceinline__ double clamp_unit(double x) {
    const unsigned long long a = abs_bits(x);
    return a > 0x3ff0000000000000ULL && a <= 0x7ff0000000000000ULL ? copysign(1.0, x) : x;
}

// ---------------------------------------------------------------------------
// Filament stretching (FilamentStretchingHarmonic.cpp:185-275) and cosine
// bending (FilamentBendingCosine.cpp:199-345) on difference vectors.
// ---------------------------------------------------------------------------
template <typename Real>
__device__ __forceinline__ Real stretch_energy(Real rx, Real ry, Real rz, Real k, Real l0) {
    const Real L = sqrt(rx * rx + ry * ry + rz * rz);
    const Real dl = L - l0;
    return (Real)0.5 * k * dl * dl;
}

// FP64 bending energy of a triple from its cylinders' r1 . r2 and lengths.
__device__ __forceinline__ double bend_energy_lengths(double l1l2, double L1, double L2, double k, double t0) {
    const double x = clamp_unit(l1l2 / (L1 * L2));
    if (theta_is_zero(t0)) return k * (1.0 - x);
    const double sinA = fmax(sqrt(1.0 - x * x), 0.0);
    return k * (1.0 - (x * cos(t0) + sinA * sin(t0)));
}

// Force on the second bead (the first gets the negation).
template <typename Real>
__device__ __forceinline__ void stretch_force(Real rx, Real ry, Real rz, Real k, Real l0, Real F[3]) {
    const Real L = sqrt(rx * rx + ry * ry + rz * rz);
    const Real invL = (Real)1 / L;
    const Real f0 = k * (L - l0) * invL;
    F[0] = -f0 * rx;
    F[1] = -f0 * ry;
    F[2] = -f0 * rz;
}

template <typename Real>
__device__ __forceinline__ Real bend_energy(const Real r1[3], const Real r2[3], Real k, Real t0) {
    const Real L1sq = r1[0] * r1[0] + r1[1] * r1[1] + r1[2] * r1[2];
    const Real L2sq = r2[0] * r2[0] + r2[1] * r2[1] + r2[2] * r2[2];
    const Real l1l2 = r1[0] * r2[0] + r1[1] * r2[1] + r1[2] * r2[2];
    const Real L1L2 = sqrt(L1sq) * sqrt(L2sq);
    Real x = l1l2 / L1L2;
    if (x < (Real)-1) x = (Real)-1;
    else if (x > (Real)1) x = (Real)1;
    if (near_zero_theta(t0)) {
        if (sizeof(Real) == 4 && l1l2 > (Real)0) {
            // 1 - cos = |r1 x r2|^2 / (L1 L2 (L1 L2 + r1.r2)): no cancellation in single precision
            const Real cx = r1[1] * r2[2] - r1[2] * r2[1];
            const Real cy = r1[2] * r2[0] - r1[0] * r2[2];
            const Real cz = r1[0] * r2[1] - r1[1] * r2[0];
            const Real om = (cx * cx + cy * cy + cz * cz) / (L1L2 * (L1L2 + l1l2));
            return k * om;
        }
        return k * ((Real)1 - x);
    }
    const Real cosA = x;
    const Real sinA = fmax(sqrt((Real)1 - cosA * cosA), (Real)0);
    const Real cAmB = cosA * cos(t0) + sinA * sin(t0);
    return k * ((Real)1 - cAmB);
}

// Fr1, Fr2 of the reference: forces are b1: -Fr1, b2: Fr1 - Fr2, b3: Fr2.
template <typename Real>
__device__ __forceinline__ void bend_force(const Real r1[3], const Real r2[3], Real k, Real t0, Real Fr1[3], Real Fr2[3]) {
    const Real L1sq = r1[0] * r1[0] + r1[1] * r1[1] + r1[2] * r1[2];
    const Real L2sq = r2[0] * r2[0] + r2[1] * r2[1] + r2[2] * r2[2];
    const Real l1l2 = r1[0] * r2[0] + r1[1] * r2[1] + r1[2] * r2[2];
    const Real A = (Real)1 / sqrt(L1sq * L2sq);
    Real x = l1l2 * A;
    const Real B = x / L1sq;
    const Real C = x / L2sq;
    Real kk;
    if (near_zero_theta(t0)) {
        kk = k;
    } else {
        if (fabs(fabs(x) - (Real)1) < (Real)0.001) x = (Real)0.999 * x;
        if (x < (Real)-1) x = (Real)-1;
        else if (x > (Real)1) x = (Real)1;
        const Real sinp = sqrt(fmax((Real)1 - x * x, (Real)0));
        const Real sinpmq = sinp * cos(t0) - x * sin(t0);
        kk = k * sinpmq / sinp;
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        Fr1[q] = kk * (r2[q] * A - r1[q] * B);
        Fr2[q] = kk * (r1[q] * A - r2[q] * C);
    }
}

// ---------------------------------------------------------------------------
// Linker / motor stretching between interpolated points
// (LinkerStretchingHarmonic.cpp:191-293).  p = b1 (1 - s) + s b2.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void lerp3(const double a[3], const double b[3], double s, double out[3]) {
    const double t = 1 - s;
    out[0] = (a[0] * t + s * b[0]);
    out[1] = (a[1] * t + s * b[1]);
    out[2] = (a[2] * t + s * b[2]);
}

// ---------------------------------------------------------------------------
// Plane distance (BoundaryElementImpl.h:49-53): (a x + b y + c z + d) / |n|.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double plane_dist(const double* pl, const double p[3]) {
    return (pl[0] * p[0] + pl[1] * p[1] + pl[2] * p[2] + pl[3]) / sqrt(pl[0] * pl[0] + pl[1] * pl[1] + pl[2] * pl[2]);
}

}  // namespace mech
