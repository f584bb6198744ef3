// Cylinder-cylinder excluded volume: the analytic double integral of 1/r^4
// over two segments (CylinderExclVolRepulsion.cpp:330-882, paths relative to
// medyan-5.4.0/src), with the reference's composite-Simpson fallbacks
// (:884-1254) for pairs whose analytic value is not usable.
//
// This file is compiled once per precision (MECH_EXVOL_REAL = double or
// float).  The FP64 object is built without FMA contraction: the formula is
// ill-conditioned for nearly coplanar pairs, and rounding each operation as
// written keeps the GPU within a few ulps of the CPU restatement there.  In
// mixed precision the pair geometry is single precision, with cancellation-free
// cross-product forms of the invariants; the 1/JJ * (sum) form still loses
// accuracy as the normalized triple product q = |(v12 x v34) . v31| /
// (|v12| |v34| |v31|) goes to zero (nearly coplanar or nearly touching
// segments), so pairs with q under a threshold are evaluated again in FP64 by
// an extended pass over a compacted list (k_exvol_ext, shaped around this
// GPU's FP64 pipe).  The reference's coplanarity move (forces only) is decided
// and applied in single precision, except for pairs whose test lies within
// rounding of its threshold, which go to the extended pass.
#include <cuda_runtime.h>

#include "mech_cg.cuh"
#include "mech_device.cuh"
#include "mech_exvol_math.cuh"

#ifndef MECH_EXVOL_REAL
#define MECH_EXVOL_REAL double
#endif

namespace mech {

constexpr int kFbNodesEnergy = 400;       // Simpson intervals, energy (:929-930)
constexpr int kFbNodesForce = 10000;      // Simpson intervals, forces (:1041-1042)

// FP64 engine: the reference's forms, for parity.
static __device__ double pair_energy_d(const double* c1, const double* c2, const double* c3, const double* c4,
                                       double kRep) {
    double v12[3], v34[3], v31[3], v14[3], v32[3], v24[3];
    diffs_of(c1, c2, c3, c4, v12, v34, v31, v14, v32, v24);
    PairInv<double> p;
    pair_inv(v12, v34, v31, v14, v32, v24, p, false);
    return energy_from(p, kRep);
}


// The reference's coplanarity decision |n . v3| / (|n| |v3|) < 0.1: on the
// squares, without its two roots and six divisions (~75 FP64 instructions),
// unless they lie so near the threshold that its rounding decides (or compare
// with nothing).
static __device__ __forceinline__ bool nearly_coplanar(const double* c1, const double* c2, const double* c3,
                                                       const double* c4) {
    double a[3], b[3], v[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        a[k] = c2[k] - c1[k];
        b[k] = c3[k] - c1[k];
        v[k] = c4[k] - c1[k];
    }
    const double n[3] = {a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]};
    const double nv = dot3(n, v), lhs = nv * nv, rhs = 0.01 * (dot3(n, n) * dot3(v, v)), gap = 1e-10 * rhs;
    if (lhs < rhs - gap) return true;
    if (lhs > rhs + gap) return false;
    return coplanarity<double>(c1, c2, c3, c4) < 0.1;
}

// FP64 forces of a pair at double positions, with the reference's coplanar
// move of c2 (:610-626, force path only).
static __device__ bool pair_forces_d(const double* c1, const double* c2in, const double* c3, const double* c4, double kRep,
                                     double out[4][3]) {
    double moved2[3];
    const double* c2 = c2in;
    if (nearly_coplanar(c1, c2in, c3, c4)) {
        push_c2(c1, c2in, c3, moved2);
        c2 = moved2;
    }
    double v12[3], v34[3], v31[3], v14[3], v32[3], v24[3];
    diffs_of(c1, c2, c3, c4, v12, v34, v31, v14, v32, v24);
    PairInv<double> p;
    pair_inv(v12, v34, v31, v14, v32, v24, p, false);
    return forces_from<false>(p, v12, v34, v31, kRep, out);
}

// ---------------------------------------------------------------------------
// composite-Simpson fallbacks (FP64, whatever the engine precision)
// ---------------------------------------------------------------------------
struct Quad {
    double a, b, c, d, e, F;
};
__device__ __forceinline__ Quad quad_of(const double* c1, const double* c2, const double* c3, const double* c4) {
    Quad q;
    double v12[3], v34[3], v31[3];
    for (int k = 0; k < 3; ++k) { v12[k] = c2[k] - c1[k]; v34[k] = c4[k] - c3[k]; v31[k] = c1[k] - c3[k]; }
    q.a = dot3(v12, v12); q.b = dot3(v34, v34); q.c = dot3(v31, v31);
    q.d = dot3(v12, v34); q.e = dot3(v12, v31); q.F = dot3(v34, v31);
    return q;
}
__device__ __forceinline__ double r2_at(const Quad& q, double s, double t) {
    return q.c + 2 * s * q.e + s * s * q.a - 2 * t * q.F - 2 * s * t * q.d + t * t * q.b;
}
// Node i of N: endpoints 0 and 1; interior nodes at (i+1)/N, the positions
// the reference's loop visits (its node counter is advanced before use).
__device__ __forceinline__ double node(int i, int N) { return i == 0 ? 0.0 : (i == N ? 1.0 : (double)(i + 1) / N); }
__device__ __forceinline__ double weight(int i, int N) { return (i == 0 || i == N) ? 1.0 : ((i & 1) ? 4.0 : 2.0); }

// Simpson energies of the flagged pairs: block `blk` of `nblk` takes entries
// blk, blk + nblk, ...
template <typename Real>
__device__ void fb_energy_blocks(const DevNet<Real>& n, int blk, int nblk, double* sh) {
    const int cnt = min(*n.ev_fb_count, kExvolFallbackCap);
    for (int k = blk; k < cnt; k += nblk) {
        const int pr = n.ev_fb_list[2 * k + 1];
        const int4 bs = n.ev_bead[pr];
        const CGState& S = n.st[n.ev_fb_list[2 * k]];
        // positions of this evaluation: the entry records the trial lambda (0: plain evaluation)
        const double lam = __longlong_as_double(((const long long*)n.ev_fb_energy)[kExvolFallbackCap + k]);
        const bool tr = lam != 0.0;
        const Direction<Real> dir = direction_of(n, lane_state(n, n.ev_fb_list[2 * k], -1));
        double c1[3], c2[3], c3[3], c4[3];
        to_double(bead_at(n.x[S.xbuf], dir, bs.x, tr, (Real)lam), c1);
        to_double(bead_at(n.x[S.xbuf], dir, bs.y, tr, (Real)lam), c2);
        to_double(bead_at(n.x[S.xbuf], dir, bs.z, tr, (Real)lam), c3);
        to_double(bead_at(n.x[S.xbuf], dir, bs.w, tr, (Real)lam), c4);
        const Quad q = quad_of(c1, c2, c3, c4);
        const int N = kFbNodesEnergy;
        double acc = 0.0;
        for (int w = threadIdx.x; w < (N + 1) * (N + 1); w += blockDim.x) {
            const int i = w / (N + 1), j = w % (N + 1);
            const double r2 = r2_at(q, node(i, N), node(j, N));
            acc += weight(i, N) * weight(j, N) * (1.0 / (r2 * r2));
        }
        acc = block_sum(acc, sh);
        if (threadIdx.x == 0) {
            const double kRepScaled = (double)n.ev_k[pr] * (double)n.ev_la[pr] * (double)n.ev_lb[pr];
            const double ds = 1.0 / N;
            const double U = kRepScaled * (ds * ds / 9.0) * acc;
            n.ev_fb_energy[k] = (bad_value(U) || U < -1.0) ? -1.0 : U;
        }
        __syncthreads();
    }
}

// The kernels of the excluded-volume chain follow one another by programmatic
// dependent launch.  Where the filament kernel leaves room on the SMs (a tile
// per resident block), the mixed engine's kernels also release their successor
// before they end; in a larger network the successor's waiting blocks hold
// registers and thread slots that the filament blocks would use, and the next
// kernel is released by the end of this one.  Per iteration without PDL / with
// / released early (released at the start): 60k cylinders 59.8 / 57.6 / 56.5
// (56.5) us, 4k 60.4 / 58.4 / 57.9 (58.0), 1M 128.4 / 127.0 / 130.4 (153.7);
// FP64 4k 65.6 / 63.6 / - (73.3).
template <typename Real>
__device__ __forceinline__ void release_next(const DevNet<Real>& n) {
    if (n.n_ftiles <= 4 * 152) pdl_trigger();
}

// Two blocks fit on an SM; a second wave of blocks that find nothing flagged
// cost 0.7 us in every force evaluation.
constexpr int kFbForceBlocks = 2 * 152;

// numeric forces: partial moments of (entry, chunk), combined by the last chunk
template <typename Real>
__global__ void __launch_bounds__(kBlock) k_exvol_fb_force(DevNet<Real> n, double* moments, int* tickets) {
    pdl_wait();      // the flagged pairs are listed
    MECH_TRACE_KERNEL(n, TK_EXVOL_FB_FORCE);
    __shared__ double sh[32];
    __shared__ int s_last;
    const int cnt = min(*n.ev_fb_count, kExvolFallbackCap);
    const int N = kFbNodesForce;
    for (int wi = blockIdx.x; wi < cnt * kFbChunks; wi += gridDim.x) {
        const int k = wi / kFbChunks, ch = wi % kFbChunks;
        const int pr = n.ev_fb_list[2 * k + 1];
        const int4 bs = n.ev_bead[pr];
        const CGState& S = n.st[n.ev_fb_list[2 * k]];
        const Real* X = n.x[S.xbuf];
        double c1[3], c2[3], c3[3], c4[3];
        to_double(load_pos(X, bs.x), c1);
        to_double(load_pos(X, bs.y), c2);
        to_double(load_pos(X, bs.z), c3);
        to_double(load_pos(X, bs.w), c4);
        const Quad q = quad_of(c1, c2, c3, c4);
        const int i0 = (int)((long long)(N + 1) * ch / kFbChunks), i1 = (int)((long long)(N + 1) * (ch + 1) / kFbChunks);
        double m[6] = {0, 0, 0, 0, 0, 0};
        for (int i = i0; i < i1; ++i) {
            const double s = node(i, N), ws = weight(i, N);
            for (int j = threadIdx.x; j <= N; j += blockDim.x) {
                const double t = node(j, N), w = ws * weight(j, N);
                const double r2 = r2_at(q, s, t);
                const double x = w * (1.0 / (r2 * r2 * r2));
                m[0] += x; m[1] += s * x; m[2] += s * s * x; m[3] += s * t * x; m[4] += t * x; m[5] += t * t * x;
            }
        }
        for (int qd = 0; qd < 6; ++qd) {
            const double v = block_sum(m[qd], sh);
            if (threadIdx.x == 0) moments[((size_t)k * kFbChunks + ch) * 6 + qd] = v;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            const int tk = atomicAdd(tickets + k, 1);
            s_last = (tk == kFbChunks - 1);
            if (s_last) tickets[k] = 0;
        }
        __syncthreads();
        if (s_last && threadIdx.x == 0) {
            __threadfence();
            double I[6] = {0, 0, 0, 0, 0, 0};
            for (int cc = 0; cc < kFbChunks; ++cc)
                for (int qd = 0; qd < 6; ++qd) I[qd] += __ldcg(moments + ((size_t)k * kFbChunks + cc) * 6 + qd);
            const double ds = 1.0 / N;
            for (int qd = 0; qd < 6; ++qd) I[qd] *= (ds * ds / 9.0);
            const double kRepScaled = (double)n.ev_k[pr] * (double)n.ev_la[pr] * (double)n.ev_lb[pr];
            double vA[3], vB[3], vC[3], out[4][3];
            for (int kk = 0; kk < 3; ++kk) { vA[kk] = c1[kk] - c2[kk]; vB[kk] = c3[kk] - c4[kk]; vC[kk] = c3[kk] - c1[kk]; }
            bool ok = true;
            for (int kk = 0; kk < 3; ++kk) {
                out[0][kk] = 4.0 * kRepScaled * (-I[0] * vC[kk] + I[1] * (vC[kk] - vA[kk]) + I[2] * vA[kk] + I[4] * vB[kk] - I[3] * vB[kk]);
                out[1][kk] = 4.0 * kRepScaled * (-I[1] * vC[kk] - I[2] * vA[kk] + I[3] * vB[kk]);
                out[2][kk] = 4.0 * kRepScaled * (I[0] * vC[kk] + I[1] * vA[kk] - I[4] * (vB[kk] + vC[kk]) - I[3] * vA[kk] + I[5] * vB[kk]);
                out[3][kk] = 4.0 * kRepScaled * (I[4] * vC[kk] + I[3] * vA[kk] - I[5] * vB[kk]);
            }
            for (int a = 0; a < 4; ++a)
                for (int kk = 0; kk < 3; ++kk) ok = ok && !bad_value(out[a][kk]);
            if (!ok) {
                // Nothing finite is left to use: the reference exits the process
                // here (CylinderExclVolRepulsion.cpp:1195-1254).
                atomicOr(n.err, 1u);
                for (int a = 0; a < 4; ++a)
                    for (int kk = 0; kk < 3; ++kk) out[a][kk] = __longlong_as_double(0x7ff8000000000000ULL);
            }
            for (int a = 0; a < 4; ++a) {
                Real* cdst = slot_ptr(n, n.slot_base[K_EXVOL] + 4 * pr + a);
                for (int kk = 0; kk < 3; ++kk) cdst[kk] = (Real)out[a][kk];
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// mixed engine: main pair kernel (per-pair energies or force contributions)
// ---------------------------------------------------------------------------
template <typename Real>
__device__ __forceinline__ void flag_fallback(const DevNet<Real>& n, int r, int pr, double lam) {
    const int k = atomicAdd(n.ev_fb_count, 1);
    if (k < kExvolFallbackCap) {
        n.ev_fb_list[2 * k] = r;
        n.ev_fb_list[2 * k + 1] = pr;
        ((long long*)n.ev_fb_energy)[kExvolFallbackCap + k] = __double_as_longlong(lam);
    } else {
        atomicOr(n.err, 2u);
    }
}

constexpr float kMixedTauEnergy = 0.005f;  // extended pass below this normalized triple product (energy)
constexpr float kMixedTauForce = 0.02f;    // (forces, whose formula loses more to cancellation)

// Warp-aggregated append of an entry (a, b) to a list of 2 n_ev entries.
template <typename Real>
__device__ __forceinline__ void append_entry(const DevNet<Real>& n, int* list, int* count, bool need, int a, int b) {
    const unsigned m = __ballot_sync(0xffffffffu, need);
    if (!m) return;
    const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(count, __popc(m));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (need) {
        const int k = base + __popc(m & ((1u << lane) - 1u));
        if (k < 2 * n.n_ev) {   // room for both trials of a two-trial pass
            list[2 * k] = a;
            list[2 * k + 1] = b;
        } else {
            atomicOr(n.err, 4u);
        }
    }
}
// (replica, pair) to the extended-pass pair list
template <typename Real>
__device__ __forceinline__ void append_fp64(const DevNet<Real>& n, bool need, int r, int pr) {
    append_entry(n, n.ev_list, n.ev_list_count, need, r, pr);
}

// How the mixed engine forms a pair's forces.  The reference moves c2 0.01 nm
// along the unit normal of (c1, c2, c3) when it judges the pair coplanar
// (|n . v3| < 0.1 with n = (c2-c1) x (c3-c1), v3 = c4 - c1; :610-626).  Pairs
// whose test single precision cannot decide, and ill-conditioned ones (q), go
// to the extended pass; the others are moved here (with q >= kMixedTauForce the
// move leaves them well conditioned).
struct ForceCase {
    bool ill;             // to the extended pass
    float nx, ny, nz;     // -n
    float nn, cop;        // |n|, the reference's test
};
__device__ __forceinline__ ForceCase force_case(const float* v12, const float* v31, const float* v14, float q) {
    ForceCase c;
    c.nx = v12[1] * v31[2] - v12[2] * v31[1];
    c.ny = v12[2] * v31[0] - v12[0] * v31[2];
    c.nz = v12[0] * v31[1] - v12[1] * v31[0];
    c.nn = sqrtf(c.nx * c.nx + c.ny * c.ny + c.nz * c.nz);
    c.cop = fabsf(c.nx * v14[0] + c.ny * v14[1] + c.nz * v14[2]) / (c.nn * sqrtf(dot3(v14, v14)));
    c.ill = !(q >= kMixedTauForce) || !(fabsf(c.cop - 0.1f) >= 2e-3f);
    return c;
}

// Mixed engine: the energy of one pair in single precision, or need64 when the
// pair is ill-conditioned (normalized triple product under kMixedTauEnergy) or
// the formula gives no number; such pairs go to the extended pass.  With `list`
// also whether the pair's forces would.
__device__ __forceinline__ float mixed_pair_energy(const Pos<float>& p1, const Pos<float>& p2, const Pos<float>& p3,
                                                   const Pos<float>& p4, float kRep, bool& need64, bool list,
                                                   bool& ill) {
    float v12[3], v34[3], v31[3], v14[3], v32[3], v24[3];
    pdiff(p2, p1, v12);
    pdiff(p4, p3, v34);
    pdiff(p1, p3, v31);
    pdiff(p4, p1, v14);
    pdiff(p2, p3, v32);
    pdiff(p4, p2, v24);
    const float cx = v12[1] * v34[2] - v12[2] * v34[1], cy = v12[2] * v34[0] - v12[0] * v34[2],
                cz = v12[0] * v34[1] - v12[1] * v34[0];
    const float trip = fabsf(cx * v31[0] + cy * v31[1] + cz * v31[2]);
    const float q = trip / (sqrtf(dot3(v12, v12)) * sqrtf(dot3(v34, v34)) * sqrtf(dot3(v31, v31)));
    if (list) ill = force_case(v12, v31, v14, q).ill;
    need64 = !(q >= kMixedTauEnergy);
    if (need64) return 0.f;
    PairInv<float> pi;
    pair_inv(v12, v34, v31, v14, v32, v24, pi, true);
    const float u = energy_value(pi, kRep);
    if (u != u) {
        need64 = true;
        return 0.f;
    }
    return u;
}

// ---------------------------------------------------------------------------
// FP64 engine: the reference's formulas for every pair, bound by the FP64 pipe
// (a warp's FP64 instruction holds its SM sub-partition's pipe for ~78 cycles
// whatever the number of active lanes).  A pair per lane takes ~800 FP64
// instructions for the energy and ~1,650 for the forces in one warp, so a few
// pairs take as long as 608 warps of them (28 and 59 us).  Split over the four
// warps of a block (32 pairs on the lanes, warp w the w-th arctangent term, the
// invariants formed by every warp), the longest warp has about a third of that.
// Full rounds of 608 warps (76 tiles of 256 pairs) go unsplit; the rest goes
// split where that beats another round: three split blocks on every SM, 57
// tiles.  Both forms make the same operations in the same order: same bits.
// 78 pairs: energy 35 -> 19 us, forces 62 -> 29 us (with the chain's other
// launches); 59,737 pairs, where a fourth round held 3% of the pairs: 131 ->
// 111 and 234 -> 189 us.
// ---------------------------------------------------------------------------
constexpr int kExvolRoundTiles = 152 * 4 * 32 / kSparseTile;
constexpr int kExvolSplitTiles = 3 * 152 * 32 / kSparseTile;
inline int exvol_split_tiles(int nt) {
    const int rest = nt % kExvolRoundTiles;
    return rest <= kExvolSplitTiles ? rest : 0;
}

// One pair's term w of the four: operands shared through shared memory.
struct SplitTerm {
    double tC, tX, te, ta;    // partials of the term (forces)
    double S;                 // N / Y * ATG
    double q[3];              // the quotients by Y that G takes (forces)
};
enum SplitDot { SD_a, SD_b, SD_c, SD_d, SD_e, SD_F, SD_g, SD_h, SD_I, SD_D2, SD_E2, SD_JJ, SD_N };
struct SplitShared {
    double c[4][3][32];       // bead positions; c2 moved off the plane for forces
    double d[SD_N][32];       // the products of pair_inv (cross = false)
    double N[3][32];          // CC, GG, DD (HH = CC + GG - DD)
    SplitTerm t[4][32];
    double G[6][32];          // G00, G01, G02, G11, G12, G22
    double J[6][32];          // the same of J
    double pref[32], m[32];   // kRep / (2 JJ), -S / JJ
    int bad[32];
};

// 32 pairs [i0, min(i0 + 32, end)) of replica r in a block of four warps.  The
// pass takes as long as the longest warp's FP64 instructions, so what more than
// one warp needs is formed by one of them, in steps of about equal length, and
// for forces what does not hang on c2 while one warp decides on its move (78
// pairs, in an iteration: energy 12.2 -> 10.8 us, forces 20.4 -> 18.1 us, against
// every warp forming the products, J and the factors for itself).
template <typename Real>
__device__ void exvol_split(const DevNet<Real>& n, int r, const Real* X, const Direction<Real>& dir, bool tr, double lam,
                            int force, int i0, int end, SplitShared& s) {
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, i = i0 + l;
    const bool valid = i < end;
    if (valid) {
        const int4 bs = n.ev_bead[i];
        const int bead = w == 0 ? bs.x : w == 1 ? bs.y : w == 2 ? bs.z : bs.w;
        double c[3];
        to_double(bead_at(X, dir, bead, tr, (Real)lam), c);
#pragma unroll
        for (int k = 0; k < 3; ++k) s.c[w][k][l] = c[k];
    }
    if (w == 0) s.bad[l] = 0;
    __syncthreads();
    auto diff = [&](int a, int b, double v[3]) {   // bead a - bead b
#pragma unroll
        for (int k = 0; k < 3; ++k) v[k] = s.c[a][k][l] - s.c[b][k][l];
    };
    double v12[3], v34[3], v31[3];
    if (force) {
        if (valid) {
            if (w == 1) {   // the reference's move of c2, decided and applied
                double c[4][3], m[3];
#pragma unroll
                for (int a = 0; a < 4; ++a)
#pragma unroll
                    for (int k = 0; k < 3; ++k) c[a][k] = s.c[a][k][l];
                if (nearly_coplanar(c[0], c[1], c[2], c[3])) {
                    push_c2(c[0], c[1], c[2], m);
#pragma unroll
                    for (int k = 0; k < 3; ++k) s.c[1][k][l] = m[k];
                }
            } else if (w == 0) {
                diff(0, 2, v31);
                s.d[SD_c][l] = dot3(v31, v31);
            } else if (w == 2) {
                diff(3, 2, v34);
                diff(0, 2, v31);
                s.d[SD_b][l] = dot3(v34, v34);
                s.d[SD_F][l] = dot3(v34, v31);
            } else {
                double v14[3];
                diff(3, 0, v14);
                diff(3, 2, v34);
                s.d[SD_D2][l] = dot3(v14, v14);
                s.d[SD_I][l] = dot3(v34, v14);
            }
        }
        __syncthreads();
    }
    if (valid) {
        if (w == 0) {
            diff(1, 0, v12);
            diff(3, 2, v34);
            diff(0, 2, v31);
            s.d[SD_a][l] = dot3(v12, v12);
            const double x21[3] = {v34[1] * v12[2] - v34[2] * v12[1], v34[2] * v12[0] - v34[0] * v12[2],
                                   v34[0] * v12[1] - v34[1] * v12[0]};
            const double trip = -(x21[0] * v31[0] + x21[1] * v31[1] + x21[2] * v31[2]);
            s.d[SD_JJ][l] = -trip * trip;
        } else if (w == 1) {
            double v14[3];
            diff(1, 0, v12);
            diff(3, 0, v14);
            s.d[SD_g][l] = dot3(v12, v14);
            if (!force) {
                diff(3, 2, v34);
                s.d[SD_D2][l] = dot3(v14, v14);
                s.d[SD_I][l] = dot3(v34, v14);
            }
        } else if (w == 2) {
            diff(1, 0, v12);
            diff(3, 2, v34);
            diff(0, 2, v31);
            s.d[SD_d][l] = dot3(v12, v34);
            s.d[SD_e][l] = dot3(v12, v31);
            if (!force) s.d[SD_c][l] = dot3(v31, v31);
        } else {
            double v32[3];
            diff(1, 2, v32);
            diff(3, 2, v34);
            s.d[SD_E2][l] = dot3(v32, v32);
            s.d[SD_h][l] = dot3(v34, v32);
            if (!force) {
                diff(0, 2, v31);
                s.d[SD_b][l] = dot3(v34, v34);
                s.d[SD_F][l] = dot3(v34, v31);
            }
        }
    }
    __syncthreads();
    double a = 0, b = 0, c = 0, d = 0, e = 0, F = 0, Y = 1, N = 0, ATG = 0, al = 0, be = 0;
    if (valid) {
        a = s.d[SD_a][l];
        b = s.d[SD_b][l];
        c = s.d[SD_c][l];
        d = s.d[SD_d][l];
        e = s.d[SD_e][l];
        F = s.d[SD_F][l];
        // term w: Y, N and the two abscissae (A, E, B, F of the reference)
        double u = a, v = c, x = e;   // Y = sqrt((sqrt(u v) + x) (sqrt(u v) - x))
        al = a + e;
        be = e;
        if (w == 0) {
            N = d * e - a * F;
        } else if (w == 1) {
            v = s.d[SD_D2][l];
            x = s.d[SD_g][l];
            N = d * x - a * s.d[SD_I][l];
            al = a + e - d;
            be = e - d;
        } else if (w == 2) {
            u = b;
            x = F;
            N = b * e - d * F;
            al = F;
            be = F - b;
        } else {
            u = b;
            v = s.d[SD_E2][l];
            x = s.d[SD_h][l];
            al = d + F;
            be = d + F - b;
        }
        const double uv = sqrt(u * v);
        Y = sqrt(fmax(0.0, (uv + x) * (uv - x)));
        if (w < 3) s.N[w][l] = N;
        ATG = atan_of(al / Y) - atan_of(be / Y);
    }
    __syncthreads();
    if (valid) {
        if (w == 3) N = s.N[0][l] + s.N[1][l] - s.N[2][l];
        SplitTerm t;
        t.S = N / Y * ATG;
        t.tC = t.tX = t.te = t.ta = t.q[0] = t.q[1] = t.q[2] = 0.0;
        if (force) {
            const double T1 = Y * Y / (Y * Y + al * al), T2 = Y * Y / (Y * Y + be * be);
            t.tC = ATG / Y;
            t.tX = -(ATG * N) / (Y * Y) + (-T1 * al + T2 * be) * N / (Y * Y * Y);
            t.te = (T1 - T2) * N / (Y * Y);
            t.ta = T1 * N / (Y * Y);
            t.q[0] = (w == 0 ? c : w == 1 ? b + c - 2 * F : b) / Y;
            t.q[1] = (w == 0 ? -e : w == 1 ? e - d : w == 2 ? c : -(d + F)) / Y;
            t.q[2] = (w == 0 || w == 1 ? a : w == 2 ? -F : a + c + 2 * e) / Y;
        }
        s.t[w][l] = t;
    }
    __syncthreads();
    if (!force) {
        if (w == 0 && valid) {
            const double kRep = (double)n.ev_k[i] * (double)n.ev_la[i] * (double)n.ev_lb[i];
            const double U = 0.5 * kRep / s.d[SD_JJ][l] * (s.t[0][l].S + s.t[1][l].S + s.t[2][l].S + s.t[3][l].S);
            const bool ok = !(bad_value(U) || U < -1.0);
            n.ev_energy[i] = ok ? U : 0.0;
            if (!ok) flag_fallback(n, r, i, tr ? lam : 0.0);
        }
        return;
    }
    if (valid) {   // entries of G and J and the factors, split over the warps
        const SplitTerm A = s.t[0][l], E = s.t[1][l], B = s.t[2][l], T = s.t[3][l];
        if (w == 0) {
            s.G[0][l] = A.tC * (-2 * F) + A.tX * A.q[0] + A.ta * 2 + E.tC * (2 * (F - b)) + E.tX * E.q[0] + E.ta * 2 +
                        T.tC * (-2 * b) + T.tX * T.q[0];
            s.G[5][l] = A.tX * A.q[2] + E.tX * E.q[2] + B.tX * B.q[0] + T.tX * T.q[0];
            s.J[5][l] = 2 * (d * d - a * b);
        } else if (w == 1) {
            s.G[1][l] = A.tC * e + E.tC * (2 * d - e) + E.tX * E.q[1] + E.te * (-1) + B.tC * (-F) + T.tC * (2 * d + F) +
                        T.tX * T.q[1] + T.te;
            s.G[2][l] = A.tC * d + A.tX * A.q[1] + A.te + E.tC * (-d) + E.tX * (-E.q[1]) + E.te + B.tC * b + T.tC * (-b) +
                        T.tX * T.q[0];
        } else if (w == 2) {
            s.G[3][l] = E.tC * (-2 * a) + E.tX * E.q[2] + B.tC * (2 * e) + B.tX * B.q[1] + B.te * (-2) + B.ta * 2 +
                        T.tC * (-2 * (a + e)) + T.tX * T.q[2] + T.te * (-2) + T.ta * 2;
            s.J[3][l] = 2 * (-a * c + e * e);
            s.J[4][l] = 2 * (-d * e + a * F);
            s.J[0][l] = 2 * (-b * c + F * F);
        } else {
            s.G[4][l] = A.tC * (-a) + E.tC * a + E.tX * (-E.q[2]) + B.tC * (-d) + B.tX * B.q[2] + B.te + T.tC * d +
                        T.tX * T.q[1] + T.te;
            s.J[1][l] = 2 * (c * d - e * F);
            s.J[2][l] = 2 * (b * e - d * F);
            const double kRep = (double)n.ev_k[i] * (double)n.ev_la[i] * (double)n.ev_lb[i];
            const double invJJ = 1.0 / s.d[SD_JJ][l];
            const double S = A.S + E.S + B.S + T.S;
            s.pref[l] = kRep * invJJ / 2.0;
            s.m[l] = -invJJ * S;
        }
    }
    __syncthreads();
    if (valid) {   // warp w: the force on bead w
        const double G[3][3] = {{s.G[0][l], s.G[1][l], s.G[2][l]}, {s.G[1][l], s.G[3][l], s.G[4][l]}, {s.G[2][l], s.G[4][l], s.G[5][l]}};
        const double J[3][3] = {{s.J[0][l], s.J[1][l], s.J[2][l]}, {s.J[1][l], s.J[3][l], s.J[4][l]}, {s.J[2][l], s.J[4][l], s.J[5][l]}};
        const double pref = s.pref[l], m = s.m[l];
        diff(1, 0, v12);
        diff(3, 2, v34);
        diff(0, 2, v31);
        double dv[3];
#pragma unroll
        for (int y = 0; y < 3; ++y) {
            const double Jw = w == 0 ? J[2][y] - J[0][y] : w == 1 ? J[0][y] : w == 2 ? -J[2][y] - J[1][y] : J[1][y];
            const double Gw = w == 0 ? G[2][y] - G[0][y] : w == 1 ? G[0][y] : w == 2 ? -G[2][y] - G[1][y] : G[1][y];
            dv[y] = pref * (m * Jw + Gw);
        }
        Real* dst = slot_ptr(n, n.slot_base[K_EXVOL] + 4 * i + w);
        bool bad = false;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const double o = -(dv[0] * v12[k] + dv[1] * v34[k] + dv[2] * v31[k]);
            if (bad_value(o)) bad = true;
            dst[k] = (Real)o;
        }
        if (bad) atomicOr(&s.bad[l], 1);
    }
    __syncthreads();
    if (w == 0 && valid && s.bad[l]) flag_fallback(n, r, i, 0.0);
}

// Blocks [0, 2 unsplit): half a tile each, a pair per thread; then eight blocks
// per split tile.
template <typename Real>
__global__ void __launch_bounds__(128) k_exvol_fp64(DevNet<Real> n, int want, int trial, int force, int tile_off,
                                                    int unsplit) {
    pdl_wait();      // the reduction before this evaluation has finished
    MECH_TRACE_KERNEL(n, TK_EXVOL);
    __shared__ SplitShared s;
    const int sb = (int)blockIdx.x - 2 * unsplit;
    int kind;
    const Tile t = sparse_tile(n, tile_off + (sb < 0 ? (int)blockIdx.x >> 1 : unsplit + (sb >> 3)), &kind);
    const int begin = t.begin + (sb < 0 ? 128 * ((int)blockIdx.x & 1) : 32 * (sb & 7));
    if (begin >= t.end) return;
    const LaneState<Real> ls = lane_state(n, t.replica, want);
    if (!ls.go) return;
    const Direction<Real> dir = direction_of(n, ls);
    const Real* X = n.x[ls.xb];
    const double lam = ls.lambda;
    const bool tr = trial != 0;
    if (sb >= 0) {
        exvol_split(n, t.replica, X, dir, tr, lam, force, begin, t.end, s);
        return;
    }
    const int i = begin + threadIdx.x;
    if (i >= t.end) return;
    const int4 bs = n.ev_bead[i];
    const double kRep = (double)n.ev_k[i] * (double)n.ev_la[i] * (double)n.ev_lb[i];
    double c1[3], c2[3], c3[3], c4[3];
    to_double(bead_at(X, dir, bs.x, tr, (Real)lam), c1);
    to_double(bead_at(X, dir, bs.y, tr, (Real)lam), c2);
    to_double(bead_at(X, dir, bs.z, tr, (Real)lam), c3);
    to_double(bead_at(X, dir, bs.w, tr, (Real)lam), c4);
    if (!force) {
        const double u = pair_energy_d(c1, c2, c3, c4, kRep);
        n.ev_energy[i] = u == u ? u : 0.0;
        if (u != u) flag_fallback(n, t.replica, i, tr ? lam : 0.0);
    } else {
        double out[4][3];
        const bool ok = pair_forces_d(c1, c2, c3, c4, kRep, out);
        for (int a = 0; a < 4; ++a) {
            Real* cdst = slot_ptr(n, n.slot_base[K_EXVOL] + 4 * i + a);
            for (int k = 0; k < 3; ++k) cdst[k] = (Real)out[a][k];
        }
        if (!ok) flag_fallback(n, t.replica, i, 0.0);
    }
}

template <typename Real>
__global__ void __launch_bounds__(kBlock) k_exvol(DevNet<Real> n, int want, int trial, int force, int tile_off) {
    pdl_wait();      // the reduction before this evaluation has finished
    MECH_TRACE_KERNEL(n, TK_EXVOL);
    int kind;
    const Tile t = sparse_tile(n, tile_off + (int)blockIdx.x, &kind);
    const int r = t.replica;
    const LaneState<Real> s = lane_state(n, r, want);
    if (!s.go) return;
    const Direction<Real> dir = direction_of(n, s);
    const Real* X = n.x[s.xb];
    const bool tr = trial != 0;
    const int i = t.begin + threadIdx.x;
    const bool valid = i < t.end;
    float ef = 0.f;
    bool need64 = false, need64b = false, ill = false, illb = false;
    // a pass with a second trial also evaluates the energy at lambda / 2
    const bool dual = !force && second_trial(trial, s.dual);
    // position buffers of the trials
    const int buf = (s.xb + 1) % 3, bufb = (s.xb + 2) % 3;
    if (valid) {
        const int4 bs = n.ev_bead[i];
        auto pos = [&](int b) -> Pos<float> { return bead_at(X, dir, b, tr, s.lam); };
        const Pos<Real> p1 = pos(bs.x), p2 = pos(bs.y), p3 = pos(bs.z), p4 = pos(bs.w);
        if (!force) {
            // mixed engine: single precision unless the pair is ill-conditioned
            const float kRep = n.ev_k[i] * n.ev_la[i] * n.ev_lb[i];
            ef = mixed_pair_energy(p1, p2, p3, p4, kRep, need64, n.prelist, ill);
            store_pair(n.ev_energy + i, ef, 0.f);
            if (dual) {
                const float lh = 0.5f * s.lam;
                const float ef2 = mixed_pair_energy(bead_at(X, dir, bs.x, true, lh), bead_at(X, dir, bs.y, true, lh),
                                                    bead_at(X, dir, bs.z, true, lh), bead_at(X, dir, bs.w, true, lh),
                                                    kRep, need64b, n.prelist, illb);
                store_pair(n.ev_energy2 + i, ef2, 0.f);
            }
            if (n.prelist) n.ev_mark[i] = (uint8_t)((ill << buf) | (illb << bufb));
        } else if (!n.prelist || !(n.ev_mark[i] >> s.xb & 1)) {
            // mixed engine, forces: single precision unless the pair is ill-conditioned
            const float kRep = n.ev_k[i] * n.ev_la[i] * n.ev_lb[i];
            float v12[3], v34[3], v31[3], v14[3], v32[3], v24[3];
            pdiff(p2, p1, v12);
            pdiff(p4, p3, v34);
            pdiff(p1, p3, v31);
            pdiff(p4, p1, v14);
            pdiff(p2, p3, v32);
            pdiff(p4, p2, v24);
            const float cx = v12[1] * v34[2] - v12[2] * v34[1], cy = v12[2] * v34[0] - v12[0] * v34[2],
                        cz = v12[0] * v34[1] - v12[1] * v34[0];
            const float trip = fabsf(cx * v31[0] + cy * v31[1] + cz * v31[2]);
            const float q = trip / (sqrtf(dot3(v12, v12)) * sqrtf(dot3(v34, v34)) * sqrtf(dot3(v31, v31)));
            const ForceCase fc = force_case(v12, v31, v14, q);
            need64 = n.prelist ? false : fc.ill;
            if (!need64 && fc.cop < 0.1f) {
                const float push = -0.01f / fc.nn;
                const float dx = push * fc.nx, dy = push * fc.ny, dz = push * fc.nz;   // c2 moves by +0.01 n / |n|
                v12[0] += dx; v12[1] += dy; v12[2] += dz;
                v32[0] += dx; v32[1] += dy; v32[2] += dz;
                v24[0] -= dx; v24[1] -= dy; v24[2] -= dz;
            }
            if (!need64) {
                PairInv<float> pi;
                pair_inv(v12, v34, v31, v14, v32, v24, pi, true);
                float out[4][3];
                if (forces_from<true>(pi, v12, v34, v31, kRep, out)) {
                    for (int a = 0; a < 4; ++a) {
                        Real* cdst = slot_ptr(n, n.slot_base[K_EXVOL] + 4 * i + a);
                        for (int k = 0; k < 3; ++k) cdst[k] = (Real)out[a][k];
                    }
                } else {
                    need64 = true;
                }
            }
        }
    }
    append_fp64(n, need64, r, i);
    if (dual) append_fp64(n, need64b, r, i | kExtSecond);   // block-uniform
    if (n.prelist && !force) {
        append_entry(n, n.ev_flist, n.ev_flist_count, ill, r | buf << kListBuffer, i);
        if (dual) append_entry(n, n.ev_flist, n.ev_flist_count, illb, r | bufb << kListBuffer, i);
    }
    release_next(n);
}

// Mixed engine's extended pass: the listed (ill-conditioned) pairs in FP64,
// split over the four warps of a block.  On this GPU a warp's FP64
// instruction holds its SM sub-partition's FP64 pipe for ~78 cycles whatever
// the number of active lanes, so the time of the pass is the FP64 instruction
// count of one warp's path, not the pair count: one pair's ~1,000 FP64
// operations in one warp took ~35 us.  Here lane l of every warp takes pair
// 32 g + l of the block's group g, and warp w evaluates the w-th of the four
// arctangent terms of the integral (A, E, B, F below: cross product, norm,
// numerator, arctangent and, for forces, its partial derivatives); the vectors
// are formed by every warp, the scalar products, the entries of the G and J
// matrices and the common factors each by one of them (forces 13.0 -> 11.9 us in
// an iteration of 60k cylinders, against every warp forming all but G), and warp
// w forms the force on bead w.  Partial results pass through shared memory.  The cancellation-free forms of pair_inv
// (cross = true) and forces_from<true> are followed term by term, with the
// reference's coplanar move of c2 (:610-626, forces only, decided without
// divisions: (n . v3)^2 < 0.01 |n|^2 |v3|^2).
constexpr int kExtBlocks = 152;   // one 4-warp block per SM: one warp per sub-partition

// per-term operands: cross product u x v, arctangent argument p . q (negated for B, F),
// and the two arctangent abscissae alpha, beta (A: a+e, e; E: a+e-d, e-d; B: F, F-b; F: d+F, d+F-b)
struct ExtTerm {
    double N, rY, ATG, tN, tXr, tlo, thi, S;
};

template <typename Real>
__global__ void __launch_bounds__(128) k_exvol_ext(DevNet<Real> n, int trial, int force, int listed) {
    pdl_wait();      // the listing pass has finished
    MECH_TRACE_KERNEL(n, TK_EXVOL_EXT);
    __shared__ double s_c[4][32][3];       // bead positions
    __shared__ double s_N[3][32];          // CC, GG, DD for the F term's HH
    __shared__ ExtTerm s_t[4][32];
    __shared__ double s_G[6][32];
    __shared__ double s_dot[6][32];        // a, b, c, d, e, F
    __shared__ double s_J[6][32];          // J00, J01, J02, J11, J12, J22
    __shared__ double s_JJ[32], s_k[32];   // JJ; kRep, then (forces) kRep / (2 JJ)
    __shared__ double s_m[32];             // -S / JJ
    __shared__ int s_bad[32];
    const int* list = listed ? n.ev_flist : n.ev_list;
    const int cnt = min(listed ? *n.ev_flist_count : *n.ev_list_count, 2 * n.n_ev);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const int ngroups = (cnt + 31) >> 5;
    for (int g = blockIdx.x; g < ngroups; g += gridDim.x) {
        const int k = 32 * g + l;
        bool valid = k < cnt;
        int r = 0, i = 0;
        bool second = false;   // the lambda / 2 trial of a two-trial pass
        double lam = 0.0;
        LaneState<Real> ls{};
        if (valid) {
            r = list[2 * k];
            i = list[2 * k + 1];
            if (listed) {   // of the accepted trial
                const int buf = r >> kListBuffer;
                r &= (1 << kListBuffer) - 1;
                ls = lane_state(n, r, PH_FORCE);
                valid = ls.go && ls.xb == buf;
            } else {
                second = (i & kExtSecond) != 0;
                i &= ~kExtSecond;
                ls = lane_state(n, r, -1);
            }
            lam = ls.lambda;
            if (second) lam *= 0.5;
        }
        // ---- positions: warp w converts bead w of every pair
        if (valid) {
            const int4 bs = n.ev_bead[i];
            const int bead = w == 0 ? bs.x : w == 1 ? bs.y : w == 2 ? bs.z : bs.w;
            double c[3];
            to_double(bead_at(n.x[ls.xb], direction_of(n, ls), bead, trial != 0, (Real)lam), c);
            s_c[w][l][0] = c[0];
            s_c[w][l][1] = c[1];
            s_c[w][l][2] = c[2];
        }
        if (w == 0) s_bad[l] = 0;
        __syncthreads();
        double v12[3], v34[3], v31[3], v14[3], v32[3], v24[3];
        double a = 0, b = 0, c = 0, d = 0, e = 0, F = 0;
        double x21[3] = {0, 0, 0};
        if (valid) {
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const double c1 = s_c[0][l][q], c2 = s_c[1][l][q], c3 = s_c[2][l][q], c4 = s_c[3][l][q];
                v12[q] = c2 - c1;
                v34[q] = c4 - c3;
                v31[q] = c1 - c3;
                v14[q] = c4 - c1;
                v32[q] = c2 - c3;
                v24[q] = c4 - c2;
            }
            if (force) {
                // n = (c2 - c1) x (c3 - c1) = -(v12 x v31), v3 = c4 - c1 = v14
                const double nx = v12[2] * v31[1] - v12[1] * v31[2], ny = v12[0] * v31[2] - v12[2] * v31[0],
                             nz = v12[1] * v31[0] - v12[0] * v31[1];
                const double nn = nx * nx + ny * ny + nz * nz, nv = nx * v14[0] + ny * v14[1] + nz * v14[2];
                if (nv * nv < 0.01 * nn * dot3(v14, v14)) {
                    const double sc = 0.01 / sqrt(nn);
                    const double dn[3] = {sc * nx, sc * ny, sc * nz};
#pragma unroll
                    for (int q = 0; q < 3; ++q) {
                        v12[q] += dn[q];
                        v32[q] += dn[q];
                        v24[q] -= dn[q];
                    }
                }
            }
            x21[0] = v34[1] * v12[2] - v34[2] * v12[1];
            x21[1] = v34[2] * v12[0] - v34[0] * v12[2];
            x21[2] = v34[0] * v12[1] - v34[1] * v12[0];
            // what every warp needs later, each formed by one of them
            if (w == 3) {
                const double trip = -(x21[0] * v31[0] + x21[1] * v31[1] + x21[2] * v31[2]);
                s_JJ[l] = -trip * trip;
                s_k[l] = (double)n.ev_k[i] * (double)n.ev_la[i] * (double)n.ev_lb[i];
            }
            if (force) {
                if (w == 0) {
                    s_dot[0][l] = dot3(v12, v12);
                    s_dot[1][l] = dot3(v34, v34);
                } else if (w == 1) {
                    s_dot[2][l] = dot3(v31, v31);
                    s_dot[3][l] = dot3(v12, v34);
                } else if (w == 2) {
                    s_dot[4][l] = dot3(v12, v31);
                    s_dot[5][l] = dot3(v34, v31);
                }
            }
        }
        // ---- term w: cross product, norm, numerator
        double xu[3] = {0, 0, 0}, Y = 1, N = 0;
        if (valid) {
            double u[3], v[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) {   // selects, not pointers: the vectors stay in registers
                u[q] = w < 2 ? v12[q] : v34[q];
                v[q] = w == 0 ? v31[q] : w == 1 ? v14[q] : w == 2 ? v31[q] : v32[q];
            }
            xu[0] = u[1] * v[2] - u[2] * v[1];
            xu[1] = u[2] * v[0] - u[0] * v[2];
            xu[2] = u[0] * v[1] - u[1] * v[0];
            Y = sqrt(dot3(xu, xu));
            if (w < 3) {
                N = dot3(xu, x21);   // CC = x13 . x21, GG = x14 . x21, DD = x21 . x23
                s_N[w][l] = N;
            }
        }
        __syncthreads();
        if (valid) {
            if (w == 3) N = s_N[0][l] + s_N[1][l] - s_N[2][l];   // HH = CC + GG - DD
            double p[3], q[3];
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                p[j] = w == 0 ? v31[j] : w == 1 ? v14[j] : w == 2 ? v31[j] : v32[j];
                q[j] = w == 0 ? v32[j] : w == 1 ? v24[j] : w == 2 ? v14[j] : v24[j];
            }
            const double arg = w < 2 ? dot3(p, q) : -dot3(p, q);
            ExtTerm t;
            t.N = N;
            t.ATG = atan2(Y, arg);
            t.rY = 1.0 / Y;
            t.S = N * t.rY * t.ATG;
            if (force) {
                a = s_dot[0][l];
                b = s_dot[1][l];
                c = s_dot[2][l];
                d = s_dot[3][l];
                e = s_dot[4][l];
                F = s_dot[5][l];
                const double al = w == 0 ? a + e : w == 1 ? a + e - d : w == 2 ? F : d + F;
                const double be = al - (w < 2 ? a : b);
                const double Y2 = Y * Y;
                const double T1 = Y2 / (Y2 + al * al), T2 = Y2 / (Y2 + be * be);
                const double r2 = t.rY * t.rY;
                t.tN = t.ATG * t.rY;
                const double tX = -(t.ATG * N) * r2 + ((-T1 * al + T2 * be) * N) * (r2 * t.rY);
                t.tXr = tX * t.rY;
                t.tlo = ((T1 - T2) * N) * r2;
                t.thi = (T1 * N) * r2;
            }
            s_t[w][l] = t;
        }
        __syncthreads();
        if (g + gridDim.x >= ngroups) release_next(n);   // the block's last group
        if (!force) {
            if (w == 0 && valid) {
                const double Ssum = s_t[0][l].S + s_t[1][l].S + s_t[2][l].S + s_t[3][l].S;
                const double U = 0.5 * s_k[l] / s_JJ[l] * Ssum;
                double* dst = (second ? n.ev_energy2 : n.ev_energy) + i;
                if (!(fabs(U) < 1.0 / 0.0) || U < -1.0) {
                    flag_fallback(n, r, i, trial != 0 ? lam : 0.0);
                    store_pair(dst, 0.f, 0.f);
                } else {
                    const float h = (float)U;
                    store_pair(dst, h, (float)(U - (double)h));
                }
            }
            __syncthreads();   // shared arrays are reused by the next group
            continue;
        }
        // ---- entries of G and J and the factors, split over the warps
        // (0: G00, G12; 1: G01, G22, J11, J12, J22; 2: G02, factors; 3: G11, J00, J01, J02)
        if (valid) {
            const ExtTerm A = s_t[0][l], E = s_t[1][l], B = s_t[2][l], FT = s_t[3][l];
            if (w == 0) {
                s_G[0][l] = A.tN * (-2 * F) + A.tXr * c + A.thi * 2 + E.tN * (2 * (F - b)) + E.tXr * (b + c - 2 * F) +
                            E.thi * 2 + FT.tN * (-2 * b) + FT.tXr * b;
                s_G[4][l] = A.tN * (-a) + E.tN * a + E.tXr * (-a) + B.tN * (-d) + B.tXr * (-F) + B.tlo + FT.tN * d +
                            FT.tXr * (-(d + F)) + FT.tlo;
            } else if (w == 1) {
                s_G[1][l] = A.tN * e + E.tN * (2 * d - e) + E.tXr * (e - d) - E.tlo + B.tN * (-F) + FT.tN * (2 * d + F) +
                            FT.tXr * (-(d + F)) + FT.tlo;
                s_G[5][l] = A.tXr * a + E.tXr * a + B.tXr * b + FT.tXr * b;
                s_J[3][l] = 2 * (-a * c + e * e);
                s_J[4][l] = 2 * (-d * e + a * F);
                s_J[5][l] = 2 * (d * d - a * b);
            } else if (w == 2) {
                const double invJJ = 1.0 / s_JJ[l];
                const double Ssum = A.S + E.S + B.S + FT.S;
                s_k[l] = s_k[l] * invJJ / 2.0;
                s_m[l] = -invJJ * Ssum;
                s_G[2][l] = A.tN * d + A.tXr * (-e) + A.tlo + E.tN * (-d) + E.tXr * (-(e - d)) + E.tlo + B.tN * b +
                            FT.tN * (-b) + FT.tXr * b;
            } else {
                s_G[3][l] = E.tN * (-2 * a) + E.tXr * a + B.tN * (2 * e) + B.tXr * c + B.tlo * (-2) + B.thi * 2 +
                            FT.tN * (-2 * (a + e)) + FT.tXr * (a + c + 2 * e) + FT.tlo * (-2) + FT.thi * 2;
                s_J[0][l] = 2 * (-b * c + F * F);
                s_J[1][l] = 2 * (c * d - e * F);
                s_J[2][l] = 2 * (b * e - d * F);
            }
        }
        __syncthreads();
        // ---- warp w: the force on bead w
        if (valid) {
            const double G[3][3] = {{s_G[0][l], s_G[1][l], s_G[2][l]},
                                    {s_G[1][l], s_G[3][l], s_G[4][l]},
                                    {s_G[2][l], s_G[4][l], s_G[5][l]}};
            const double J[3][3] = {{s_J[0][l], s_J[1][l], s_J[2][l]},
                                    {s_J[1][l], s_J[3][l], s_J[4][l]},
                                    {s_J[2][l], s_J[4][l], s_J[5][l]}};
            const double pref = s_k[l], m = s_m[l];
            double dv[3];
#pragma unroll
            for (int y = 0; y < 3; ++y) {
                const double Jw = w == 0 ? J[2][y] - J[0][y] : w == 1 ? J[0][y] : w == 2 ? -J[2][y] - J[1][y] : J[1][y];
                const double Gw = w == 0 ? G[2][y] - G[0][y] : w == 1 ? G[0][y] : w == 2 ? -G[2][y] - G[1][y] : G[1][y];
                dv[y] = pref * (m * Jw + Gw);
            }
            Real* cdst = slot_ptr(n, n.slot_base[K_EXVOL] + 4 * i + w);
            bool bad = false;
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const double o = -(dv[0] * v12[q] + dv[1] * v34[q] + dv[2] * v31[q]);
                if (!(fabs(o) < 1.0 / 0.0)) bad = true;
                cdst[q] = (Real)o;
            }
            if (bad) atomicOr(&s_bad[l], 1);
        }
        __syncthreads();
        if (w == 0 && valid && s_bad[l]) flag_fallback(n, r, i, 0.0);
        __syncthreads();   // shared arrays are reused by the next group
    }
}

// The end of an energy evaluation's excluded-volume chain, one launch:
// blocks [0, kFbEnergyBlocks) compute the Simpson energies of flagged pairs;
// the following blocks form the deterministic per-tile sums of the per-pair
// energies (one block per exvol tile).
constexpr int kFbEnergyBlocks = 64;
template <typename Real>
__global__ void __launch_bounds__(kBlock) k_exvol_energy_tail(DevNet<Real> n, int want, int trial, int tile_off) {
    pdl_wait();      // the per-pair energies are complete
    MECH_TRACE_KERNEL(n, TK_EXVOL_TAIL);
    __shared__ double sh[32];   // block_pair_sums<2>: 32 floats
    if ((int)blockIdx.x < kFbEnergyBlocks) {
        fb_energy_blocks(n, blockIdx.x, kFbEnergyBlocks, sh);
    } else {
        const int ti = tile_off + (int)blockIdx.x - kFbEnergyBlocks;
        int kind;
        const Tile t = sparse_tile(n, ti, &kind);
        const LaneState<Real> s = lane_state(n, t.replica, want);
        const bool go = s.go;
        if constexpr (sizeof(Real) == 4) {
            if (go) {   // block-uniform
                // per-pair energies as (hi, lo) pairs, summed compensated in single precision
                const int i = t.begin + threadIdx.x;
                if (second_trial(trial, s.dual)) {   // both trials of the pass
                    FF a[2];
                    if (i < t.end) {
                        add_pair(a[0], load_pair(n.ev_energy + i));
                        add_pair(a[1], load_pair(n.ev_energy2 + i));
                    }
                    const FF se = block_pair_sums<2>(a, reinterpret_cast<float*>(sh));
                    if (threadIdx.x < 2) store_pair((threadIdx.x ? n.part_sp2 : n.part_sp) + ti, se.h, se.l);
                } else {
                    FF a[1];
                    if (i < t.end) add_pair(a[0], load_pair(n.ev_energy + i));
                    const FF se = block_pair_sums<1>(a, reinterpret_cast<float*>(sh));
                    if (threadIdx.x == 0) store_pair(n.part_sp + ti, se.h, se.l);
                }
            }
        } else if (go) {
            const int i = t.begin + threadIdx.x;
            const double e = block_sum(i < t.end ? n.ev_energy[i] : 0.0, sh);
            if (threadIdx.x == 0) n.part_sp[ti] = e;
        }
    }
}

// zero the extended-pass and fallback work-list counts (one memset when they are
// neighbours in one buffer)
template <typename Real>
static inline void reset_counts(const DevNet<Real>& n, cudaStream_t s) {
    if (n.ev_fb_count == n.ev_list_count + 2) {
        cudaMemsetAsync(n.ev_list_count, 0, 4 * sizeof(int), s);
    } else {
        cudaMemsetAsync(n.ev_list_count, 0, sizeof(int), s);
        cudaMemsetAsync(n.ev_fb_count, 0, sizeof(int), s);
    }
}

template <typename Real>
static inline int ev_tiles_of(const DevNet<Real>& n, int* off) {
    *off = n.sp_tiles[K_LINKER] + n.sp_tiles[K_MOTOR];
    return n.sp_tiles[K_EXVOL];
}

// Inside an evaluation (standalone = false) the work-list counts are zero on
// entry: the energy's reduction, or the force gather, has zeroed them behind
// their last reader, which keeps a memset off the head of the excluded-volume lane.  A standalone
// launch zeroes them first and leaves them as they end.  `L`, unless null, are
// the evaluation's lanes: `s` is the side lane, and L->join is recorded behind
// the chain.
template <typename Real>
int launch_exvol_energy(const DevNet<Real>& n, int want, int trial, cudaStream_t s, bool standalone, const Lanes* L) {
    int off = 0;
    const int nt = ev_tiles_of(n, &off);
    const cudaEvent_t done = L ? L->join : nullptr;
    if (nt == 0) {
        if (done) cudaEventRecord(done, s);
        return 0;
    }
    if (standalone) reset_counts(n, s);
    int k = 1;
    if constexpr (sizeof(Real) == 8) {
        const int split = exvol_split_tiles(nt);
        launch_k(false, nullptr, k_exvol_fp64<Real>, 2 * (nt - split) + 8 * split, 128, s, n, want, trial, 0, off, nt - split);
    } else {
        launch_k(false, nullptr, k_exvol<Real>, nt, kBlock, s, n, want, trial, 0, off);
        launch_k(n.pdl, nullptr, k_exvol_ext<Real>, kExtBlocks, 128, s, n, trial, 0, 0);
        ++k;
    }
    launch_k(n.pdl, n.pdl ? done : nullptr, k_exvol_energy_tail<Real>, kFbEnergyBlocks + nt, kBlock, s, n, want, trial, off);
    if (done && !n.pdl) cudaEventRecord(done, s);
    return k + 1;
}

template <typename Real>
int launch_exvol_forces(const DevNet<Real>& n, int want, cudaStream_t s, bool standalone, const Lanes* L) {
    int off = 0;
    const int nt = ev_tiles_of(n, &off);
    const cudaEvent_t done = L ? L->join : nullptr;
    if (nt == 0) {
        if (done) cudaEventRecord(done, s);
        return 0;
    }
    if (standalone) reset_counts(n, s);
    int k = 1;
    if constexpr (sizeof(Real) == 8) {
        const int split = exvol_split_tiles(nt);
        launch_k(false, nullptr, k_exvol_fp64<Real>, 2 * (nt - split) + 8 * split, 128, s, n, want, 0, 1, off, nt - split);
    } else {
        launch_k(false, nullptr, k_exvol<Real>, nt, kBlock, s, n, want, 0, 1, off);
        if (n.prelist) {
            cudaStreamWaitEvent(L->side3, L->fork, 0);
            launch_k(false, L->join3, k_exvol_ext<Real>, kExtBlocks, 128, L->side3, n, 0, 1, 1);
            ++k;
        }
        launch_k(n.pdl, nullptr, k_exvol_ext<Real>, kExtBlocks, 128, s, n, 0, 1, 0);
        ++k;
        if (n.prelist) cudaStreamWaitEvent(s, L->join3, 0);
    }
    launch_k(n.pdl, n.pdl ? done : nullptr, k_exvol_fb_force<Real>, kFbForceBlocks, kBlock, s, n, n.fb_moments, n.fb_tickets);
    if (done && !n.pdl) cudaEventRecord(done, s);
    return k + 1;
}

template int launch_exvol_energy<MECH_EXVOL_REAL>(const DevNet<MECH_EXVOL_REAL>&, int, int, cudaStream_t, bool, const Lanes*);
template int launch_exvol_forces<MECH_EXVOL_REAL>(const DevNet<MECH_EXVOL_REAL>&, int, cudaStream_t, bool, const Lanes*);

}  // namespace mech
