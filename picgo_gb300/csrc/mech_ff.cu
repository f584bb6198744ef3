// Filament, linker/motor and boundary force-field kernels, the CG vector
// kernels and the per-replica finalizers of the device-resident minimizer.
//
// Reference behaviour restated here (paths relative to medyan-5.4.0/src):
//   FilamentStretchingHarmonic.cpp:185-275, FilamentBendingCosine.cpp:199-345,
//   LinkerStretchingHarmonic.cpp:191-293, MotorGhostStretchingHarmonic.cpp:234-340,
//   BoundaryCylinderRepulsionExp.cpp:27-110, ForceFieldManager.cpp:96-290,
//   CGMethod.hpp:238-373 and :826-1743, CGMethod.cpp:317-360,
//   MController.h:273-339 (recovery move).
//
// Filament forces are computed owner-side: a block loads a tile's beads (254 in
// mixed precision, 253 in FP64: kForceBeads) plus a two-bead halo into shared
// memory, evaluates every cylinder and bending triple touching them once, and
// each bead sums its own terms in a fixed order (the filament's, then the sparse
// force fields' through the CSR gather), so no floating-point atomics are used.
#include <cuda_runtime.h>

#include <algorithm>

#include "mech_bulk.cuh"
#include "mech_cg.cuh"
#include "mech_device.cuh"

namespace mech {

// ---------------------------------------------------------------------------
// helpers
// ---------------------------------------------------------------------------
// The three products of one bead, in the engine's precision.  The fused forms
// are written out so that a product rounds alike in whatever kernel it is
// formed: beta, and with it the trajectory, hangs on the last bits of F.F and
// F.Fprev (which round their first two products in different orders).
__device__ __forceinline__ double bead_dot(double a0, double a1, double a2, double b0, double b1, double b2) {
    return fma(a2, b2, fma(a1, b1, a0 * b0));
}
__device__ __forceinline__ float bead_dot(float a0, float a1, float a2, float b0, float b1, float b2) {
    return fmaf(a2, b2, fmaf(a1, b1, a0 * b0));
}
__device__ __forceinline__ double bead_dot_prev(const double F[3], double p0, double p1, double p2) {
    return fma(F[2], p2, fma(F[0], p0, F[1] * p1));
}
__device__ __forceinline__ float bead_dot_prev(const float F[3], float p0, float p1, float p2) {
    return bead_dot(F[0], F[1], F[2], p0, p1, p2);
}

// plane distance of a position (BoundaryElementImpl.h:49-53)
__device__ __forceinline__ double plane_dist_p(const double* pl, const Pos<double>& p) { return plane_dist(pl, p.x); }
__device__ __forceinline__ float plane_dist_p(const double* pl, const Pos<float>& p) {
    const float a = (float)pl[0], b = (float)pl[1], c = (float)pl[2], d = (float)pl[3];
    const float hi = a * p.h[0] + b * p.h[1] + c * p.h[2] + d;
    const float lo = a * p.l[0] + b * p.l[1] + c * p.l[2];
    return (hi + lo) / sqrtf(a * a + b * b + c * c);
}

// vector from the point at s1 on (c1, c2) to the point at s2 on (c3, c4)
// (LinkerStretchingHarmonic.cpp:200-216).  FP64: the interpolated points
// themselves, as the reference; mixed: the same vector from differences only,
// (c3 - c1) + s2 (c4 - c3) - s1 (c2 - c1).
__device__ __forceinline__ void bond_vector(const Pos<double>& c1, const Pos<double>& c2, const Pos<double>& c3,
                                            const Pos<double>& c4, double s1, double s2, double v[3]) {
    double p1[3], p2[3];
    lerp3(c1.x, c2.x, s1, p1);
    lerp3(c3.x, c4.x, s2, p2);
    v[0] = p2[0] - p1[0];
    v[1] = p2[1] - p1[1];
    v[2] = p2[2] - p1[2];
}
__device__ __forceinline__ void bond_vector(const Pos<float>& c1, const Pos<float>& c2, const Pos<float>& c3,
                                            const Pos<float>& c4, float s1, float s2, float v[3]) {
    float d31[3], d43[3], d21[3];
    pdiff(c3, c1, d31);
    pdiff(c4, c3, d43);
    pdiff(c2, c1, d21);
#pragma unroll
    for (int k = 0; k < 3; ++k) v[k] = fmaf(s2, d43[k], fmaf(-s1, d21[k], d31[k]));
}

// ---------------------------------------------------------------------------
// Conditions of the minimizer's conditional graph (GraphConds).
// ---------------------------------------------------------------------------
constexpr int kCondTrial = 2, kCondForce = 3;   // counter slots

// Which phases the replicas are in, read past L1 (other blocks wrote the
// states); every thread of one block calls it, thread 0 sets the handles.
// `head`: the kernel at the head of a loop body, which also counts bodies and
// decides whether the loop runs another one after this body.
template <typename Real>
__device__ void set_conditions(const DevNet<Real>& n, bool head, int phase_slot) {
    int tr = 0, fo = 0, host = 0;
    for (int r = threadIdx.x; r < n.R; r += blockDim.x) {
        const int ph = __ldcg(&n.st[r].phase);
        tr |= ph == PH_LS_TRIAL;
        fo |= ph == PH_FORCE;
        host |= ph >= PH_RECOVER;   // the recovery move is sequenced by the host
    }
    tr = __syncthreads_or(tr);
    fo = __syncthreads_or(fo);
    host = __syncthreads_or(host);
    if (threadIdx.x != 0) return;
    cudaGraphSetConditional(n.cond.trial, tr ? 1u : 0u);
    cudaGraphSetConditional(n.cond.force, fo ? 1u : 0u);
    if (phase_slot >= 0) n.cond.counter[phase_slot]++;
    if (head) {
        // the loop ends after this body when nothing is left to do on the
        // device, an error is latched or the body budget of the launch is spent
        const int bodies = ++n.cond.counter[0];
        const bool more = (tr | fo) && !host && __ldcg(n.err) == 0 && bodies < n.cond.cap;
        cudaGraphSetConditional(n.cond.loop, more ? 1u : 0u);
    }
}

// Zero the excluded-volume work-list counts for the next evaluation, once every
// kernel that reads them has ended (one thread).
template <typename Real>
__device__ __forceinline__ void zero_counts(const DevNet<Real>& n, bool force) {
    if (n.ev_list_count) *n.ev_list_count = 0;
    if (n.ev_fb_count) *n.ev_fb_count = 0;
    if (n.prelist && force) *n.ev_flist_count = 0;
}
// After an energy's per-replica reduction, which reads the fallback list: the last
// block zeroes the counts (a force evaluation's gather, behind the last reader,
// has done that: with 32 replicas the ticket took 1 us).  Then, after both, it
// sets the graph conditions when there are any.
template <typename Real>
__device__ void after_evaluation(const DevNet<Real>& n, int phase_slot, int* s_flag) {
    const bool force = phase_slot == kCondForce;
    if (force && !n.cond.on) return;
    if (gridDim.x == 1) __syncthreads();   // one replica: this block is the last, no ticket needed
    else if (!last_tile(n.gticket, 0, gridDim.x, s_flag)) return;
    if (threadIdx.x == 0 && !force) zero_counts(n, false);
    if (n.cond.on) set_conditions(n, false, phase_slot);
}

// The head of an unrolled graph (launch_graph_head).
__global__ void k_graph_head() {}

// The kernel at the head of every body of the minimizer's while loop.
template <typename Real>
__global__ void __launch_bounds__(kBlock) k_body_head(DevNet<Real> n) {
    MECH_TRACE_KERNEL(n, TK_BODY_HEAD);
    set_conditions(n, true, -1);
}

// ---------------------------------------------------------------------------
// FP64 engine: filament energy and forces.  Bound by the FP64 pipe (a warp's
// FP64 instruction holds its sub-partition's pipe for ~78 cycles), so what
// counts is FP64 instructions per bead: every cylinder's vector, length and
// reciprocal length is formed once and read by the bending terms on both of its
// ends, comparisons are made on the bits of the numbers, and the sums of a warp
// share the additions of their trees.
// ---------------------------------------------------------------------------
// Stretching + bending energy of the tile's own cylinders and triples.  1M
// beads: 86 us, against 121 us (66 FP64 instructions per bead) with each length
// formed two or three times and a tree per sum.
__global__ void __launch_bounds__(kBlock) k_fil_energy(DevNet<double> n, int want, int trial) {
    pdl_wait();      // the previous kernel of the main lane has finished
    MECH_TRACE_KERNEL(n, TK_FIL_ENERGY);
    __shared__ double xs[3][kFilTile + 2];    // beads begin - 1 .. end
    __shared__ double rs[4][kFilTile + 1];    // cylinders begin - 1 .. end - 1: vector, length
    __shared__ double dF[kFilTile];           // d . F of each bead (a new direction)
    __shared__ double sh[4 * kBlock / 32];
    const bool tr = trial != 0;
    const Tile t = fil_tile(n, blockIdx.x);
    const LaneState<double> s = lane_state(n, t.replica, want);
    if (!s.go) return;
    const Direction<double> dir = direction_of(n, s);
    const int T = t.end - t.begin;
    const double* X = n.x[s.xb];
    const bool pend = tr && dir.F;     // this pass forms the direction
    const bool backup = pend && n.st[t.replica].backupPending;
    double e[4] = {0.0, 0.0, 0.0, 0.0};   // stretching, bending, d . F
    for (int i = threadIdx.x; i < T + 2; i += blockDim.x) {
        const int b = t.begin - 1 + i;
        if (b < 0 || b >= n.nb) continue;
        Pos<double> p = load_pos(X, b);
        if (tr) {
            const bool own = i >= 1 && i <= T;
            double d[3];
            direction_at(dir, b, d);
            if (pend && own) {
                double* o = dir.out + 3 * (size_t)b;
                const double* F = dir.F + 3 * (size_t)b;
                o[0] = d[0];
                o[1] = d[1];
                o[2] = d[2];
                dF[i - 1] = bead_dot(d[0], d[1], d[2], F[0], F[1], F[2]);
                if (backup) store_pos(n.xbest, b, p);
            }
            p = moved(p, d, s.lambda);
            if (own) store_pos(n.x[s.xb ^ 1], b, p);   // materialize the owned trial position
        }
        xs[0][i] = p.x[0];
        xs[1][i] = p.x[1];
        xs[2][i] = p.x[2];
    }
    __syncthreads();
    const int i = threadIdx.x, j = t.begin + i;
    const int fl = i < T ? n.bflag[j] : 0;
    if (pend && i < T) e[2] = dF[i];
    double r2[3] = {0, 0, 0}, L2 = 0.0, ks = 0.0, l0 = 0.0, kb = 0.0, th = 0.0;
    if (fl & 1) {
        load_par(n.bpar, j, ks, l0, kb, th);
#pragma unroll
        for (int q = 0; q < 3; ++q) r2[q] = xs[q][i + 2] - xs[q][i + 1];
        L2 = sqrt(r2[0] * r2[0] + r2[1] * r2[1] + r2[2] * r2[2]);
        const double dl = L2 - l0;
        e[0] = 0.5 * ks * dl * dl;
#pragma unroll
        for (int q = 0; q < 3; ++q) rs[q][i + 1] = r2[q];
        rs[3][i + 1] = L2;
    }
    if (i == kFilTile - 32 && (n.bflag[t.begin] & 2)) {   // the cylinder that ends at the first bead
        double r[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) rs[q][0] = r[q] = xs[q][1] - xs[q][0];
        rs[3][0] = sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
    }
    __syncthreads();
    if ((fl & 3) == 3) {
        const double l1l2 = rs[0][i] * r2[0] + rs[1][i] * r2[1] + rs[2][i] * r2[2];
        e[1] = bend_energy_lengths(l1l2, rs[3][i], L2, kb, th);
    }
    if (n.terms && (fl & 1)) {
        n.terms[j] = e[0];
        n.terms[(size_t)n.nb + j] = e[1];
    }
    const double a = block_sums<4>(e, sh);
    if (threadIdx.x < 2) n.part_fil[4 * (size_t)blockIdx.x + threadIdx.x] = a;
    if (threadIdx.x == 2) n.part_df[blockIdx.x] = a;
}

// Filament forces of the tile's own beads (the sparse force fields' shares are
// added by k_force_gather once they are written), each cylinder's and triple's
// terms formed once, and each bead's sum in the reference's order (stretching
// of its two cylinders, bending of the three triples it is in): the FP64
// engine's minimizations amplify a changed rounding by up to ~1e8 over a hundred
// iterations, so the forces keep every operation.  A triple reads its
// cylinders' vectors and squared lengths instead of forming them again.
// Bound by the FP64 pipe, where a warp with three active lanes costs as much as
// a full one: a block of 256 beads has 259 cylinders and 258 triples, nine warps
// of each; no sum crosses a bead here, and a block takes 253 beads
// (kForceBeads), eight warps of each (1M beads: 214 -> 190 us).
__global__ void __launch_bounds__(kBlock) k_fil_force(DevNet<double> n, int want) {
    pdl_wait();      // the previous kernel of the main lane has finished
    MECH_TRACE_KERNEL(n, TK_FIL_FORCE);
    __shared__ double xs[3][kFilTile + 4];                          // beads begin - 2 .. end + 1
    __shared__ double rs[3][kFilTile + 3], Ls[kFilTile + 3];        // cylinders begin - 2 .. end: vector, L^2
    __shared__ double fs[3][kFilTile + 3];                          // their stretching forces on the second bead
    __shared__ double f1[3][kFilTile + 2], f2[3][kFilTile + 2];     // triples on begin - 1 .. end
    const Tile t = force_tile(n, blockIdx.x);
    const LaneState<double> s = lane_state(n, t.replica, want);
    if (!s.go) return;
    const int T = t.end - t.begin;
    const double* X = n.x[s.xb];
    for (int i = threadIdx.x; i < T + 4; i += blockDim.x) {
        const int b = t.begin - 2 + i;
        if (b < 0 || b >= n.nb) continue;
        const Pos<double> p = load_pos(X, b);
        xs[0][i] = p.x[0];
        xs[1][i] = p.x[1];
        xs[2][i] = p.x[2];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < T + 3; i += blockDim.x) {
        const int c = t.begin - 2 + i;
        double F[3] = {0, 0, 0};
        if (c >= 0 && c < n.nb && (n.bflag[c] & 1)) {
            const double2 kl = reinterpret_cast<const double2*>(n.bpar)[2 * (size_t)c];
            double r[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) rs[q][i] = r[q] = xs[q][i + 1] - xs[q][i];
            const double L2 = r[0] * r[0] + r[1] * r[1] + r[2] * r[2];
            Ls[i] = L2;
            const double L = sqrt(L2), invL = 1.0 / L, f0 = kl.x * (L - kl.y) * invL;
#pragma unroll
            for (int q = 0; q < 3; ++q) F[q] = -f0 * r[q];
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) fs[q][i] = F[q];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < T + 2; i += blockDim.x) {
        const int c = t.begin - 1 + i;   // cylinders c - 1, c at i, i + 1
        double a[3] = {0, 0, 0}, b[3] = {0, 0, 0};
        if (c >= 0 && c < n.nb && (n.bflag[c] & 3) == 3) {
            const double2 kt = reinterpret_cast<const double2*>(n.bpar)[2 * (size_t)c + 1];
            const double r1[3] = {rs[0][i], rs[1][i], rs[2][i]}, r2[3] = {rs[0][i + 1], rs[1][i + 1], rs[2][i + 1]};
            const double L1 = Ls[i], L2 = Ls[i + 1];
            const double l1l2 = r1[0] * r2[0] + r1[1] * r2[1] + r1[2] * r2[2];
            const double A = 1.0 / sqrt(L1 * L2);
            double x = l1l2 * A;
            const double B = x / L1, C = x / L2;
            double kk = kt.x;
            if (!theta_is_zero(kt.y)) {
                if (fabs(fabs(x) - 1.0) < 0.001) x = 0.999 * x;
                x = clamp_unit(x);
                const double sinp = sqrt(fmax(1.0 - x * x, 0.0));
                const double sinpmq = sinp * cos(kt.y) - x * sin(kt.y);
                kk = kt.x * sinpmq / sinp;
            }
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                a[q] = kk * (r2[q] * A - r1[q] * B);
                b[q] = kk * (r1[q] * A - r2[q] * C);
            }
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            f1[q][i] = a[q];
            f2[q][i] = b[q];
        }
    }
    __syncthreads();
    const int i = threadIdx.x;
    if (i < T) {
        double* Fo = n.f[s.fb ^ 1] + 3 * (size_t)(t.begin + i);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            double v = fs[q][i + 1];
            v += -fs[q][i + 2];
            v += f2[q][i];
            v += f1[q][i + 1] - f2[q][i + 1];
            v += -f1[q][i + 2];
            Fo[q] = v;
        }
    }
}

// ---------------------------------------------------------------------------
// Every bead adds its sparse contributions (contiguous, in the CSR order) to
// its filament force, then the CG partials: max |F|, F.F, F.Fprev per tile,
// reduced by k_finalize_force (a per-tile completion ticket on one address per
// replica would serialize thousands of atomics).  Each block takes
// kGatherTiles consecutive tiles and issues the loads of all of them before
// the reduction.  FP64 engine: FP64-pipe bound (43 us on 1M beads, 94 us with a
// tree per sum, and the maximum and the finiteness tests in FP64); the maximum
// is formed on the bits.  The mixed engine's
// version is k_force_gather_mx below.
// ---------------------------------------------------------------------------
constexpr int kGatherAhead = 4;   // contributions loaded together
// `acc` plus `count` contributions, 3 numbers apart from `g` on, in order.  The
// first are loaded together: one after another, each costs a round trip to L2.
template <typename Real, int N>
__device__ __forceinline__ void add_contributions(const Real* g, int count, Real (&acc)[N]) {
    Real v[kGatherAhead][N];
#pragma unroll
    for (int k = 0; k < kGatherAhead; ++k)
        if (k < count)
#pragma unroll
            for (int q = 0; q < N; ++q) v[k][q] = g[3 * k + q];
#pragma unroll
    for (int k = 0; k < kGatherAhead; ++k)
        if (k < count)
#pragma unroll
            for (int q = 0; q < N; ++q) acc[q] += v[k][q];
    for (int k = kGatherAhead; k < count; ++k)
#pragma unroll
        for (int q = 0; q < N; ++q) acc[q] += g[3 * (size_t)k + q];
}
template <typename Real>
__device__ __forceinline__ void gather_force(const DevNet<Real>& n, int b, int fb, Real F[3], Real& ff, Real& ffp) {
    Real* Fo = n.f[fb ^ 1] + 3 * (size_t)b;
    const Real* Fp = n.f[fb] + 3 * (size_t)b;
    Real acc[3] = {Fo[0], Fo[1], Fo[2]};
    const Real p0 = Fp[0], p1 = Fp[1], p2 = Fp[2];
    const int c0 = n.csr_off[b], c1 = n.csr_off[b + 1];
    add_contributions<Real, 3>(n.contrib + 3 * (size_t)c0, c1 - c0, acc);
#pragma unroll
    for (int q = 0; q < 3; ++q) Fo[q] = F[q] = acc[q];
    ff = bead_dot(F[0], F[1], F[2], F[0], F[1], F[2]);
    ffp = bead_dot_prev(F, p0, p1, p2);
}
// a non-finite component makes the bead's max infinite (fmax would drop a NaN)
__device__ __forceinline__ void gather_bead(const DevNet<float>& n, int b, int fb, float& mx, float& ff, float& ffp) {
    float F[3];
    gather_force(n, b, fb, F, ff, ffp);
    const bool fin = F[0] - F[0] == 0 && F[1] - F[1] == 0 && F[2] - F[2] == 0;
    mx = fin ? fmaxf(fmaxf(fabsf(F[0]), fabsf(F[1])), fabsf(F[2])) : INFINITY;
}
// the same on bits: infinity and NaN have the largest, cut to infinity's
__device__ __forceinline__ unsigned long long max_bits(const double F[3]) {
    return min(max(max(abs_bits(F[0]), abs_bits(F[1])), abs_bits(F[2])), 0x7ff0000000000000ULL);
}
// FP64, the beads of a warp together: an addition costs the warp the same for
// one lane as for 32, and few beads have contributions, so the components of
// those that have some are spread over the lanes (a third of the additions of a
// warp that adds three for every contribution of its busiest bead).  The gather
// of 1M beads 52.5 -> 40 us; not in a small network, where a block has an SM for
// itself and the detour through shared memory is 0.3 us of latency.
struct GatherWarp {
    double F[96];      // components of the beads with contributions
    int2 range[32];    // their first contribution and count
};
__device__ __forceinline__ void gather_warp(const DevNet<double>& n, int b, bool own, int fb, GatherWarp& s,
                                            unsigned long long& mx, double& ff, double& ffp) {
    const int lane = threadIdx.x & 31;
    double* Fo = n.f[fb ^ 1] + 3 * (size_t)b;
    const double* Fp = n.f[fb] + 3 * (size_t)b;
    double F[3] = {0, 0, 0}, p0 = 0, p1 = 0, p2 = 0;
    int c0 = 0, count = 0;
    if (own) {
        c0 = n.csr_off[b];
        count = n.csr_off[b + 1] - c0;
        F[0] = Fo[0];
        F[1] = Fo[1];
        F[2] = Fo[2];
        p0 = Fp[0];
        p1 = Fp[1];
        p2 = Fp[2];
    }
    const unsigned some = __ballot_sync(0xffffffffu, count > 0);
    if (some) {
        const int rank = __popc(some & ((1u << lane) - 1u)), items = 3 * __popc(some);
        if (count > 0) {
            s.range[rank] = make_int2(c0, count);
#pragma unroll
            for (int q = 0; q < 3; ++q) s.F[3 * rank + q] = F[q];
        }
        __syncwarp();
        for (int t = lane; t < items; t += 32) {
            const int e = t / 3;
            const int2 r = s.range[e];
            double acc[1] = {s.F[t]};
            add_contributions<double, 1>(n.contrib + 3 * (size_t)r.x + (t - 3 * e), r.y, acc);
            s.F[t] = acc[0];
        }
        __syncwarp();
        if (count > 0) {
#pragma unroll
            for (int q = 0; q < 3; ++q) F[q] = s.F[3 * rank + q];
        }
        __syncwarp();   // the next tile's beads use the same arrays
    }
    if (own) {
        Fo[0] = F[0];
        Fo[1] = F[1];
        Fo[2] = F[2];
        ff = bead_dot(F[0], F[1], F[2], F[0], F[1], F[2]);
        ffp = bead_dot_prev(F, p0, p1, p2);
        mx = max_bits(F);
    }
}

// NT tiles per block (DevNet::gtiles).  Four blocks on an SM (64 registers) hold
// 997 blocks of the 1M-bead network in two rounds; with three there were three,
// the last of them a fifth full (iteration 712 -> 706 us).
template <int NT>
__global__ void __launch_bounds__(kBlock, 4) k_force_gather(DevNet<double> n, int want) {
    pdl_wait();      // the force kernels have finished
    pdl_trigger();   // the next kernel of the main lane may be scheduled now
    MECH_TRACE_KERNEL(n, TK_GATHER);
    if (blockIdx.x == 0 && threadIdx.x == 0) zero_counts(n, true);   // their readers have finished
    __shared__ double sh[2 * NT * kBlock / 32];
    __shared__ unsigned long long s_mx[NT * kBlock / 32];
    __shared__ GatherWarp s_warp[NT > 1 ? kBlock / 32 : 1];
    const int t0 = blockIdx.x * NT;
    unsigned long long mx[NT];
    double v[2 * NT];   // F.F of each tile, then F.Fprev
    unsigned go = 0;
#pragma unroll
    for (int j = 0; j < NT; ++j) {
        mx[j] = 0;
        v[j] = v[NT + j] = 0.0;
        if (t0 + j >= n.n_ftiles) continue;
        const Tile t = fil_tile(n, t0 + j);
        const LaneState<double> s = lane_state(n, t.replica, want);
        if (!s.go) continue;
        go |= 1u << j;
        const int b = t.begin + threadIdx.x;
        if constexpr (NT > 1) {
            gather_warp(n, b, b < t.end, s.fb, s_warp[threadIdx.x >> 5], mx[j], v[j], v[NT + j]);
        } else if (b < t.end) {
            double F[3];
            gather_force(n, b, s.fb, F, v[0], v[1]);
            mx[0] = max_bits(F);
        }
    }
    if (!go) return;   // block-uniform
    const unsigned long long m = block_maxima<NT>(mx, s_mx);
    const double a = block_sums<2 * NT>(v, sh);
    if (threadIdx.x < 2 * NT) {
        const int j = threadIdx.x % NT;
        if (go >> j & 1) {
            double* slot = n.part_fil + 4 * (size_t)(t0 + j);
            if (threadIdx.x < NT) slot[0] = __longlong_as_double((long long)m);
            slot[1 + threadIdx.x / NT] = a;
        }
    }
}

// Mixed engine gather: 64 threads per tile, n.gtiles tiles per block, each
// thread taking 4 consecutive beads whose force records (4 x 12 B) move as three
// 16-byte vectors and whose contributions, contiguous too, are loaded up to
// kGatherAheadMx together, when the tile starts on a multiple of 4 beads (always,
// unless a replica before it has a bead count that is not; a partial group at
// the tile's end goes bead by bead); otherwise 4 beads strided by 64.  The
// block's partials combine, in warp order, the warps of each run of its tiles
// that belong to one replica, into the slot of the run's first tile (run_slot
// with stride n.gtiles).
constexpr int kGatherAheadMx = 8;
__global__ void __launch_bounds__(kBlock) k_force_gather_mx(DevNet<float> n, int want) {
    pdl_wait();      // the force kernels have finished
    static_assert(kFilTile == 256 && kBlock == 64 * kGatherTiles, "64 threads x 4 beads per tile");
    pdl_trigger();   // the next kernel of the main lane may be scheduled now
    MECH_TRACE_KERNEL(n, TK_GATHER_MX);
    if (blockIdx.x == 0 && threadIdx.x == 0) zero_counts(n, true);   // their readers have finished
    __shared__ float sh[8][5];   // per warp: F.F (hi, lo), F.Fprev (hi, lo), max
    __shared__ int s_go[kGatherTiles], s_rep[kGatherTiles];
    const int nt = blockDim.x >> 6;   // tiles of this block
    const int j = threadIdx.x >> 6, tt = threadIdx.x & 63;
    const int ti = blockIdx.x * nt + j;
    Tile t{-1, 0, 0, 0};
    bool go = false;
    int fb = 0;
    if (n.R == 1 && !lane_state(n, 0, want).go) return;
    if (ti < n.n_ftiles) {
        t = fil_tile(n, ti);
        const LaneState<float> s = lane_state(n, t.replica, want);
        go = s.go;
        fb = s.fb;
    }
    if (tt == 0) {
        s_go[j] = go;
        s_rep[j] = t.replica;
    }
    const int t0 = blockIdx.x * nt;
    FF aff, affp;
    float mx = 0.f;
    if (go) {   // uniform over the tile's two warps
        const int b0 = t.begin + 4 * tt;
        const bool vec_tile = (t.begin & 3) == 0;   // uniform over the tile
        if (vec_tile && b0 + 4 <= t.end) {
            float* Fo = n.f[fb ^ 1] + 3 * (size_t)b0;
            const float* Fp = n.f[fb] + 3 * (size_t)b0;
            const float4 u0 = reinterpret_cast<const float4*>(Fo)[0], u1 = reinterpret_cast<const float4*>(Fo)[1],
                         u2 = reinterpret_cast<const float4*>(Fo)[2];
            const float4 p0 = reinterpret_cast<const float4*>(Fp)[0], p1 = reinterpret_cast<const float4*>(Fp)[1],
                         p2 = reinterpret_cast<const float4*>(Fp)[2];
            float F[12] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w, u2.x, u2.y, u2.z, u2.w};
            const float P[12] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w, p2.x, p2.y, p2.z, p2.w};
            int off[5];
#pragma unroll
            for (int q = 0; q < 5; ++q) off[q] = n.csr_off[b0 + q];
            float g[kGatherAheadMx][3];
#pragma unroll
            for (int m = 0; m < kGatherAheadMx; ++m)
                if (off[0] + m < off[4])
#pragma unroll
                    for (int q = 0; q < 3; ++q) g[m][q] = n.contrib[3 * (size_t)(off[0] + m) + q];
#pragma unroll
            for (int m = 0; m < kGatherAheadMx; ++m) {
                const int c = off[0] + m;
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (c >= off[k] && c < off[k + 1])
#pragma unroll
                        for (int q = 0; q < 3; ++q) F[3 * k + q] += g[m][q];
            }
            if (off[4] - off[0] > kGatherAheadMx) {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    for (int c = max(off[k], off[0] + kGatherAheadMx); c < off[k + 1]; ++c) {
                        F[3 * k] += n.contrib[3 * (size_t)c];
                        F[3 * k + 1] += n.contrib[3 * (size_t)c + 1];
                        F[3 * k + 2] += n.contrib[3 * (size_t)c + 2];
                    }
            }
            reinterpret_cast<float4*>(Fo)[0] = make_float4(F[0], F[1], F[2], F[3]);
            reinterpret_cast<float4*>(Fo)[1] = make_float4(F[4], F[5], F[6], F[7]);
            reinterpret_cast<float4*>(Fo)[2] = make_float4(F[8], F[9], F[10], F[11]);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float* f = F + 3 * k;
                const bool fin = f[0] - f[0] == 0 && f[1] - f[1] == 0 && f[2] - f[2] == 0;
                mx = fmaxf(mx, fin ? fmaxf(fmaxf(fabsf(f[0]), fabsf(f[1])), fabsf(f[2])) : INFINITY);
                aff.add(bead_dot(f[0], f[1], f[2], f[0], f[1], f[2]));
                affp.add(bead_dot(f[0], f[1], f[2], P[3 * k], P[3 * k + 1], P[3 * k + 2]));
            }
        } else {
            // the partial group at the end of a vector tile, or a tile that
            // starts off the 4-bead grid: 4 beads strided by 64
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int b = vec_tile ? b0 + q : t.begin + tt + 64 * q;
                if (b < t.end) {
                    float m1, f1, f2;
                    gather_bead(n, b, fb, m1, f1, f2);
                    mx = fmaxf(mx, m1);
                    aff.add(f1);
                    affp.add(f2);
                }
            }
        }
    }
    FF sums[2] = {aff, affp};
    const int which = warp_pair_sums<2>(sums);   // lane 0: F.F, lane 16: F.Fprev
    const unsigned wm = __reduce_max_sync(0xffffffffu, __float_as_uint(mx));   // none negative: ordered like the bits
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 15) == 0) {
        sh[w][2 * which] = sums[0].h;
        sh[w][2 * which + 1] = sums[0].l;
        sh[w][4] = __uint_as_float(wm);
    }
    __syncthreads();
    const int j0 = threadIdx.x;
    if (j0 < nt && s_go[j0] && (j0 == 0 || s_rep[j0 - 1] != s_rep[j0])) {
        // thread j0 starts a run: its tile and the following tiles of the same
        // replica, their warps' pairs added in order to compensated sums
        FF f1, f2;
        float m = 0.f;
        for (int q = j0; q < nt && s_rep[q] == s_rep[j0]; ++q)
            for (int w = 2 * q; w < 2 * q + 2; ++w) {
                f1.add(sh[w][0]);
                f1.add(sh[w][1]);
                f2.add(sh[w][2]);
                f2.add(sh[w][3]);
                m = fmaxf(m, sh[w][4]);
            }
        float* p = reinterpret_cast<float*>(n.part_fil + 4 * (size_t)(t0 + j0));
        *reinterpret_cast<float4*>(p) = make_float4(m, f1.h, f1.l, f2.h);
        p[4] = f2.l;
    }
}

// One block per replica: max |F|, the dots and the CG step logic after the gather.
template <typename Real>
__global__ void __launch_bounds__(kBlock, 1) k_finalize_force(DevNet<Real> n, int want) {
    pdl_wait();      // the previous kernel of the main lane has finished
    pdl_trigger();   // the next kernel of the main lane may be scheduled now
    MECH_TRACE_KERNEL(n, TK_FIN_FORCE);
    __shared__ double sh[32 * 3];
    __shared__ int s_flag;
    const int r = blockIdx.x;
    CGState S;
    if (threadIdx.x == 0) S = n.st[r];   // issued together with the loads below
    const RepTiles rt = rep_tiles(n, r);
    if (replica_selected(n.st[r], want)) finalize_force(n, r, rt, S, sh);
    if (n.snap && threadIdx.x == 0) {   // what the host looks at after each graph
        if (S.phase == PH_DONE || S.phase >= PH_ERROR) n.snap[9 + r] = S.phase;
        if (r == 0) {
            const unsigned err = __ldcg(n.err);
            if (err) n.snap[0] = (int)err;
        }
    }
    after_evaluation(n, kCondForce, &s_flag);
}

// One block per replica: the energy reduction and the line-search step, after
// every kernel of the evaluation has written its partial sums.
template <typename Real>
__global__ void __launch_bounds__(kBlock, 1) k_finalize_energy(DevNet<Real> n, int want, int trial) {
    pdl_wait();      // every kernel of the evaluation has finished
    pdl_trigger();   // the next kernel of the main lane may be scheduled now
    MECH_TRACE_KERNEL(n, TK_FIN_ENERGY);
    __shared__ double sh[kFinSums * kBlock / 32];   // block_pair_sums<16>: 16 pairs of floats per warp
    __shared__ int s_flag;
    const int r = blockIdx.x;
    CGState S;
    if (threadIdx.x == 0) S = n.st[r];   // issued together with the loads below
    const RepTiles rt = rep_tiles(n, r);
    if (replica_selected(n.st[r], want)) finalize_energy(n, r, trial, rt, S, sh);
    after_evaluation(n, kCondTrial, &s_flag);
}

// ---------------------------------------------------------------------------
// Mixed engine: persistent, barrier-free filament kernels.  Each block walks
// `ptiles` consecutive tiles; every thread owns one bead per tile and
// recomputes in single precision the few neighbouring stretching and bending
// terms it needs (cheaper than staging through shared memory at the FP32
// rate), keeps compensated sums in registers across tiles, and the block
// reduces once per run of tiles of the same replica.
// ---------------------------------------------------------------------------


// Store a run's compensated partial sums as (hi, lo) pairs in the slot of its
// first tile; the reduction kernel that follows the evaluation reads them.
// a: stretching, bending, d . F and, with a second trial, its stretching and bending.
template <int N>
__device__ __forceinline__ void write_run(const DevNet<float>& n, int first, const FF (&a)[N], float* sh) {
    constexpr int P = N <= 4 ? 4 : 8;   // the packed trees take a power of two
    FF v[P];
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = a[k];
    const FF s = block_pair_sums<P>(v, sh);
    const int k = threadIdx.x;
    if (k < N)
        store_pair(k == 2 ? n.part_df + first : n.part_fil + 4 * (size_t)first + (k < 2 ? k : k - 1), s.h, s.l);
    __syncthreads();   // `sh` may be used again
}

// ---------------------------------------------------------------------------
// Mixed engine, bulk-staged filament energy: a persistent walk over runs of
// tiles with run-start partial slots (see write_run), where each selected
// tile's positions (with a one-bead halo),
// constants, flags and (for a trial) search direction arrive in shared memory
// by cp.async.bulk on an mbarrier ring, so a block keeps several
// ~14-18 KB transfers in flight instead of per-thread dependent loads.  Ranges
// are rounded outward to the 16-byte copy granularity; the bead arrays are
// allocated with the padding that rounding needs.
// ---------------------------------------------------------------------------
constexpr int kBulkStages = 3;                // forces
// Energy: with the forces of a new direction staged too, three stages would
// leave room for three blocks on an SM instead of four.  Staged forces and
// stores in whole vectors: a two-trial pass that forms the direction 46.9 -> 41.7
// us on 1M beads, an iteration of the 1M-cylinder network 117.3 -> 115.5 us.
constexpr int kEnergyStages = 2;
constexpr int kBulkXBeads = kFilTile + 4;    // tile + 1-bead halo, even-aligned ends
constexpr int kBulkDBeads = kFilTile + 8;    // tile + halo, 4-bead aligned ends
constexpr int kBulkFlags = kFilTile + 32;    // tile + halo, 16-byte aligned ends
constexpr int kBulkWaitLimit = 1 << 22;      // mbarrier polls before a stage counts as lost

struct __align__(16) EnergyStage {
    float x[6 * kBulkXBeads];      // float-float positions, beads [xs, xe)
    float4 par[kFilTile];          // k_str, l0, k_bend, theta0, beads [tb, te)
    float d[3 * kBulkDBeads];      // search direction, beads [ds, de)
    float f[3 * kBulkDBeads];      // forces of a new direction, the same beads
    uint8_t flag[kBulkFlags];      // bead flags, beads [fs, fe)
};

struct StageRange {
    int xs, xe, ds, de, fs, fe;
};
// Staged ranges of tile [tb, te) with `halo` beads each side, clamped to the
// network and rounded outward: positions to even beads (24 B each), the
// direction to multiples of 4 beads (12 B), flags to 16 beads (1 B).
__device__ __forceinline__ StageRange stage_range(int tb, int te, int nb, int halo) {
    StageRange r;
    const int lo = max(tb - halo, 0), hi = min(te + halo, nb);
    r.xs = lo & ~1;
    r.xe = (hi + 1) & ~1;
    r.ds = lo & ~3;
    r.de = (hi + 3) & ~3;
    r.fs = lo & ~15;
    r.fe = (hi + 15) & ~15;
    return r;
}

// A block's tile descriptors, read once at kernel start (one thread per tile)
// so the producing thread issues copies without chasing global pointers:
// (begin, end, replica, bits) with bit 0 = selected by this launch, bits 1-2 =
// xbuf, bit 3 = fbuf of the tile's replica, bit 4 = its pass has a second trial,
// bit 5 = dPending, 6 = dIsF, 7 = dbuf, 8 = backupPending, plus that replica's
// lambda and beta.  A
// replica's state cannot change while this block still holds unprocessed
// tiles of it (its finalizer waits for every tile), so the copies stay valid.
constexpr int kBulkMaxTiles = kFilBulkMaxTiles;

__device__ __forceinline__ int4 descriptor(const Tile& t, const LaneState<float>& s, int backup) {
    return make_int4(t.begin, t.end, t.replica,
                     (s.go ? 1 : 0) | (s.xb << 1) | (s.fb << 3) | (s.dual ? 16 : 0) | (s.dPending << 5) |
                         (s.dIsF << 6) | (s.dbuf << 7) | (backup << 8));
}
__device__ __forceinline__ void load_descriptors(const DevNet<float>& n, bool force, int t0, int nt, int want,
                                                 int4* desc, float2* step) {
    for (int k = threadIdx.x; k < nt; k += blockDim.x) {
        const Tile t = force ? force_tile(n, t0 + k) : fil_tile(n, t0 + k);
        const LaneState<float> s = lane_state(n, t.replica, want);
        desc[k] = descriptor(t, s, n.st[t.replica].backupPending);
        step[k] = make_float2(s.lam, s.beta);
    }
}

// The direction that a tile's pass starts from (direction_of on descriptor bits).
__device__ __forceinline__ const float* staged_direction(const DevNet<float>& n, int bits) {
    const int fb = (bits >> 3) & 1;
    return bits & 64 ? n.f[bits & 32 ? fb ^ 1 : fb] : n.d[(bits >> 7) & 1];
}

// Issue the copies of a tile into stage `st` (thread 0).  A range that fails
// the alignment check is not copied: the barrier is completed without it and
// the error word records it.
__device__ void issue_energy_stage(const DevNet<float>& n, int4 t, bool tr, EnergyStage* st, uint64_t* bar) {
    const float* X = n.x[(t.w >> 1) & 3];
    const StageRange rg = stage_range(t.x, t.y, n.nb, 1);
    const unsigned vec = 12u * (unsigned)(rg.de - rg.ds);
    const void* src[5] = {X + 6 * (size_t)rg.xs, n.bpar + 4 * (size_t)t.x, n.bflag + rg.fs,
                          staged_direction(n, t.w) + 3 * (size_t)rg.ds, n.f[(t.w >> 3) & 1] + 3 * (size_t)rg.ds};
    void* dst[5] = {st->x, st->par, st->flag, st->d, st->f};
    const unsigned bytes[5] = {24u * (unsigned)(rg.xe - rg.xs), 16u * (unsigned)(t.y - t.x), (unsigned)(rg.fe - rg.fs),
                               tr ? vec : 0u, tr && (t.w & 32) ? vec : 0u};
    unsigned total = 0;
    bool ok = true;
    for (int k = 0; k < 5; ++k) {
        if (!bytes[k]) continue;
        if (!aligned16(src[k], bytes[k]) || !aligned16(dst[k], bytes[k])) ok = false;
        total += bytes[k];
    }
    fence_proxy_async_smem();
    if (!ok) {
        atomicOr(n.err, 16u);
        mbar_arrive_expect_tx(bar, 0);
        return;
    }
    mbar_arrive_expect_tx(bar, total);
    for (int k = 0; k < 5; ++k)
        if (bytes[k]) bulk_copy_g2s(dst[k], src[k], bytes[k], bar);
}

// True in every thread when a launch selects no replica of the block's tile
// range [t0, t1): tiles are ordered by replica, so a range whose first and
// last tiles share a replica belongs to it alone.  The block then exits before
// any barrier or descriptor setup.
__device__ __forceinline__ bool idle_range(const DevNet<float>& n, const Tile* tiles, int t0, int t1, int want,
                                           int* s_flag) {
    if (n.R == 1) return t1 <= t0 || !lane_state(n, 0, want).go;   // the same in every thread
    if (threadIdx.x == 0) {
        int idle = t1 <= t0;
        if (!idle) {
            const int ra = tiles[t0].replica, rb = tiles[t1 - 1].replica;
            idle = ra == rb && !replica_selected(n.st[ra], want);
        }
        *s_flag = idle;
    }
    __syncthreads();
    return *s_flag != 0;
}

// `count` floats from shared to consecutive global memory, by the whole block,
// in the widest vectors that both allow (16 bytes in a single network, 8 or 4
// where a replica before has a bead count that is not a multiple of 4; a record
// of 12 or 24 bytes per thread takes three store instructions that each touch
// all its sectors).
template <typename Vec>
__device__ __forceinline__ void store_vectors(float* dst, const float* src, int count) {
    constexpr int W = sizeof(Vec) / sizeof(float);
    const int whole = count / W;
    for (int k = threadIdx.x; k < whole; k += blockDim.x)
        reinterpret_cast<Vec*>(dst)[k] = reinterpret_cast<const Vec*>(src)[k];
    const int k = whole * W + threadIdx.x;
    if (k < count) dst[k] = src[k];
}
__device__ __forceinline__ void store_records(float* dst, const float* src, int count) {
    const unsigned off = (unsigned)(reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src));
    if ((off & 15u) == 0) store_vectors<float4>(dst, src, count);
    else if ((off & 7u) == 0) store_vectors<float2>(dst, src, count);
    else store_vectors<float>(dst, src, count);
}

__global__ void __launch_bounds__(kBlock, 4) k_fil_energy_bulk(DevNet<float> n, int want, int trial) {
    pdl_wait();      // the previous kernel of the main lane has finished
    MECH_TRACE_KERNEL(n, TK_FIL_ENERGY_BULK);
    __shared__ EnergyStage stage[kEnergyStages];
    __shared__ __align__(8) uint64_t bar[kEnergyStages];
    __shared__ int4 s_desc[kBulkMaxTiles];
    __shared__ float2 s_step[kBulkMaxTiles];
    __shared__ float sh[2 * 8 * kBlock / 32];   // block_pair_sums<8>
    __shared__ __align__(16) float s_mv[6 * kBulkXBeads];   // the staged beads moved to a trial
    __shared__ __align__(16) float s_d[3 * kFilTile];       // the tile's new direction
    __shared__ int s_abort;
    const int t0 = blockIdx.x * n.ptiles[0], t1 = min(t0 + n.ptiles[0], n.n_ftiles);
    const int nt = t1 - t0;
    const bool tr = trial != 0;
    if (idle_range(n, n.ftile, t0, t1, want, &s_abort)) return;
    if (threadIdx.x == 0) {
        for (int k = 0; k < kEnergyStages; ++k) mbar_init(&bar[k], 1);
        mbar_init_fence();
        s_abort = 0;
    }
    if (nt > kBulkMaxTiles) {   // the launch geometry caps tiles per block; refuse rather than overrun
        if (threadIdx.x == 0) atomicOr(n.err, 16u);
        return;
    }
    load_descriptors(n, false, t0, nt, want, s_desc, s_step);
    __syncthreads();
    // producer state (thread 0): next tile to consider, copies issued
    int pi = 0, issued = 0;
    if (threadIdx.x == 0) {
        for (; pi < nt && issued < kEnergyStages; ++pi)
            if (s_desc[pi].w & 1) {
                issue_energy_stage(n, s_desc[pi], tr, &stage[issued % kEnergyStages], &bar[issued % kEnergyStages]);
                ++issued;
            }
    }
    // a pass with a second trial: energies at lambda into slots 0, 1 of the run
    // and at lambda / 2 into slots 2, 3; trial positions into the two buffers
    // after the current one
    bool dual = false;
    int cur = -1, first = 0, cnt = 0, xb = 0, j = 0;
    bool go = false;
    bool pend = false;   // the pass forms the direction F + beta d
    float lf = 0.f, beta = 0.f;
    FF es, eb, es2, eb2, df;
    auto flush = [&]() {
        if (dual) {
            FF a[5] = {es, eb, df, es2, eb2};
            write_run(n, first, a, sh);
        } else {
            FF a[3] = {es, eb, df};
            write_run(n, first, a, sh);
        }
    };
    for (int k = 0; k < nt; ++k) {
        const int4 t = s_desc[k];
        if (t.z != cur) {
            if (cnt) flush();
            cur = t.z;
            first = t0 + k;
            cnt = 0;
            es = FF();
            eb = FF();
            es2 = FF();
            eb2 = FF();
            df = FF();
            go = t.w & 1;
            xb = (t.w >> 1) & 3;
            dual = second_trial(trial, t.w & 16);
            pend = tr && (t.w & 32);
            lf = s_step[k].x;
            beta = s_step[k].y;
        }
        if (!go) continue;
        ++cnt;
        const int sidx = j % kEnergyStages;
        const int b = t.x + threadIdx.x;
        const StageRange rg = stage_range(t.x, t.y, n.nb, 1);
        const bool own = b < t.y;
        if (!mbar_wait_bounded(&bar[sidx], (unsigned)((j / kEnergyStages) & 1), kBulkWaitLimit)) {
            atomicOr(n.err, 32u);
            s_abort = 1;
        }
        const EnergyStage& S = stage[sidx];
        int fl = 0;
        float4 pr = make_float4(0.f, 0.f, 0.f, 0.f);
        if (own) {
            fl = S.flag[b - rg.fs];
            pr = S.par[b - t.x];
        }
        // one trial per pass of this loop (two in a two-trial pass: lambda,
        // then lambda / 2, exact in float).  For a trial the block first moves
        // every staged bead once (tile and halo) into shared memory, so each
        // bead's neighbours are read, not moved again by every thread that
        // needs them; a plain evaluation reads the staged positions directly.
#pragma unroll 1
        for (int ch = 0; ch < (dual ? 2 : 1); ++ch) {
            const float* P = S.x;
            if (tr) {
                const float lch = ch ? 0.5f * lf : lf;
                for (int q = threadIdx.x; q < rg.xe - rg.xs; q += blockDim.x) {
                    const Pos<float> p = load_pos(S.x, q);
                    const int bq = rg.xs + q, dq = 3 * (bq - rg.ds);
                    float d[3] = {S.d[dq], S.d[dq + 1], S.d[dq + 2]};
                    if (pend) {
                        const float F[3] = {S.f[dq], S.f[dq + 1], S.f[dq + 2]};
#pragma unroll
                        for (int m = 0; m < 3; ++m) d[m] = new_direction(F[m], beta, d[m]);
                        if (!ch && bq >= t.x && bq < t.y) {   // the tile's own bead: the direction, d . F, the backup
                            float* o = s_d + 3 * (bq - t.x);
                            o[0] = d[0];
                            o[1] = d[1];
                            o[2] = d[2];
                            df.add(bead_dot(d[0], d[1], d[2], F[0], F[1], F[2]));
                            if (t.w & 256) store_pos(n.xbest, bq, p);
                        }
                    }
                    store_pos(s_mv, q, moved(p, d, lch));
                }
                __syncthreads();
                P = s_mv;
                // materialize the owned trial positions and the new direction
                store_records(n.x[(xb + 1 + ch) % 3] + 6 * (size_t)t.x, s_mv + 6 * (t.x - rg.xs), 6 * (t.y - t.x));
                if (pend && !ch)
                    store_records(n.d[((t.w >> 7) & 1) ^ 1] + 3 * (size_t)t.x, s_d, 3 * (t.y - t.x));
            }
            if (own) {
                const Pos<float> p0 = load_pos(P, b - rg.xs);
                if (fl & 1) {
                    const Pos<float> pp = load_pos(P, b + 1 - rg.xs);
                    float r2[3];
                    pdiff(pp, p0, r2);
                    const float ts = stretch_energy<float>(r2[0], r2[1], r2[2], pr.x, pr.y);
                    if (ch) es2.add(ts);
                    else es.add(ts);
                    float tb = 0.f;
                    if (fl & 2) {
                        const Pos<float> pm = load_pos(P, b - 1 - rg.xs);
                        float r1[3];
                        pdiff(p0, pm, r1);
                        tb = bend_energy<float>(r1, r2, pr.z, pr.w);
                        if (ch) eb2.add(tb);
                        else eb.add(tb);
                    }
                    if (n.terms && !ch) {
                        n.terms[b] = ts;
                        n.terms[(size_t)n.nb + b] = tb;
                    }
                }
            }
            if (tr) __syncthreads();   // s_mv is refilled by the next trial or tile
        }
        ++j;
        __syncthreads();   // stage sidx fully read
        if (s_abort) break;
        if (threadIdx.x == 0) {
            for (; pi < nt; ++pi)
                if (s_desc[pi].w & 1) {
                    issue_energy_stage(n, s_desc[pi], tr, &stage[issued % kEnergyStages], &bar[issued % kEnergyStages]);
                    ++issued;
                    ++pi;
                    break;
                }
        }
    }
    if (s_abort) {
        // drain: copies still in flight must land before the block's shared memory is released
        if (threadIdx.x == 0)
            for (int q = max(j - 1, 0); q < issued; ++q)
                mbar_wait_bounded(&bar[q % kEnergyStages], (unsigned)((q / kEnergyStages) & 1), kBulkWaitLimit);
        return;
    }
    if (cnt) flush();
}


// ---------------------------------------------------------------------------
// Mixed engine, bulk-staged filament forces: the same walk (k_fil_force_bulk).
// ---------------------------------------------------------------------------
constexpr int kBulkFXBeads = kFilTile + 8;    // tile + 2-bead halo, even-aligned ends
constexpr int kBulkFPar = kFilTile + 4;       // constants of beads tb - 1 .. te

struct __align__(16) ForceStage {
    float x[6 * kBulkFXBeads];
    float4 par[kBulkFPar];
    uint8_t flag[kBulkFlags];
};

struct ForceRange {
    int xs, xe, ps, pe, fs, fe;
};
__device__ __forceinline__ ForceRange force_range(int tb, int te, int nb) {
    ForceRange r;
    const int lo2 = max(tb - 2, 0), hi2 = min(te + 2, nb);
    r.xs = lo2 & ~1;
    r.xe = (hi2 + 1) & ~1;
    r.ps = max(tb - 1, 0);
    r.pe = min(te + 1, nb);
    r.fs = lo2 & ~15;
    r.fe = (hi2 + 15) & ~15;
    return r;
}

__device__ void issue_force_stage(const DevNet<float>& n, int4 t, ForceStage* st, uint64_t* bar) {
    const float* X = n.x[(t.w >> 1) & 3];
    const ForceRange rg = force_range(t.x, t.y, n.nb);
    const void* src[3] = {X + 6 * (size_t)rg.xs, n.bpar + 4 * (size_t)rg.ps, n.bflag + rg.fs};
    void* dst[3] = {st->x, st->par, st->flag};
    const unsigned bytes[3] = {24u * (unsigned)(rg.xe - rg.xs), 16u * (unsigned)(rg.pe - rg.ps),
                               (unsigned)(rg.fe - rg.fs)};
    unsigned total = 0;
    bool ok = true;
    for (int k = 0; k < 3; ++k) {
        if (!bytes[k]) continue;
        if (!aligned16(src[k], bytes[k]) || !aligned16(dst[k], bytes[k])) ok = false;
        total += bytes[k];
    }
    fence_proxy_async_smem();
    if (!ok) {
        atomicOr(n.err, 16u);
        mbar_arrive_expect_tx(bar, 0);
        return;
    }
    mbar_arrive_expect_tx(bar, total);
    for (int k = 0; k < 3; ++k)
        if (bytes[k]) bulk_copy_g2s(dst[k], src[k], bytes[k], bar);
}

// Mixed engine, bulk-staged filament forces: each selected tile's positions
// (two-bead halo), the constants and flags of its beads and their neighbours
// arrive by cp.async.bulk like k_fil_energy_bulk; every bead's filament force
// is written to the force buffer, where k_force_gather adds the bead's sparse
// contributions and forms the CG partials.  A tile is 254 beads (kForceBeads):
// with 256 the block's first warp ran the term phase a second time for the two
// slots beyond, and the other seven waited for it (iteration of the 1M-cylinder
// network 121.1 -> 119.6 us, of 32 replicas 85.5 -> 84.4 us).
__global__ void __launch_bounds__(kBlock) k_fil_force_bulk(DevNet<float> n, int want) {
    pdl_wait();      // the previous kernel of the main lane has finished
    MECH_TRACE_KERNEL(n, TK_FIL_FORCE_BULK);
    __shared__ ForceStage stage[kBulkStages];
    __shared__ __align__(8) uint64_t bar[kBulkStages];
    __shared__ int4 s_desc[kBulkMaxTiles];
    __shared__ float2 s_step[kBulkMaxTiles];
    __shared__ int s_abort;
    // per tile: stretching force of each cylinder (q, q + 1) and the two bending
    // terms of each triple centred on q, for q = tile begin - 1 .. tile end
    __shared__ float s_st[kFilTile + 2][3], s_a1[kFilTile + 2][3], s_a2[kFilTile + 2][3];
    const int t0 = blockIdx.x * n.ptiles[1], t1 = min(t0 + n.ptiles[1], n.n_force_tiles);
    const int nt = t1 - t0;
    if (idle_range(n, n.ftile_force, t0, t1, want, &s_abort)) return;
    if (threadIdx.x == 0) {
        for (int k = 0; k < kBulkStages; ++k) mbar_init(&bar[k], 1);
        mbar_init_fence();
        s_abort = 0;
    }
    if (nt > kBulkMaxTiles) {   // the launch geometry caps tiles per block; refuse rather than overrun
        if (threadIdx.x == 0) atomicOr(n.err, 16u);
        return;
    }
    load_descriptors(n, true, t0, nt, want, s_desc, s_step);
    __syncthreads();
    int pi = 0, issued = 0;
    if (threadIdx.x == 0) {
        for (; pi < nt && issued < kBulkStages; ++pi)
            if (s_desc[pi].w & 1) {
                issue_force_stage(n, s_desc[pi], &stage[issued % kBulkStages], &bar[issued % kBulkStages]);
                ++issued;
            }
    }
    int j = 0;
    for (int k = 0; k < nt; ++k) {
        const int4 t = s_desc[k];
        if (!(t.w & 1)) continue;
        const int fb = (t.w >> 3) & 1;
        const int sidx = j % kBulkStages;
        if (!mbar_wait_bounded(&bar[sidx], (unsigned)((j / kBulkStages) & 1), kBulkWaitLimit)) {
            atomicOr(n.err, 32u);
            s_abort = 1;
        }
        const ForceStage& S = stage[sidx];
        const ForceRange rg = force_range(t.x, t.y, n.nb);
        // every stretching and bending term touching the tile, once: term slot i
        // belongs to bead q = t.x - 1 + i (the cylinder (q, q + 1) and the triple
        // centred on q), for the tile and one halo bead on each side
        for (int i = threadIdx.x; i < t.y - t.x + 2; i += blockDim.x) {
            const int q = t.x - 1 + i;
            if (q < 0 || q >= n.nb) continue;
            const int fq = S.flag[q - rg.fs];
            if (!(fq & 1)) continue;
            const Pos<float> c0 = load_pos(S.x, q - rg.xs), c1 = load_pos(S.x, q + 1 - rg.xs);
            const float4 pq = S.par[q - rg.ps];
            float rp[3], st[3];
            pdiff(c1, c0, rp);
            stretch_force<float>(rp[0], rp[1], rp[2], pq.x, pq.y, st);
            s_st[i][0] = st[0]; s_st[i][1] = st[1]; s_st[i][2] = st[2];
            if (fq & 2) {
                const Pos<float> cm = load_pos(S.x, q - 1 - rg.xs);
                float rm[3], a1[3], a2[3];
                pdiff(c0, cm, rm);
                bend_force<float>(rm, rp, pq.z, pq.w, a1, a2);
                s_a1[i][0] = a1[0]; s_a1[i][1] = a1[1]; s_a1[i][2] = a1[2];
                s_a2[i][0] = a2[0]; s_a2[i][1] = a2[1]; s_a2[i][2] = a2[2];
            }
        }
        __syncthreads();
        const int b = t.x + threadIdx.x;
        if (b < t.y) {
            const int f0 = S.flag[b - rg.fs];
            const int fm = (f0 & 2) ? S.flag[b - 1 - rg.fs] : 0;
            const int fp = (f0 & 1) ? S.flag[b + 1 - rg.fs] : 0;
            const int i = threadIdx.x + 1;   // this bead's term slot
            // stretching: cylinder (b-1, b) then (b, b+1); bending: triples centred on b-1, b, b+1
            float F[3] = {0.f, 0.f, 0.f};
            if (f0 & 2) { F[0] += s_st[i - 1][0]; F[1] += s_st[i - 1][1]; F[2] += s_st[i - 1][2]; }
            if (f0 & 1) { F[0] += -s_st[i][0]; F[1] += -s_st[i][1]; F[2] += -s_st[i][2]; }
            if ((f0 & 2) && (fm & 2)) { F[0] += s_a2[i - 1][0]; F[1] += s_a2[i - 1][1]; F[2] += s_a2[i - 1][2]; }
            if ((f0 & 3) == 3) {
                F[0] += s_a1[i][0] - s_a2[i][0];
                F[1] += s_a1[i][1] - s_a2[i][1];
                F[2] += s_a1[i][2] - s_a2[i][2];
            }
            if ((f0 & 1) && (fp & 1)) { F[0] += -s_a1[i + 1][0]; F[1] += -s_a1[i + 1][1]; F[2] += -s_a1[i + 1][2]; }
            float* Fo = n.f[fb ^ 1] + 3 * (size_t)b;
            Fo[0] = F[0];
            Fo[1] = F[1];
            Fo[2] = F[2];
        }
        ++j;
        __syncthreads();   // stage sidx fully read
        if (s_abort) break;
        if (threadIdx.x == 0) {
            for (; pi < nt; ++pi)
                if (s_desc[pi].w & 1) {
                    issue_force_stage(n, s_desc[pi], &stage[issued % kBulkStages], &bar[issued % kBulkStages]);
                    ++issued;
                    ++pi;
                    break;
                }
        }
    }
    if (s_abort && threadIdx.x == 0)   // drain copies still in flight before shared memory is released
        for (int q = max(j - 1, 0); q < issued; ++q)
            mbar_wait_bounded(&bar[q % kBulkStages], (unsigned)((q / kBulkStages) & 1), kBulkWaitLimit);
}

// ---------------------------------------------------------------------------
// linker, motor and boundary interactions (energy or force contributions)
// ---------------------------------------------------------------------------
template <typename Real>
__global__ void __launch_bounds__(kBlock) k_bond_bnd(DevNet<Real> n, int want, int trial, int force, int n_lm_tiles,
                                                     int ev_tiles) {
    pdl_wait();      // the reduction before this evaluation has finished
    MECH_TRACE_KERNEL(n, TK_BOND);
    __shared__ double sh[32];   // block_pair_sums<2>: 32 floats
    const int ti = blockIdx.x < n_lm_tiles ? blockIdx.x : blockIdx.x + ev_tiles;
    int kind;
    const Tile t = sparse_tile(n, ti, &kind);
    const LaneState<Real> s = lane_state(n, t.replica, want);
    if (!s.go) return;
    const Direction<Real> dir = direction_of(n, s);
    const Real* X = n.x[s.xb];
    const bool tr = trial != 0;
    // a pass with a second trial also evaluates the energy at lambda / 2 (mixed engine)
    const bool dual = sizeof(Real) == 4 && !force && second_trial(trial, s.dual);
    auto pos = [&](int b) -> Pos<Real> { return bead_at(X, dir, b, tr, s.lam); };
    const Real lh = (Real)0.5 * s.lam;
    auto pos2 = [&](int b) -> Pos<Real> { return bead_at(X, dir, b, true, lh); };   // the second trial
    const int i = t.begin + threadIdx.x;
    Real e = 0, e2 = 0;
    if (i < t.end) {
        if (kind == K_BOUNDARY) {
            const int b = n.bb_bead[i];
            const double* pl = n.planes + 4 * n.bb_plane[i];
            const Pos<Real> p = pos(b);
            const Real rr = plane_dist_p(pl, p);
            const Real K = n.bb_k[i], sl = n.bb_slen[i];
            const Real R = -rr / sl;
            const Real ex = exp(R);
            if (!force) {
                e = K * ex;
                if (dual) {
                    const Real rr2 = plane_dist_p(pl, pos2(b));
                    e2 = K * exp(-rr2 / sl);
                }
            } else {
                const Real f0 = K * ex / sl;
                Real* c = slot_ptr(n, n.slot_base[K_BOUNDARY] + i);
                c[0] = f0 * (Real)pl[0];
                c[1] = f0 * (Real)pl[1];
                c[2] = f0 * (Real)pl[2];
            }
        } else {
            const bool lk = kind == K_LINKER;
            const int4 bs = lk ? n.lk_bead[i] : n.mt_bead[i];
            const Real k = lk ? n.lk_k[i] : n.mt_k[i];
            const Real l0 = lk ? n.lk_l0[i] : n.mt_l0[i];
            const Real s1 = lk ? n.lk_s1[i] : n.mt_s1[i];
            const Real s2 = lk ? n.lk_s2[i] : n.mt_s2[i];
            const Pos<Real> c1 = pos(bs.x), c2 = pos(bs.y), c3 = pos(bs.z), c4 = pos(bs.w);
            Real v[3];
            bond_vector(c1, c2, c3, c4, s1, s2, v);
            const Real lx = v[0], ly = v[1], lz = v[2];
            const Real dist = sqrt(lx * lx + ly * ly + lz * lz);
            if (!force) {
                const Real dd = dist - l0;
                e = (Real)0.5 * k * dd * dd;
                if (dual) {
                    Real w[3];
                    bond_vector(pos2(bs.x), pos2(bs.y), pos2(bs.z), pos2(bs.w), s1, s2, w);
                    const Real d2 = sqrt(w[0] * w[0] + w[1] * w[1] + w[2] * w[2]) - l0;
                    e2 = (Real)0.5 * k * d2 * d2;
                }
            } else {
                const Real invL = (Real)1 / dist;
                const Real f0 = k * (dist - l0) * invL;
                const Real Fl[3] = {-f0 * lx, -f0 * ly, -f0 * lz};
                const int sb = n.slot_base[kind] + 4 * i;
                Real* ca = slot_ptr(n, sb);
                Real* cb = slot_ptr(n, sb + 1);
                Real* cc = slot_ptr(n, sb + 2);
                Real* cd = slot_ptr(n, sb + 3);
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    ca[q] = -Fl[q] * ((Real)1 - s1);
                    cb[q] = -Fl[q] * (s1);
                    cc[q] = Fl[q] * ((Real)1 - s2);
                    cd[q] = Fl[q] * (s2);
                }
                (lk ? n.lk_sf : n.mt_sf)[i] = (double)(f0 / invL);
            }
        }
    }
    if (!force) {
        if constexpr (sizeof(Real) == 4) {
            if (dual) {
                FF a[2];
                a[0].h = e;
                a[1].h = e2;
                const FF se = block_pair_sums<2>(a, reinterpret_cast<float*>(sh));
                if (threadIdx.x < 2) store_pair((threadIdx.x ? n.part_sp2 : n.part_sp) + ti, se.h, se.l);
            } else {
                FF a[1];
                a[0].h = e;
                const FF se = block_pair_sums<1>(a, reinterpret_cast<float*>(sh));
                if (threadIdx.x == 0) store_pair(n.part_sp + ti, se.h, se.l);
            }
        } else {
            const double se = block_sum(e, sh);
            if (threadIdx.x == 0) n.part_sp[ti] = se;
        }
    }
}

// Recovery move: step = maxDist / max_i |d_i|, x += step d (MController.h:273-339).
template <typename Real>
__global__ void __launch_bounds__(kBlock) k_recover_maxabs(DevNet<Real> n) {
    MECH_TRACE_KERNEL(n, TK_RECOVER_MAXABS);
    __shared__ double sh[32];
    __shared__ int s_go, s_flag;
    __shared__ Direction<Real> s_dir;
    const Tile t = n.ftile[blockIdx.x];
    const int r = t.replica;
    if (threadIdx.x == 0) {
        const LaneState<Real> s = lane_state(n, r, PH_RECOVER);
        s_go = s.go;
        s_dir = direction_of(n, s);
    }
    __syncthreads();
    if (!s_go) return;
    const int b = t.begin + threadIdx.x;
    Real m = 0;
    if (b < t.end) {
        Real D[3];
        direction_at(s_dir, b, D);
        m = fmax(fmax(fabs(D[0]), fabs(D[1])), fabs(D[2]));
    }
    const double sm = block_max_r(m, sh);
    if (threadIdx.x == 0) n.part_fil[4 * (size_t)blockIdx.x + 3] = sm;
    const RepTiles rt = n.rt[r];
    if (last_tile(n.ticket, r, rt.fil_end - rt.fil_begin, &s_flag)) {
        const double mx = max_slots(n.part_fil, 4, 3, rt.fil_begin, rt.fil_end, sh);
        if (threadIdx.x == 0) {
            CGState& S = n.st[r];
            const double step = S.maxDist / mx;
            if (!(step < (1.0 / 0.0))) {   // "step size is infinity" (MController.h:311-316)
                S.status = MECH_ERR_NONFINITE;
                S.phase = PH_ERROR;
            } else {
                S.lambda = step;
                S.phase = PH_RECOVER_MOVE;
            }
        }
    }
}

template <typename Real>
__global__ void __launch_bounds__(kBlock) k_recover_move(DevNet<Real> n) {
    MECH_TRACE_KERNEL(n, TK_RECOVER_MOVE);
    __shared__ int s_go, s_xb, s_flag;
    __shared__ Real s_step;
    __shared__ Direction<Real> s_dir;
    const Tile t = n.ftile[blockIdx.x];
    const int r = t.replica;
    if (threadIdx.x == 0) {
        const CGState& S = n.st[r];
        s_go = S.phase == PH_RECOVER_MOVE;
        s_xb = S.xbuf;
        s_step = (Real)S.lambda;
        s_dir = direction_of(n, lane_state(n, r, PH_RECOVER_MOVE));
    }
    __syncthreads();
    if (!s_go) return;
    const int b = t.begin + threadIdx.x;
    if (b < t.end) {   // coord += step * d (MController.h:321-323)
        Real* X = n.x[s_xb];
        store_pos(X, b, bead_at(X, s_dir, b, true, s_step));
    }
    const RepTiles rt = n.rt[r];
    if (last_tile(n.ticket, r, rt.fil_end - rt.fil_begin, &s_flag)) {
        if (threadIdx.x == 0) n.st[r].phase = PH_RECOVER_FORCE;
    }
}

template <typename Real>
__global__ void __launch_bounds__(kBlock) k_backup_restore(DevNet<Real> n) {
    MECH_TRACE_KERNEL(n, TK_BACKUP);
    const Tile t = n.ftile[blockIdx.x];
    const CGState& S = n.st[t.replica];
    if (!S.restore || S.backupPending) return;   // pending: the current positions are the backup
    const int b = t.begin + threadIdx.x;
    if (b < t.end) store_pos(n.x[S.xbuf], b, load_pos(n.xbest, b));
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
template <typename Real>
static int n_lm_tiles(const DevNet<Real>& n, int* ev_tiles, int* bb_tiles) {
    *ev_tiles = n.sp_tiles[K_EXVOL];
    *bb_tiles = n.sp_tiles[K_BOUNDARY];
    return n.sp_tiles[K_LINKER] + n.sp_tiles[K_MOTOR];
}

template <typename Real>
static void launch_gather(const DevNet<Real>& n, int want, cudaStream_t s, bool pdl) {
    const int grid = (n.n_ftiles + n.gtiles - 1) / n.gtiles;
    if constexpr (sizeof(Real) == 4) launch_k(pdl, nullptr, k_force_gather_mx, grid, 64 * n.gtiles, s, n, want);
    else if (n.gtiles == 1) launch_k(pdl, nullptr, k_force_gather<1>, grid, kBlock, s, n, want);
    else launch_k(pdl, nullptr, k_force_gather<kGatherTiles>, grid, kBlock, s, n, want);
}

// The three lanes of an evaluation: the excluded-volume chain and the
// linker/motor/boundary kernel on side lanes, the filament kernel (`fil`) on the
// main lane, which then waits for the others.
// The filament kernel of an evaluation is launched before the side lanes when
// its residency is capped (n.fil_first[k]): its blocks then start streaming at
// once and the excluded-volume and linker kernels fill the room the cap leaves;
// uncapped, it fills every SM and is launched after them.
// With n.pdl the lanes fork and join by programmatic events, so that a kernel's
// blocks are on the SMs when the ones it waits for end.  Per iteration, with
// plain events / programmatic: 60k cylinders 56.2 / 54.4 us, 4k 57.9 / 56.5,
// 32 replicas 95.5 / 93.7, 1M 127.0 / 127.2; FP64 4k 61.0 / 59.5, 1M 684 / 682.
// All three lanes have to start together: where the filament kernel comes first
// it takes the SMs and the excluded-volume chain, which is the longer lane, ends
// later (60k: 62 us).  So the side lanes' kernels, which follow the fork's event
// alone, are not serialized with the previous ones of their streams, and an
// evaluation that does not fork from a reduction (L.forked) has a plain edge to
// its filament kernel, as to the others.
template <typename Real, typename Fil>
static int launch_lanes(const DevNet<Real>& n, int want, int trial, bool force, const Lanes& L, Fil&& fil) {
    int ev_t = 0, bb_t = 0;
    const int lm = n_lm_tiles(n, &ev_t, &bb_t);
    if (!L.forked) cudaEventRecord(L.fork, L.main);
    cudaStreamWaitEvent(L.side, L.fork, 0);
    cudaStreamWaitEvent(L.side2, L.fork, 0);
    if (n.fil_first[force]) fil();
    int launched = 1;
    launched += force ? launch_exvol_forces<Real>(n, want, L.side, false, &L)
                      : launch_exvol_energy<Real>(n, want, trial, L.side, false, &L);
    if (lm + bb_t > 0) {
        launch_k(false, n.pdl ? L.join2 : nullptr, k_bond_bnd<Real>, lm + bb_t, kBlock, L.side2, n, want, trial,
                 force ? 1 : 0, lm, ev_t);
        ++launched;
    }
    if (!n.pdl || lm + bb_t == 0) cudaEventRecord(L.join2, L.side2);
    if (!n.fil_first[force]) fil();
    cudaStreamWaitEvent(L.main, L.join, 0);
    cudaStreamWaitEvent(L.main, L.join2, 0);
    return launched;
}

// An evaluation's reduction follows its lanes on the main lane; with n.pdl it
// records the event that a following evaluation forks from (Lanes::forked).
template <typename Real>
int launch_energy(const DevNet<Real>& n, int want, int trial, const Lanes& L) {
    const int k = launch_lanes(n, want, trial, false, L, [&] {
        if constexpr (sizeof(Real) == 4)
            launch_k(L.forked, nullptr, k_fil_energy_bulk, n.pgrid[0], kBlock, L.main, n, want, trial);
        else launch_k(L.forked, nullptr, k_fil_energy, n.n_ftiles, kBlock, L.main, n, want, trial);
    });
    launch_k(n.pdl, n.pdl ? L.fork : nullptr, k_finalize_energy<Real>, n.R, kBlock, L.main, n, want, trial);
    return k + 1;
}

template <typename Real>
int launch_forces(const DevNet<Real>& n, int want, const Lanes& L) {
    const int k = launch_lanes(n, want, 0, true, L, [&] {
        if constexpr (sizeof(Real) == 4)
            launch_k(L.forked, nullptr, k_fil_force_bulk, n.pgrid[1], kBlock, L.main, n, want);
        else launch_k(L.forked, nullptr, k_fil_force, n.n_force_tiles, kBlock, L.main, n, want);
    });
    launch_gather(n, want, L.main, n.pdl);
    launch_k(n.pdl, n.pdl ? L.fork : nullptr, k_finalize_force<Real>, n.R, kBlock, L.main, n, want);
    return k + 2;
}

int launch_graph_head(cudaStream_t s) {
    k_graph_head<<<1, 32, 0, s>>>();
    return 1;
}

template <typename Real>
int launch_body_head(const DevNet<Real>& n, cudaStream_t s) {
    k_body_head<Real><<<1, kBlock, 0, s>>>(n);
    return 1;
}


template <typename Real>
int launch_recover(const DevNet<Real>& n, const Lanes& L) {
    int k = 0;
    k_recover_maxabs<Real><<<n.n_ftiles, kBlock, 0, L.main>>>(n);
    k_recover_move<Real><<<n.n_ftiles, kBlock, 0, L.main>>>(n);
    k += 2;
    k += launch_forces<Real>(n, PH_RECOVER_FORCE, L);
    k += launch_energy<Real>(n, PH_RECOVER_ENERGY, 0, L);
    return k;
}

template <typename Real>
int launch_backup_restore(const DevNet<Real>& n, cudaStream_t s) {
    k_backup_restore<Real><<<n.n_ftiles, kBlock, 0, s>>>(n);
    return 1;
}

template <typename Real>
int launch_part(const DevNet<Real>& n, int which, cudaStream_t s) {
    int ev_t = 0, bb_t = 0;
    const int lm = n_lm_tiles(n, &ev_t, &bb_t);
    switch (which) {
        case 0:
            if constexpr (sizeof(Real) == 4) k_fil_energy_bulk<<<n.pgrid[0], kBlock, 0, s>>>(n, -1, 0);
            else k_fil_energy<<<n.n_ftiles, kBlock, 0, s>>>(n, -1, 0);
            return 1;
        case 1:
            if constexpr (sizeof(Real) == 4) k_fil_force_bulk<<<n.pgrid[1], kBlock, 0, s>>>(n, -1);
            else k_fil_force<<<n.n_force_tiles, kBlock, 0, s>>>(n, -1);
            launch_gather(n, -1, s, false);
            k_finalize_force<Real><<<n.R, kBlock, 0, s>>>(n, -1);
            return 3;
        case 2: if (lm + bb_t > 0) { k_bond_bnd<Real><<<lm + bb_t, kBlock, 0, s>>>(n, -1, 0, 0, lm, ev_t); return 1; } return 0;
        case 3: if (lm + bb_t > 0) { k_bond_bnd<Real><<<lm + bb_t, kBlock, 0, s>>>(n, -1, 0, 1, lm, ev_t); return 1; } return 0;
        case 4:   // filament energy of a line-search pass (positions x + lambda d formed and written;
                  // mixed: the two-trial pass, lambda and lambda / 2)
            if constexpr (sizeof(Real) == 4) k_fil_energy_bulk<<<n.pgrid[0], kBlock, 0, s>>>(n, -1, kTrialBoth);
            else k_fil_energy<<<n.n_ftiles, kBlock, 0, s>>>(n, -1, 1);
            return 1;
        case 5:   // filament forces alone
            if constexpr (sizeof(Real) == 4) k_fil_force_bulk<<<n.pgrid[1], kBlock, 0, s>>>(n, -1);
            else k_fil_force<<<n.n_force_tiles, kBlock, 0, s>>>(n, -1);
            return 1;
        case 6:   // the sparse gather with the CG partials alone
            launch_gather(n, -1, s, false);
            return 1;
    }
    return 0;
}

// Grid of the mixed engine's persistent filament kernels: every SM holding as
// many blocks as fit, or at most `per_sm` of them (leaving room on each SM for
// the kernels of the other lanes).
int persistent_blocks(int device, int which, int per_sm) {
    static int cached_dev = -1, sms = 0, occ[2] = {0, 0};
    if (cached_dev != device) {
        int b[2] = {0, 0};
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b[0], k_fil_energy_bulk, kBlock, 0);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b[1], k_fil_force_bulk, kBlock, 0);
        for (int k = 0; k < 2; ++k) occ[k] = std::max(1, b[k]);
        sms = std::max(1, sms);
        cached_dev = device;
    }
    const int per = per_sm > 0 ? std::min(per_sm, occ[which]) : occ[which];
    return sms * per;
}

#define MECH_INSTANTIATE(R)                                                             \
    template int launch_part<R>(const DevNet<R>&, int, cudaStream_t);                   \
    template int launch_energy<R>(const DevNet<R>&, int, int, const Lanes&);            \
    template int launch_forces<R>(const DevNet<R>&, int, const Lanes&);                 \
    template int launch_body_head<R>(const DevNet<R>&, cudaStream_t);                   \
    template int launch_recover<R>(const DevNet<R>&, const Lanes&);                     \
    template int launch_backup_restore<R>(const DevNet<R>&, cudaStream_t);
MECH_INSTANTIATE(double)
MECH_INSTANTIATE(float)
#undef MECH_INSTANTIATE

}  // namespace mech
