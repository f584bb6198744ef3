// Hessian-vector products of the full energy (one product: dual numbers; a
// solve: the Hessian's blocks, set up once) and the solves built on them
// (FP64 engine): the conjugate-gradient solve of (H + shift I) y = b used by
// the implicit adjoint and by Newton refinement of an equilibrium, and the
// per-linker parameter gradient of the adjoint.
//
// H v is the forward-mode derivative of the force routines along v: every
// force field is evaluated once on dual numbers (value, derivative) at x + eps v,
// and -dF/deps is written where the force kernels write F, so the sparse force
// fields scatter to the same bead-ordered contribution slots and each bead
// gathers its own (no float atomics; the order is fixed).  The excluded-volume
// pair uses the cancellation-free invariants and atan2 forms (identical
// functions to the reference's, better conditioned).  The reference's force
// routine moves nearly coplanar pairs off their plane before evaluating them
// (CylinderExclVolRepulsion.cpp:610-626, paths relative to medyan-5.4.0/src),
// so its forces are not exactly the energy's gradient there: the solves use
// the exact (symmetric) Hessian of the energy, and the force Jacobian with the
// move differentiated is available separately.  Positions are read from x[0]:
// callers bring every replica's current coordinates there first.
#include <cuda_runtime.h>

#include "mech_device.cuh"
#include "mech_dual.cuh"
#include "mech_exvol_math.cuh"

namespace mech {

namespace {

constexpr int kHvpBlock = 256;

__device__ __forceinline__ void dual_bead(const double* X, const double* V, int b, Dual p[3]) {
#pragma unroll
    for (int k = 0; k < 3; ++k) p[k] = Dual(X[3 * (size_t)b + k], V[3 * (size_t)b + k]);
}

// write -dF/deps (= the H v part) of one bead's contribution
__device__ __forceinline__ void put_hv(const DevNet<double>& n, int slot, const Dual F[3]) {
    double* c = slot_ptr(n, slot);
    c[0] = -F[0].d;
    c[1] = -F[1].d;
    c[2] = -F[2].d;
}

// Excluded-volume pair forces on dual positions; `jac` applies the
// reference's coplanarity move as its force routine does (the force Jacobian,
// not symmetric), otherwise the energy's own gradient (the exact Hessian).
__device__ bool pair_forces_dual(const Dual* c1, const Dual* c2in, const Dual* c3, const Dual* c4, double kRep,
                                 bool jac, Dual out[4][3]) {
    double w1[3], w2[3], w3[3], w4[3];
    for (int k = 0; k < 3; ++k) {
        w1[k] = c1[k].v;
        w2[k] = c2in[k].v;
        w3[k] = c3[k].v;
        w4[k] = c4[k].v;
    }
    Dual c2[3] = {c2in[0], c2in[1], c2in[2]};
    if (jac && coplanarity<double>(w1, w2, w3, w4) < 0.1) {
        Dual a[3], b[3];
        for (int k = 0; k < 3; ++k) {
            a[k] = c2in[k] - c1[k];
            b[k] = c3[k] - c1[k];
        }
        const Dual nx = a[1] * b[2] - a[2] * b[1], ny = a[2] * b[0] - a[0] * b[2], nz = a[0] * b[1] - a[1] * b[0];
        const Dual nn = sqrt(nx * nx + ny * ny + nz * nz);
        c2[0] = c2in[0] + (nx / nn) * 0.01;
        c2[1] = c2in[1] + (ny / nn) * 0.01;
        c2[2] = c2in[2] + (nz / nn) * 0.01;
    }
    Dual v12[3], v34[3], v31[3], v14[3], v32[3], v24[3];
    for (int k = 0; k < 3; ++k) {
        v12[k] = c2[k] - c1[k];
        v34[k] = c4[k] - c3[k];
        v31[k] = c1[k] - c3[k];
        v14[k] = c4[k] - c1[k];
        v32[k] = c2[k] - c3[k];
        v24[k] = c4[k] - c2[k];
    }
    PairInv<Dual> p;
    pair_inv(v12, v34, v31, v14, v32, v24, p, true);
    return forces_from<true>(p, v12, v34, v31, Dual(kRep), out);
}

// A warp of pairs takes ~1,500 FP64 instructions, ~50 us of its sub-partition's
// pipe: blocks of two warps spread them over the SMs (60,000 cylinders, 45 warps
// of pairs: 119 us with eight warps a block, 77 with two).
constexpr int kHvpSparseBlock = 64;
__global__ void __launch_bounds__(kHvpSparseBlock) k_hvp_sparse(DevNet<double> n, const double* __restrict__ V, int jac) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const double* X = n.x[0];
    const int nlm = n.n_lk + n.n_mt;
    if (i < nlm) {
        const bool lk = i < n.n_lk;
        const int j = lk ? i : i - n.n_lk;
        const int4 bs = lk ? n.lk_bead[j] : n.mt_bead[j];
        const double k = lk ? n.lk_k[j] : n.mt_k[j], l0 = lk ? n.lk_l0[j] : n.mt_l0[j];
        const double s1 = lk ? n.lk_s1[j] : n.mt_s1[j], s2 = lk ? n.lk_s2[j] : n.mt_s2[j];
        Dual c1[3], c2[3], c3[3], c4[3];
        dual_bead(X, V, bs.x, c1);
        dual_bead(X, V, bs.y, c2);
        dual_bead(X, V, bs.z, c3);
        dual_bead(X, V, bs.w, c4);
        Dual l[3];
        for (int q = 0; q < 3; ++q) l[q] = (c3[q] + (c4[q] - c3[q]) * s2) - (c1[q] + (c2[q] - c1[q]) * s1);
        const Dual dist = sqrt(l[0] * l[0] + l[1] * l[1] + l[2] * l[2]);
        const Dual f0 = k * (dist - l0) / dist;
        Dual Fa[3], Fb[3], Fc[3], Fd[3];
        for (int q = 0; q < 3; ++q) {
            const Dual Fl = -f0 * l[q];
            Fa[q] = -Fl * (1.0 - s1);
            Fb[q] = -Fl * s1;
            Fc[q] = Fl * (1.0 - s2);
            Fd[q] = Fl * s2;
        }
        const int sb = n.slot_base[lk ? K_LINKER : K_MOTOR] + 4 * j;
        put_hv(n, sb, Fa);
        put_hv(n, sb + 1, Fb);
        put_hv(n, sb + 2, Fc);
        put_hv(n, sb + 3, Fd);
        return;
    }
    const int e = i - nlm;
    if (e < n.n_ev) {
        const int4 bs = n.ev_bead[e];
        Dual c1[3], c2[3], c3[3], c4[3];
        dual_bead(X, V, bs.x, c1);
        dual_bead(X, V, bs.y, c2);
        dual_bead(X, V, bs.z, c3);
        dual_bead(X, V, bs.w, c4);
        Dual out[4][3];
        if (!pair_forces_dual(c1, c2, c3, c4, n.ev_k[e] * n.ev_la[e] * n.ev_lb[e], jac != 0, out)) atomicOr(n.err, 8u);
        for (int a = 0; a < 4; ++a) put_hv(n, n.slot_base[K_EXVOL] + 4 * e + a, out[a]);
        return;
    }
    const int m = e - n.n_ev;
    if (m < n.n_bb) {
        const int b = n.bb_bead[m];
        const double* pl = n.planes + 4 * n.bb_plane[m];
        Dual p[3];
        dual_bead(X, V, b, p);
        const double nrm = sqrt(pl[0] * pl[0] + pl[1] * pl[1] + pl[2] * pl[2]);
        const Dual r = (p[0] * pl[0] + p[1] * pl[1] + p[2] * pl[2] + pl[3]) / nrm;
        const double K = n.bb_k[m], sl = n.bb_slen[m];
        const Dual f0 = K * exp(-r / sl) / sl;
        const Dual F[3] = {f0 * pl[0], f0 * pl[1], f0 * pl[2]};
        put_hv(n, n.slot_base[K_BOUNDARY] + m, F);
    }
}

// Owner side: the filament terms touching each bead on duals, plus the bead's
// gathered sparse contributions; hv = -dF + shift v.  Bound by the FP64 pipe, so
// every cylinder's and triple's terms are formed once and read by the beads they
// act on, and a block takes the beads whose cylinders, three more, fill its warps
// (60,000 cylinders: 41 us; 85 with each bead forming its two and three).
constexpr int kHvpFilBeads = kHvpBlock - 3;
__global__ void __launch_bounds__(kHvpBlock) k_hvp_fil(DevNet<double> n, const double* __restrict__ V, double shift,
                                                      double* __restrict__ HV) {
    __shared__ double s_p[6][kHvpBlock + 1];                       // beads first - 2 .. : value and direction
    __shared__ double s_r[6][kHvpBlock];                           // cylinders first - 2 .. : vector
    __shared__ double s_S[3][kHvpBlock];                           // d(force) of their stretching on the second bead
    __shared__ double s_1[3][kHvpBlock], s_2[3][kHvpBlock];        // d of the triples' terms, on first - 1 ..
    const int first = blockIdx.x * kHvpFilBeads, T = min(kHvpFilBeads, n.nb - first);
    const double* X = n.x[0];
    for (int i = threadIdx.x; i < T + 4; i += blockDim.x) {
        const int b = first - 2 + i;
        if (b < 0 || b >= n.nb) continue;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            s_p[q][i] = X[3 * (size_t)b + q];
            s_p[3 + q][i] = V[3 * (size_t)b + q];
        }
    }
    __syncthreads();
    const int i = threadIdx.x;
    Dual r2[3];
    double ks = 0, l0 = 0, kb = 0, th = 0;
    {
        const int c = first - 2 + i;
        double S[3] = {0, 0, 0};
        if (i < T + 3 && c >= 0 && c < n.nb && (n.bflag[c] & 1)) {
            load_par(n.bpar, c, ks, l0, kb, th);
            Dual F[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                r2[q] = Dual(s_p[q][i + 1], s_p[3 + q][i + 1]) - Dual(s_p[q][i], s_p[3 + q][i]);
                s_r[q][i] = r2[q].v;
                s_r[3 + q][i] = r2[q].d;
            }
            stretch_force<Dual>(r2[0], r2[1], r2[2], Dual(ks), Dual(l0), F);
#pragma unroll
            for (int q = 0; q < 3; ++q) S[q] = F[q].d;
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) s_S[q][i] = S[q];
    }
    __syncthreads();
    {   // thread i: the triple on bead first - 2 + i, at whose second cylinder it is already
        const int c = first - 2 + i;
        double A[3] = {0, 0, 0}, B[3] = {0, 0, 0};
        if (i >= 1 && i < T + 3 && c >= 0 && c < n.nb && (n.bflag[c] & 3) == 3) {
            Dual r1[3], a1[3], a2[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) r1[q] = Dual(s_r[q][i - 1], s_r[3 + q][i - 1]);
            bend_force<Dual>(r1, r2, Dual(kb), Dual(th), a1, a2);
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                A[q] = a1[q].d;
                B[q] = a2[q].d;
            }
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            s_1[q][i] = A[q];
            s_2[q][i] = B[q];
        }
    }
    __syncthreads();
    if (i >= T) return;
    const int b = first + i;   // bead b's own cylinder and triple are at i + 2
    double h[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        double F = s_S[q][i + 1];
        F -= s_S[q][i + 2];
        F += s_2[q][i + 1];
        F += s_1[q][i + 2] - s_2[q][i + 2];
        F -= s_1[q][i + 3];
        h[q] = -F;
    }
    const int c0 = n.csr_off[b], c1 = n.csr_off[b + 1];
    for (int c = c0; c < c1; ++c) {
        h[0] += n.contrib[3 * (size_t)c];
        h[1] += n.contrib[3 * (size_t)c + 1];
        h[2] += n.contrib[3 * (size_t)c + 2];
    }
    for (int q = 0; q < 3; ++q) HV[3 * (size_t)b + q] = h[q] + shift * V[3 * (size_t)b + q];
}

// ---- The Hessian of a solve, held as blocks ------------------------------------
// A solve applies one H to many vectors, and an application by duals costs
// 77 + 41 us on 60,000 cylinders (FP64 pipe: ~1,500 instructions per excluded-
// volume pair and ~250 per bead, most of them the same for every vector).  So a
// solve first evaluates the duals along the unit vectors of each interaction's
// difference vectors and keeps the derivatives:
//   filaments  with u_c = v_{c+1} - v_c of the cylinder (c, c+1), the derivative of
//              the force between the beads is G_c = D_c u_c + M_c u_{c-1} + P_c u_{c+1}
//              (3x3 each: stretching, and the bending triples on c and c+1), and
//              (H v)_c = G_{c-1} - G_c; arrays of [nb] per entry, D, M, P and the
//              part of D that the triple on c+1 adds
//   linkers    H dl = f0 dl + beta (l . dl) l along the linker's vector l: 5 values
//   exvol      the 9x9 matrix over (v12, v34, v31), 81 arrays of [pairs]
//   boundary   (H v) = c (n . v) n: one value
// An application is then ~45 FP64 instructions per bead and ~60 per 8 pairs, and
// reads the blocks once, coalesced (the 216 bytes per cylinder bound it from
// about 100,000 cylinders on, when they leave L2).  Setting them up costs about
// two applications by duals.  They take 288 bytes per bead and 648 per pair; where
// that cannot be had a solve applies the duals in every iteration.
__device__ __forceinline__ Dual unit(double v, bool on) { return Dual(v, on ? 1.0 : 0.0); }

__global__ void __launch_bounds__(kHvpBlock) k_hess_fil(DevNet<double> n, double* __restrict__ A) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n.nb) return;
    const size_t N = n.nb;
    double *D = A + c, *M = A + 9 * N + c, *P = A + 18 * N + c, *T = A + 27 * N + c;
    const int fl = n.bflag[c];
    if (!(fl & 1)) {   // no cylinder starts here
        for (int k = 0; k < 9; ++k) D[k * N] = M[k * N] = P[k * N] = T[k * N] = 0.0;
        return;
    }
    const double* X = n.x[0] + 3 * (size_t)c;
    double ks, l0, kb, th;
    load_par(n.bpar, c, ks, l0, kb, th);
    const double r2[3] = {X[3] - X[0], X[4] - X[1], X[5] - X[2]};
    double d[9];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        Dual F[3];
        stretch_force<Dual>(unit(r2[0], j == 0), unit(r2[1], j == 1), unit(r2[2], j == 2), Dual(ks), Dual(l0), F);
#pragma unroll
        for (int q = 0; q < 3; ++q) d[3 * q + j] = -F[q].d;
    }
    if (fl & 2) {   // the triple on c: (c-1, c, c+1)
        const double r1[3] = {X[0] - X[-3], X[1] - X[-2], X[2] - X[-1]};
#pragma unroll 1
        for (int j = 0; j < 3; ++j) {
            const Dual a[3] = {unit(r1[0], j == 0), unit(r1[1], j == 1), unit(r1[2], j == 2)};
            const Dual b[3] = {Dual(r2[0]), Dual(r2[1]), Dual(r2[2])};
            Dual F1[3], F2[3];
            bend_force<Dual>(a, b, Dual(kb), Dual(th), F1, F2);
            for (int q = 0; q < 3; ++q) {
                T[(3 * q + j) * N - 1] = -F1[q].d;   // on u_{c-1}, of the force across cylinder c-1
                M[(3 * q + j) * N] = -F2[q].d;
            }
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const Dual a[3] = {Dual(r1[0]), Dual(r1[1]), Dual(r1[2])};
            const Dual b[3] = {unit(r2[0], j == 0), unit(r2[1], j == 1), unit(r2[2], j == 2)};
            Dual F1[3], F2[3];
            bend_force<Dual>(a, b, Dual(kb), Dual(th), F1, F2);
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                P[(3 * q + j) * N - 1] = -F1[q].d;
                d[3 * q + j] -= F2[q].d;
            }
        }
    } else {
        for (int k = 0; k < 9; ++k) M[k * N] = 0.0;
    }
    for (int k = 0; k < 9; ++k) D[k * N] = d[k];
    if (!(n.bflag[c + 1] & 1)) {   // the filament's last cylinder: no triple on c+1
        for (int k = 0; k < 9; ++k) P[k * N] = T[k * N] = 0.0;
    }
}
__global__ void __launch_bounds__(kHvpBlock) k_hess_fil_sum(long long n9, double* __restrict__ D,
                                                           const double* __restrict__ T) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i < n9) D[i] += T[i];
}

__global__ void __launch_bounds__(kHvpBlock) k_hess_bonds(DevNet<double> n, double* __restrict__ lm,
                                                         double* __restrict__ bb) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const double* X = n.x[0];
    const int nlm = n.n_lk + n.n_mt;
    if (i < nlm) {
        const bool lk = i < n.n_lk;
        const int j = lk ? i : i - n.n_lk;
        const int4 bs = lk ? n.lk_bead[j] : n.mt_bead[j];
        const double k = lk ? n.lk_k[j] : n.mt_k[j], l0 = lk ? n.lk_l0[j] : n.mt_l0[j];
        const double s1 = lk ? n.lk_s1[j] : n.mt_s1[j], s2 = lk ? n.lk_s2[j] : n.mt_s2[j];
        double l[3];
        for (int q = 0; q < 3; ++q) {
            const double c1 = X[3 * (size_t)bs.x + q], c2 = X[3 * (size_t)bs.y + q], c3 = X[3 * (size_t)bs.z + q],
                         c4 = X[3 * (size_t)bs.w + q];
            l[q] = (c3 + (c4 - c3) * s2) - (c1 + (c2 - c1) * s1);
        }
        const double d = sqrt(l[0] * l[0] + l[1] * l[1] + l[2] * l[2]);
        const size_t N = nlm;
        lm[i] = k * (d - l0) / d;             // f0
        lm[N + i] = k * l0 / (d * d * d);     // beta
        for (int q = 0; q < 3; ++q) lm[(2 + q) * N + i] = l[q];
        return;
    }
    const int m = i - nlm;
    if (m < n.n_bb) {
        const double* pl = n.planes + 4 * n.bb_plane[m];
        const double* x = X + 3 * (size_t)n.bb_bead[m];
        const double nrm = sqrt(pl[0] * pl[0] + pl[1] * pl[1] + pl[2] * pl[2]);
        const double r = (x[0] * pl[0] + x[1] * pl[1] + x[2] * pl[2] + pl[3]) / nrm;
        const double sl = n.bb_slen[m];
        bb[m] = n.bb_k[m] * exp(-r / sl) / sl / (sl * nrm);
    }
}

// One thread per pair and column; the columns of a pair are one grid row apart,
// so that a warp's loads and stores stay coalesced over pairs.
__global__ void __launch_bounds__(128) k_hess_exvol(DevNet<double> n, double* __restrict__ H) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y;
    if (e >= n.n_ev) return;
    const double* X = n.x[0];
    const int4 bs = n.ev_bead[e];
    const double* c[4] = {X + 3 * (size_t)bs.x, X + 3 * (size_t)bs.y, X + 3 * (size_t)bs.z, X + 3 * (size_t)bs.w};
    Dual v12[3], v34[3], v31[3], v14[3], v32[3], v24[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const double da = j == q ? 1.0 : 0.0, db = j == 3 + q ? 1.0 : 0.0, dc = j == 6 + q ? 1.0 : 0.0;
        v12[q] = Dual(c[1][q] - c[0][q], da);
        v34[q] = Dual(c[3][q] - c[2][q], db);
        v31[q] = Dual(c[0][q] - c[2][q], dc);
        v14[q] = Dual(c[3][q] - c[0][q], db - dc);
        v32[q] = Dual(c[1][q] - c[2][q], da + dc);
        v24[q] = Dual(c[3][q] - c[1][q], db - dc - da);
    }
    PairInv<Dual> p;
    pair_inv(v12, v34, v31, v14, v32, v24, p, true);
    Dual out[4][3];
    if (!forces_from<true>(p, v12, v34, v31, Dual(n.ev_k[e] * n.ev_la[e] * n.ev_lb[e]), out)) atomicOr(n.err, 8u);
    const size_t N = n.n_ev;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        H[(9 * q + j) * N + e] = -out[1][q].d;
        H[(9 * (3 + q) + j) * N + e] = -out[3][q].d;
        H[(9 * (6 + q) + j) * N + e] = -out[0][q].d - out[1][q].d;
    }
}

// The sparse interactions' part of H v to the contribution slots: blocks
// [0, lm_blocks) linkers and motors, then excluded-volume pairs (four lanes a
// pair: lane k < 3 the gradient along the k-th difference vector, lane a bead
// a's share), then boundary beads.
__global__ void __launch_bounds__(kHvpBlock) k_hess_apply_sparse(DevNet<double> n, const double* __restrict__ V,
                                                                HvpBlocks h, int lm_blocks, int ev_blocks) {
    const int blk = blockIdx.x;
    if (blk < lm_blocks) {
        const int i = blk * blockDim.x + threadIdx.x, nlm = n.n_lk + n.n_mt;
        if (i >= nlm) return;
        const bool lk = i < n.n_lk;
        const int j = lk ? i : i - n.n_lk;
        const int4 bs = lk ? n.lk_bead[j] : n.mt_bead[j];
        const double s1 = lk ? n.lk_s1[j] : n.mt_s1[j], s2 = lk ? n.lk_s2[j] : n.mt_s2[j];
        double dl[3], l[3], dot = 0.0;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const double v1 = V[3 * (size_t)bs.x + q], v2 = V[3 * (size_t)bs.y + q], v3 = V[3 * (size_t)bs.z + q],
                         v4 = V[3 * (size_t)bs.w + q];
            dl[q] = (v3 + (v4 - v3) * s2) - (v1 + (v2 - v1) * s1);
            l[q] = h.lm[(2 + q) * (size_t)nlm + i];
            dot += l[q] * dl[q];
        }
        const double f0 = h.lm[i], bd = h.lm[(size_t)nlm + i] * dot;
        const int sb = n.slot_base[lk ? K_LINKER : K_MOTOR] + 4 * j;
        const double w[4] = {s1 - 1.0, -s1, 1.0 - s2, s2};
        double g[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) g[q] = f0 * dl[q] + bd * l[q];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            double* c = slot_ptr(n, sb + a);
#pragma unroll
            for (int q = 0; q < 3; ++q) c[q] = w[a] * g[q];
        }
        return;
    }
    if (blk < lm_blocks + ev_blocks) {
        const int t = (blk - lm_blocks) * blockDim.x + threadIdx.x;
        const int e = t >> 2, a = t & 3, k = a < 3 ? a : 2;
        const bool valid = e < n.n_ev;
        double g[3] = {0, 0, 0};
        if (valid) {
            const int4 bs = n.ev_bead[e];
            double w[9];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const double v1 = V[3 * (size_t)bs.x + q], v2 = V[3 * (size_t)bs.y + q], v3 = V[3 * (size_t)bs.z + q],
                             v4 = V[3 * (size_t)bs.w + q];
                w[q] = v2 - v1;
                w[3 + q] = v4 - v3;
                w[6 + q] = v1 - v3;
            }
            const size_t N = n.n_ev;
#pragma unroll
            for (int q = 0; q < 3; ++q)
#pragma unroll
                for (int j = 0; j < 9; ++j) g[q] += h.ev[(9 * (3 * k + q) + j) * N + e] * w[j];
        }
        const int base = threadIdx.x & 28;
        double o[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const double g12 = __shfl_sync(0xffffffffu, g[q], base), g34 = __shfl_sync(0xffffffffu, g[q], base + 1),
                         g31 = __shfl_sync(0xffffffffu, g[q], base + 2);
            o[q] = a == 0 ? g31 - g12 : a == 1 ? g12 : a == 2 ? -g34 - g31 : g34;
        }
        if (valid) {
            double* c = slot_ptr(n, n.slot_base[K_EXVOL] + 4 * e + a);
            c[0] = o[0];
            c[1] = o[1];
            c[2] = o[2];
        }
        return;
    }
    const int m = (blk - lm_blocks - ev_blocks) * blockDim.x + threadIdx.x;
    if (m < n.n_bb) {
        const double* pl = n.planes + 4 * n.bb_plane[m];
        const double* v = V + 3 * (size_t)n.bb_bead[m];
        const double f = h.bb[m] * (v[0] * pl[0] + v[1] * pl[1] + v[2] * pl[2]);
        double* c = slot_ptr(n, n.slot_base[K_BOUNDARY] + m);
        c[0] = f * pl[0];
        c[1] = f * pl[1];
        c[2] = f * pl[2];
    }
}

// ---- CG kernels: deterministic dots (per-block slots, the last block sums the
// slots in order and forms the step) and fused updates --------------------------
constexpr int kCgBlocks = 304;

// scal: [0], [1] r.r of the even and odd iterations, [2] alpha, [3] b.b,
// [4] kCgRunning, or why the iterate is frozen, [5] beta
constexpr double kCgRunning = 0.0, kCgCurvature = 1.0, kCgConverged = 2.0;
// Sum over the grid's blocks; `finish` gets it in one thread of the last block.
template <typename F>
__device__ __forceinline__ void grid_dot(double v, double* part, unsigned* ticket, double* sh, F&& finish) {
    v = block_sum(v, sh);
    __shared__ bool last;
    if (threadIdx.x == 0) {
        part[blockIdx.x] = v;
        __threadfence();
        last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double a = 0.0;
    for (int k = threadIdx.x; k < (int)gridDim.x; k += blockDim.x) a += __ldcg(part + k);
    a = block_sum(a, sh);
    if (threadIdx.x == 0) {
        *ticket = 0u;
        finish(a);
    }
}

__global__ void __launch_bounds__(kHvpBlock) k_cg_start(const double* __restrict__ b, double* __restrict__ x,
                                                        double* __restrict__ r, double* __restrict__ p, long long n,
                                                        double* scal, double* part, unsigned* ticket) {
    __shared__ double sh[32];
    double v = 0.0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const double bi = b[i];
        x[i] = 0.0;
        r[i] = bi;
        p[i] = bi;
        v += bi * bi;
    }
    grid_dot(v, part, ticket, sh, [&](double bb) { scal[0] = scal[3] = bb; });
}

// The CG step alpha = r.r / p.Ap from p.Ap.  No positive curvature freezes the
// iterate (alpha = 0): the truncated solution is what the caller gets, as
// non-positive curvature, or, where the residual is within the tolerance already,
// as the solution.  The host looks every kCheck iterations, and by then a residual
// in few of H's eigenvectors can have underflowed to 0, with p.Ap = 0.
__device__ __forceinline__ void cg_alpha(double pAp, double* scal, int odd, double tol2) {
    if (scal[4] == kCgRunning && !(pAp > 0.0)) scal[4] = scal[odd] <= tol2 ? kCgConverged : kCgCurvature;
    scal[2] = scal[4] != kCgRunning ? 0.0 : scal[odd] / pAp;
}

// hv = H v + shift v at the beads (the filaments' blocks and the gathered sparse
// contributions), v . hv, and the CG step.
__global__ void __launch_bounds__(kHvpBlock) k_hess_apply_fil(DevNet<double> n, const double* __restrict__ V,
                                                             const double* __restrict__ A, double shift,
                                                             double* __restrict__ HV, double* scal, int odd,
                                                             double tol2, double* part, unsigned* ticket) {
    __shared__ double sh[32];
    __shared__ double su[kHvpBlock + 3][3];   // u of cylinders first - 2 .. first + kHvpBlock
    __shared__ double sg[kHvpBlock + 1][3];   // G of cylinders first - 1 .. first + kHvpBlock - 1
    const int first = blockIdx.x * kHvpBlock, nb = n.nb;
    const size_t N = nb;
    for (int i = threadIdx.x; i < kHvpBlock + 3; i += kHvpBlock) {
        const int c = first - 2 + i;
        const bool ok = c >= 0 && c + 1 < nb;
#pragma unroll
        for (int q = 0; q < 3; ++q) su[i][q] = ok ? V[3 * (size_t)(c + 1) + q] - V[3 * (size_t)c + q] : 0.0;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kHvpBlock + 1; i += kHvpBlock) {
        const int c = first - 1 + i;
        double g[3] = {0, 0, 0};
        if (c >= 0 && c < nb) {
            const double* a = A + c;
#pragma unroll
            for (int q = 0; q < 3; ++q)
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    g[q] += a[(3 * q + j) * N] * su[i + 1][j];
                    g[q] += a[(9 + 3 * q + j) * N] * su[i][j];
                    g[q] += a[(18 + 3 * q + j) * N] * su[i + 2][j];
                }
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) sg[i][q] = g[q];
    }
    __syncthreads();
    const int b = first + threadIdx.x;
    double v = 0.0;
    if (b < nb) {
        double h[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) h[q] = sg[threadIdx.x][q] - sg[threadIdx.x + 1][q];
        const int c0 = n.csr_off[b], c1 = n.csr_off[b + 1];
        for (int c = c0; c < c1; ++c)
#pragma unroll
            for (int q = 0; q < 3; ++q) h[q] += n.contrib[3 * (size_t)c + q];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const double vq = V[3 * (size_t)b + q];
            h[q] += shift * vq;
            HV[3 * (size_t)b + q] = h[q];
            v += vq * h[q];
        }
    }
    grid_dot(v, part, ticket, sh, [&](double pAp) { cg_alpha(pAp, scal, odd, tol2); });
}

// the CG step of a product formed by duals: v . hv
__global__ void __launch_bounds__(kHvpBlock) k_cg_alpha(const double* __restrict__ v, const double* __restrict__ hv,
                                                        long long n, double* scal, int odd, double tol2, double* part,
                                                        unsigned* ticket) {
    __shared__ double sh[32];
    double a = 0.0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        a += v[i] * hv[i];
    grid_dot(a, part, ticket, sh, [&](double pAp) { cg_alpha(pAp, scal, odd, tol2); });
}

// x += alpha p, r -= alpha Ap; the new r . r and beta
__global__ void __launch_bounds__(kHvpBlock) k_cg_step(double* __restrict__ x, double* __restrict__ r,
                                                       const double* __restrict__ p, const double* __restrict__ Ap,
                                                       long long n, double* scal, int odd, double* part,
                                                       unsigned* ticket) {
    __shared__ double sh[32];
    const double alpha = scal[2];
    double v = 0.0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        x[i] += alpha * p[i];
        const double ri = r[i] - alpha * Ap[i];
        r[i] = ri;
        v += ri * ri;
    }
    grid_dot(v, part, ticket, sh, [&](double rr) {
        scal[5] = scal[odd] > 0.0 ? rr / scal[odd] : 0.0;
        scal[odd ^ 1] = rr;
    });
}

// p = r + beta p
__global__ void __launch_bounds__(kHvpBlock) k_cg_dir(double* __restrict__ p, const double* __restrict__ r, long long n,
                                                      const double* scal) {
    const double beta = scal[5];
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        p[i] = r[i] + beta * p[i];
}

// Linker parameter gradient of the implicit adjoint, per linker j:
// dL/dk = wE (d - l0)^2 / 2 - (d - l0) g,  dL/dl0 = -wE k (d - l0) + k g,
// with g = lambda . grad_x d (the linker's length gradient at its beads).
__global__ void __launch_bounds__(kHvpBlock) k_linker_grad(DevNet<double> n, int lk0, int nlk,
                                                           const double* __restrict__ L, double wE,
                                                           double* __restrict__ dk, double* __restrict__ dl0) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nlk) return;
    const int j = lk0 + t;
    const int4 bs = n.lk_bead[j];
    const double* X = n.x[0];
    const double s1 = n.lk_s1[j], s2 = n.lk_s2[j], k = n.lk_k[j], l0 = n.lk_l0[j];
    double l[3], lam[3];
    for (int q = 0; q < 3; ++q) {
        const double p1 = X[3 * (size_t)bs.x + q] + (X[3 * (size_t)bs.y + q] - X[3 * (size_t)bs.x + q]) * s1;
        const double p2 = X[3 * (size_t)bs.z + q] + (X[3 * (size_t)bs.w + q] - X[3 * (size_t)bs.z + q]) * s2;
        l[q] = p2 - p1;
        lam[q] = ((1.0 - s2) * L[3 * (size_t)bs.z + q] + s2 * L[3 * (size_t)bs.w + q]) -
                 ((1.0 - s1) * L[3 * (size_t)bs.x + q] + s1 * L[3 * (size_t)bs.y + q]);
    }
    const double d = sqrt(l[0] * l[0] + l[1] * l[1] + l[2] * l[2]);
    const double g = (l[0] * lam[0] + l[1] * lam[1] + l[2] * lam[2]) / d;
    const double dd = d - l0;
    dk[t] = wE * 0.5 * dd * dd - dd * g;
    dl0[t] = -wE * k * dd + k * g;
}

}  // namespace

int launch_hvp(const DevNet<double>& n, const double* v, double* hv, double shift, bool jacobian, cudaStream_t s) {
    const int ns = n.n_lk + n.n_mt + n.n_ev + n.n_bb;
    int k = 0;
    if (ns > 0) {
        k_hvp_sparse<<<(ns + kHvpSparseBlock - 1) / kHvpSparseBlock, kHvpSparseBlock, 0, s>>>(n, v, jacobian ? 1 : 0);
        ++k;
    }
    k_hvp_fil<<<(n.nb + kHvpFilBeads - 1) / kHvpFilBeads, kHvpBlock, 0, s>>>(n, v, shift, hv);
    return k + 1;
}

// Blocks of the Hessian at x[0] into h; returns the kernels launched.
static int assemble_hessian(const DevNet<double>& n, const HvpBlocks& h, cudaStream_t s) {
    const int B = kHvpBlock, nbnd = n.n_lk + n.n_mt + n.n_bb;
    int k = 2;
    k_hess_fil<<<(n.nb + B - 1) / B, B, 0, s>>>(n, h.fil);
    const long long n9 = 9LL * n.nb;
    k_hess_fil_sum<<<(unsigned)((n9 + B - 1) / B), B, 0, s>>>(n9, h.fil, h.fil + 27 * (size_t)n.nb);
    if (nbnd > 0) {
        k_hess_bonds<<<(nbnd + B - 1) / B, B, 0, s>>>(n, h.lm, h.bb);
        ++k;
    }
    if (n.n_ev > 0) {
        k_hess_exvol<<<dim3((unsigned)((n.n_ev + 127) / 128), 9), 128, 0, s>>>(n, h.ev);
        ++k;
    }
    return k;
}

cudaError_t hvp_cg_solve(const DevNet<double>& n, const double* b, double* x, const HvpCgWork& w, double rel_tol,
                         int max_iter, double shift, cudaStream_t s, HvpCgResult* res) {
    const long long N = 3LL * n.nb;
    const int G = kCgBlocks, B = kHvpBlock;
    cudaError_t e;
    *res = HvpCgResult{};
    // x = 0, r = b, p = b; rr = bb = b . b; no curvature flag
    if ((e = cudaMemsetAsync(w.scal, 0, sizeof(double) * 8, s)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(w.ticket, 0, sizeof(unsigned), s)) != cudaSuccess) return e;
    k_cg_start<<<G, B, 0, s>>>(b, x, w.r, w.p, N, w.scal, w.part, w.ticket);
    double h[5];
    if ((e = cudaMemcpyAsync(h, w.scal, sizeof(h), cudaMemcpyDeviceToHost, s)) != cudaSuccess) return e;
    if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return e;
    const double bb = h[3];
    if (!(bb > 0.0)) {
        res->converged = 1;
        return cudaSuccess;
    }
    const double tol2 = rel_tol * rel_tol * bb;
    const bool blocks = w.blocks.fil != nullptr;
    if (blocks) res->launches = assemble_hessian(n, w.blocks, s);
    // kCheck iterations per CUDA graph launch; the host reads the residual between launches
    constexpr int kCheck = 16;   // even: a graph starts on an even iteration
    const int lm_blocks = (n.n_lk + n.n_mt + B - 1) / B, ev_blocks = (int)((4LL * n.n_ev + B - 1) / B),
              sp_blocks = lm_blocks + ev_blocks + (n.n_bb + B - 1) / B;
    int per_iter = 0;
    auto iteration = [&](int it) {
        const int odd = it & 1;
        per_iter = 3;
        if (!blocks) {
            per_iter += launch_hvp(n, w.p, w.Ap, shift, false, s);
            k_cg_alpha<<<G, B, 0, s>>>(w.p, w.Ap, N, w.scal, odd, tol2, w.part, w.ticket);
        } else {
            if (sp_blocks > 0) {
                k_hess_apply_sparse<<<sp_blocks, B, 0, s>>>(n, w.p, w.blocks, lm_blocks, ev_blocks);
                ++per_iter;
            }
            k_hess_apply_fil<<<(n.nb + B - 1) / B, B, 0, s>>>(n, w.p, w.blocks.fil, shift, w.Ap, w.scal, odd, tol2, w.part, w.ticket);
        }
        k_cg_step<<<G, B, 0, s>>>(x, w.r, w.p, w.Ap, N, w.scal, odd, w.part, w.ticket);
        k_cg_dir<<<G, B, 0, s>>>(w.p, w.r, N, w.scal);
    };
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    if ((e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal)) != cudaSuccess) return e;
    for (int j = 0; j < kCheck; ++j) iteration(j);
    e = cudaStreamEndCapture(s, &graph);
    if (e == cudaSuccess) e = cudaGraphInstantiate(&exec, graph, 0);
    if (graph) cudaGraphDestroy(graph);
    if (e != cudaSuccess) return e;
    for (int it = 0; it < max_iter;) {
        if (max_iter - it >= kCheck) {
            e = cudaGraphLaunch(exec, s);
            it += kCheck;
            res->launches += (long long)kCheck * per_iter;
        } else {
            for (; it < max_iter; ++it) {
                iteration(it);
                res->launches += per_iter;
            }
            e = cudaGetLastError();
        }
        if (e != cudaSuccess) break;
        if ((e = cudaMemcpyAsync(h, w.scal, sizeof(h), cudaMemcpyDeviceToHost, s)) != cudaSuccess) break;
        if ((e = cudaStreamSynchronize(s)) != cudaSuccess) break;
        const double rr = h[it & 1];
        res->iterations = it;
        res->rel_residual = sqrt(rr / bb);
        if (h[4] == kCgCurvature) {   // non-positive curvature met: the iterate stopped there
            res->negative_curvature = 1;
            break;
        }
        if (rr <= tol2) {
            res->converged = 1;
            break;
        }
    }
    cudaGraphExecDestroy(exec);
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

void launch_linker_grad(const DevNet<double>& n, int lk0, int nlk, const double* lambda, double wE, double* dk,
                        double* dl0, cudaStream_t s) {
    if (nlk <= 0) return;
    k_linker_grad<<<(nlk + kHvpBlock - 1) / kHvpBlock, kHvpBlock, 0, s>>>(n, lk0, nlk, lambda, wE, dk, dl0);
}

}  // namespace mech
