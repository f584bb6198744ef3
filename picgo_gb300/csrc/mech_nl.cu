// Neighbor-list rebuild on the device, the exclusive scan it uses, and the
// bead-to-contribution CSR index of the sparse force fields.
//
// Cylinder-cylinder half list (HybridCylinderCylinderNL, paths relative to
// medyan-5.4.0/src: Structure/HybridNeighborListImpl.cpp:176-471 and
// Structure/BinGrid.h:134-199): midpoints binned on a uniform grid whose cell
// edge is at least rMax, a 27-cell stencil, and the reference's predicate --
// keep (c, n) when id_c > id_n, the two are not within two positions of the
// same filament, and rMin^2 <= |m_n - m_c|^2 <= rMax^2 with the square summed
// in double from zero and the bounds rounded to float as the reference stores
// them.  The stencil covers every cell that can hold a neighbor, so the set is
// the same for every cell edge >= rMax; a single-precision distance with a
// conservative margin decides all but the candidates near the cutoff.  Each
// cylinder's neighbors are written in ascending cylinder order.
//
// Boundary-cylinder list (Structure/NeighborListImpl.cpp:738-751): per plane,
// every cylinder whose midpoint lies closer than BoundaryCutoff (signed
// distance), plane by plane in cylinder order; a filament's minus-end cylinder
// contributes its first bead as well as its second
// (Mechanics/ForceField/Boundary/BoundaryCylinderRepulsion.cpp:33-88).
#include <cuda_runtime.h>

#include "mech_device.cuh"
#include "mech_nl.cuh"

namespace mech {

#ifdef MECH_ALLOC_LIMIT
// builds for tests of what follows a failed allocation: larger ones fail
extern "C" size_t mech_alloc_limit = MECH_ALLOC_LIMIT;
#endif

cudaError_t DeviceBuffer::ensure(size_t nbytes) {
    if (nbytes <= bytes && p) return cudaSuccess;
    release();
#ifdef MECH_ALLOC_LIMIT
    if (nbytes > mech_alloc_limit) return cudaErrorMemoryAllocation;
#endif
    size_t want = nbytes < 256 ? 256 : nbytes;
    cudaError_t e = cudaMalloc(&p, want);
    if (e != cudaSuccess) {
        cudaGetLastError();   // returned here, and not found again by the next call's launches
        p = nullptr;
        bytes = 0;
        return e;
    }
    bytes = want;
    return cudaSuccess;
}

void DeviceBuffer::release() {
    if (p) cudaFree(p);
    p = nullptr;
    bytes = 0;
}

// ---------------------------------------------------------------------------
// exclusive scan: tile scans and their sums, the sums scanned (recursively),
// then added back.  HBM-bound: 4 reads and writes of the array; 16 items per
// thread in four 16-byte vectors, so that a tile takes two barriers.
// ---------------------------------------------------------------------------
constexpr int kScanBlock = 256;
constexpr int kScanVecs = 4;                              // int4 vectors per thread
constexpr int kScanTile = 4 * kScanVecs * kScanBlock;

__device__ __forceinline__ int warp_scan_incl(int v) {
    const int l = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, o);
        if (l >= o) v += u;
    }
    return v;
}
// Exclusive prefix of v over a kScanBlock block; *total receives the block sum.
__device__ __forceinline__ int block_scan_excl(int v, int* sh /* [kScanBlock / 32] */, int* total) {
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const int incl = warp_scan_incl(v);
    if (l == 31) sh[w] = incl;
    __syncthreads();
    int pre = 0, tot = 0;
#pragma unroll
    for (int k = 0; k < kScanBlock / 32; ++k) {
        const int t = sh[k];
        if (k < w) pre += t;
        tot += t;
    }
    *total = tot;
    return pre + incl - v;
}

// `end`: where the total goes when one tile holds the whole array (else null)
__global__ void __launch_bounds__(kScanBlock) k_scan_tile(const int* in, int* out, int* sums, int* end, long long n) {
    __shared__ int sh[kScanBlock / 32];
    const long long base = (long long)blockIdx.x * kScanTile + (long long)threadIdx.x * (4 * kScanVecs);
    int v[4 * kScanVecs];
    int run = 0;
    if (base + 4 * kScanVecs <= n) {
#pragma unroll
        for (int k = 0; k < kScanVecs; ++k) {
            const int4 q = reinterpret_cast<const int4*>(in + base)[k];
            v[4 * k] = q.x; v[4 * k + 1] = q.y; v[4 * k + 2] = q.z; v[4 * k + 3] = q.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < 4 * kScanVecs; ++k) v[k] = base + k < n ? in[base + k] : 0;
    }
#pragma unroll
    for (int k = 0; k < 4 * kScanVecs; ++k) run += v[k];
    int total;
    int pre = block_scan_excl(run, sh, &total);
#pragma unroll
    for (int k = 0; k < 4 * kScanVecs; ++k) {
        const int x = v[k];
        v[k] = pre;
        pre += x;
    }
    if (base + 4 * kScanVecs <= n) {
#pragma unroll
        for (int k = 0; k < kScanVecs; ++k)
            reinterpret_cast<int4*>(out + base)[k] = make_int4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
    } else {
#pragma unroll
        for (int k = 0; k < 4 * kScanVecs; ++k)
            if (base + k < n) out[base + k] = v[k];
    }
    if (threadIdx.x == 0) {
        sums[blockIdx.x] = total;
        if (end) *end = total;
    }
}

// offs: the scanned tile sums, [tiles] the total
__global__ void __launch_bounds__(kScanBlock) k_scan_add(int* out, const int* offs, long long n) {
    const long long base = (long long)blockIdx.x * kScanTile;
    const int add = offs[blockIdx.x];
#pragma unroll
    for (int k = 0; k < kScanVecs; ++k) {
        const long long i = base + 4LL * (k * kScanBlock + threadIdx.x);
        if (i + 4 <= n) {
            int4 q = *reinterpret_cast<const int4*>(out + i);
            q.x += add; q.y += add; q.z += add; q.w += add;
            *reinterpret_cast<int4*>(out + i) = q;
        } else {
            for (long long j = i; j < n; ++j) out[j] += add;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) out[n] = offs[gridDim.x];
}

// scratch of a level: its tile sums and their scan, each rounded to 16 bytes
static inline long long scan_level(long long tiles) { return 2 * (((tiles + 1) + 3) & ~3LL); }

static cudaError_t scan_rec(const int* in, int* out, long long n, int* tmp, cudaStream_t s) {
    const long long nb = (n + kScanTile - 1) / kScanTile;
    int* sums = tmp;
    int* sums_scan = tmp + scan_level(nb) / 2;
    k_scan_tile<<<(unsigned)nb, kScanBlock, 0, s>>>(in, out, sums, nb == 1 ? out + n : nullptr, n);
    if (nb > 1) {
        cudaError_t e = scan_rec(sums, sums_scan, nb, tmp + scan_level(nb), s);
        if (e != cudaSuccess) return e;
        k_scan_add<<<(unsigned)nb, kScanBlock, 0, s>>>(out, sums_scan, n);
    }
    return cudaGetLastError();
}

cudaError_t exclusive_scan_i32(const int* in, int* out, long long n, DeviceBuffer& tmp, cudaStream_t s) {
    if (n <= 0) return cudaMemsetAsync(out, 0, sizeof(int), s);
    long long need = 0;
    for (long long m = n;;) {
        m = (m + kScanTile - 1) / kScanTile;
        need += scan_level(m);
        if (m <= 1) break;
    }
    cudaError_t e = tmp.ensure(sizeof(int) * (size_t)need);
    if (e != cudaSuccess) return e;
    return scan_rec(in, out, n, tmp.as<int>(), s);
}

// ---------------------------------------------------------------------------
// cylinder pair list
// ---------------------------------------------------------------------------
// Bin of a single-precision midpoint coordinate.  Any binning by a monotone
// function gives the full stencil as long as two midpoints within rMax fall at
// most one bin apart: `inv` is the reciprocal of an edge that exceeds rMax by
// more than the rounding of the midpoint and of this product (rebuild()).
__device__ __forceinline__ int cell_axis(float m, float inv, int g) {
    const int i = (int)floorf(m * inv);
    return i < 0 ? 0 : (i >= g ? g - 1 : i);
}

// 0.5 * (b1 + b2) (Structure/Cylinder.cpp:45-46); equal to the boundary
// list's b1 * 0.5 + 0.5 * b2 bit for bit.  Formed where a decision needs it:
// a midpoint costs 9 (mixed: 21) instructions of the slow FP64 pipe.
__device__ __forceinline__ void exact_mid(const void* x, int mixed, int b, double m[3]) {
    double x1[3], x2[3];
    if (mixed) {
        to_double(load_pos(static_cast<const float*>(x), b), x1);
        to_double(load_pos(static_cast<const float*>(x), b + 1), x2);
    } else {
        to_double(load_pos(static_cast<const double*>(x), b), x1);
        to_double(load_pos(static_cast<const double*>(x), b + 1), x2);
    }
    for (int k = 0; k < 3; ++k) m[k] = __dmul_rn(0.5, __dadd_rn(x1[k], x2[k]));
}

// Single-precision midpoints (within 2 ulp) and the bin of each cylinder.
__global__ void k_nl_mid(NLInput in, float4* midf, int* cell_of, int* cell_count) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= in.ncyl) return;
    const int b = in.cyl_b1[c];
    float m[3];
    if (in.mixed) {
        const Pos<float> p = load_pos(static_cast<const float*>(in.x), b), q = load_pos(static_cast<const float*>(in.x), b + 1);
#pragma unroll
        for (int k = 0; k < 3; ++k) m[k] = 0.5f * ((p.h[k] + q.h[k]) + (p.l[k] + q.l[k]));
    } else {
        const double* p = static_cast<const double*>(in.x) + 3 * (size_t)b;
#pragma unroll
        for (int k = 0; k < 3; ++k) m[k] = 0.5f * (float)(p[k] + p[k + 3]);
    }
    midf[c] = make_float4(m[0], m[1], m[2], __int_as_float(c));
    const NLReplica& R = in.rep[in.R == 1 ? 0 : in.cyl_rep[c]];
    const int4 g = R.dims;
    const int id = g.w + (cell_axis(m[0], R.inv, g.x) * g.y + cell_axis(m[1], R.inv, g.y)) * g.z + cell_axis(m[2], R.inv, g.z);
    cell_of[c] = id;
    atomicAdd(cell_count + id, 1);
}

// Midpoints (with their cylinder) in bin order; each bin's count runs down to zero.
__global__ void k_nl_scatter(int n, const int* cell_of, const int* cell_start, int* cell_count, const float4* midf,
                             float4* sorted) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const int id = cell_of[c];
    sorted[cell_start[id] + atomicSub(cell_count + id, 1) - 1] = midf[c];
}

// Visit every candidate of the cylinder at `fc`; accept(n) is called for its
// neighbors.  Bins along z are consecutive, so the 27-bin stencil is nine runs
// of bin-ordered midpoints, whose bounds are all loaded before the first run.
template <typename F>
__device__ __forceinline__ void nl_visit(const NLInput& in, const int* cell_start, const float4* sorted, float4 fc,
                                         F&& accept) {
    const int c = __float_as_int(fc.w);
    const NLReplica& R = in.rep[in.R == 1 ? 0 : in.cyl_rep[c]];
    const int4 g = R.dims;
    const int ix = cell_axis(fc.x, R.inv, g.x), iy = cell_axis(fc.y, R.inv, g.y), iz = cell_axis(fc.z, R.inv, g.z);
    const int z0 = max(iz - 1, 0), z1 = min(iz + 1, g.z - 1) + 1;
    const bool far = !(fmaxf(fmaxf(fabsf(fc.x), fabsf(fc.y)), fabsf(fc.z)) <= R.reach);
    const float pre = far ? INFINITY : R.pre, sure = far ? -INFINITY : R.sure;
    int s0[9], s1[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const int jx = ix + k / 3 - 1, jy = iy + k % 3 - 1;
        const bool ok = jx >= 0 && jx < g.x && jy >= 0 && jy < g.y;
        const int row = g.w + (jx * g.y + jy) * g.z;
        s0[k] = ok ? cell_start[row + z0] : 0;
        s1[k] = ok ? cell_start[row + z1] : 0;
    }
    bool have = false;
    long long idc = 0;
    int filc = 0, posc = 0;
#pragma unroll
    for (int k = 0; k < 9; ++k)
        for (int s = s0[k]; s < s1[k]; ++s) {
            const float4 fn = sorted[s];
            const float ex = fn.x - fc.x, ey = fn.y - fc.y, ez = fn.z - fc.z;
            const float f2 = ex * ex + ey * ey + ez * ez;
            if (f2 > pre) continue;
            const int n = __float_as_int(fn.w);
            if (n == c) continue;
            if (!have) {   // the cylinder's own data, for the few that have a candidate
                have = true;
                idc = in.cyl_id[c];
                filc = in.cyl_fil[c];
                posc = in.cyl_pos[c];
            }
            if (idc <= in.cyl_id[n]) continue;
            if (filc == in.cyl_fil[n] && abs(posc - in.cyl_pos[n]) <= 2) continue;
            if (!(f2 < sure)) {   // within the rounding of the cutoff: the reference's test on the exact midpoints
                double mc[3], mn[3], d2 = 0.0;
                exact_mid(in.x, in.mixed, in.cyl_b1[c], mc);
                exact_mid(in.x, in.mixed, in.cyl_b1[n], mn);
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    const double d = mn[q] - mc[q];
                    d2 = __dadd_rn(d2, __dmul_rn(d, d));
                }
                if (d2 < R.rmin2 || d2 > R.rmax2) continue;
            }
            accept(n);
        }
}

// Neighbor counts, and the first kNlKeep neighbors of each cylinder, so that
// the list is written without visiting the candidates again.  Threads take the
// cylinders in bin order: a warp's stencils overlap, and its loads hit L1.
// Latency-bound on the run bounds: 95 us for the count and 17 us for the write
// on 1M cylinders (2M bins), against 348 + 344 us for two visits of 27 separate
// bins in cylinder order with the exact test on stored FP64 midpoints, and 264
// us for this count when every candidate past the prefilter took that test.
constexpr int kNlKeep = 8;
__global__ void __launch_bounds__(128) k_nl_count(NLInput in, const int* cell_start, const float4* sorted, int* cnt,
                                                  int* keep) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= in.ncyl) return;
    const float4 fc = sorted[t];
    const int c = __float_as_int(fc.w);
    int k = 0;
    nl_visit(in, cell_start, sorted, fc, [&](int n) {
        if (k < kNlKeep) keep[kNlKeep * (size_t)c + k] = n;
        ++k;
    });
    cnt[c] = k;
}

// The pairs of each cylinder at its offset, in ascending neighbor order.
__global__ void k_nl_write(NLInput in, const int* cell_start, const float4* sorted, const float4* midf, const int* cnt,
                           const int* keep, const int* off, int2* pairs) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= in.ncyl) return;
    const int k = cnt[c];
    if (k == 0) return;
    int2* out = pairs + off[c];
    if (k <= kNlKeep) {
        for (int i = 0; i < k; ++i) out[i] = make_int2(c, keep[kNlKeep * (size_t)c + i]);
    } else {
        int i = 0;
        nl_visit(in, cell_start, sorted, midf[c], [&](int n) { out[i++] = make_int2(c, n); });
    }
    for (int i = 1; i < k; ++i) {   // insertion sort of this cylinder's short segment
        const int2 v = out[i];
        int j = i - 1;
        while (j >= 0 && out[j].y > v.y) {
            out[j + 1] = out[j];
            --j;
        }
        out[j + 1] = v;
    }
}

cudaError_t count_pairs(const NLInput& in, PairBuild& pb, cudaStream_t s) {
    cudaError_t e;
    const int n = in.ncyl;
    if ((e = pb.cell_count.ensure(sizeof(int) * (size_t)(in.ncells + 1))) != cudaSuccess) return e;
    if ((e = pb.cell_start.ensure(sizeof(int) * (size_t)(in.ncells + 1))) != cudaSuccess) return e;
    if ((e = pb.sorted.ensure(sizeof(float4) * (size_t)n)) != cudaSuccess) return e;
    if ((e = pb.midf.ensure(sizeof(float4) * (size_t)n)) != cudaSuccess) return e;
    if ((e = pb.cell_of.ensure(sizeof(int) * (size_t)n)) != cudaSuccess) return e;
    if ((e = pb.keep.ensure(sizeof(int) * kNlKeep * (size_t)n)) != cudaSuccess) return e;
    if ((e = pb.cnt.ensure(sizeof(int) * (size_t)(n + 1))) != cudaSuccess) return e;
    if ((e = pb.off.ensure(sizeof(int) * (size_t)(n + 1))) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(pb.cell_count.p, 0, sizeof(int) * (size_t)(in.ncells + 1), s)) != cudaSuccess) return e;
    const int tb = 256, nblk = (n + tb - 1) / tb;
    k_nl_mid<<<nblk, tb, 0, s>>>(in, pb.midf.as<float4>(), pb.cell_of.as<int>(), pb.cell_count.as<int>());
    if ((e = exclusive_scan_i32(pb.cell_count.as<int>(), pb.cell_start.as<int>(), in.ncells, pb.scan_tmp, s)) !=
        cudaSuccess)
        return e;
    k_nl_scatter<<<nblk, tb, 0, s>>>(n, pb.cell_of.as<int>(), pb.cell_start.as<int>(), pb.cell_count.as<int>(),
                                     pb.midf.as<float4>(), pb.sorted.as<float4>());
    k_nl_count<<<(n + 127) / 128, 128, 0, s>>>(in, pb.cell_start.as<int>(), pb.sorted.as<float4>(), pb.cnt.as<int>(),
                                               pb.keep.as<int>());
    return exclusive_scan_i32(pb.cnt.as<int>(), pb.off.as<int>(), n, pb.scan_tmp, s);
}

cudaError_t write_pairs(const NLInput& in, PairBuild& pb, long long total, cudaStream_t s) {
    cudaError_t e;
    if ((e = pb.pairs.ensure(sizeof(int2) * (size_t)(total > 0 ? total : 1))) != cudaSuccess) return e;
    if (total > 0)
        k_nl_write<<<(in.ncyl + 255) / 256, 256, 0, s>>>(in, pb.cell_start.as<int>(), pb.sorted.as<float4>(),
                                                        pb.midf.as<float4>(), pb.cnt.as<int>(), pb.keep.as<int>(),
                                                        pb.off.as<int>(), pb.pairs.as<int2>());
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// boundary list
// ---------------------------------------------------------------------------
// entry q of replica r: plane p = q / nc_r, cylinder c = q % nc_r (replica-local)
struct BndEntry {
    int r, plane;          // replica, plane index within it
    unsigned nc, cyl;      // the replica's cylinders, cylinder within it
};
__device__ __forceinline__ BndEntry bnd_entry(const BndInput& in, long long q) {
    int lo = 0, hi = in.R - 1;   // last r with bnd_begin <= q
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (in.rep[mid].bnd_begin <= q) lo = mid;
        else hi = mid - 1;
    }
    BndEntry e;
    e.r = lo;
    e.nc = (unsigned)in.rep[lo].ncyl;
    const long long lq = q - in.rep[lo].bnd_begin;
    if (lq <= 0xffffffffLL) {
        e.plane = (int)((unsigned)lq / e.nc);
        e.cyl = (unsigned)lq - (unsigned)e.plane * e.nc;
    } else {
        e.plane = (int)(lq / e.nc);
        e.cyl = (unsigned)(lq - (long long)e.plane * e.nc);
    }
    return e;
}
// the next entry (planes without cylinders do not exist: a replica has at least one cylinder)
__device__ __forceinline__ void bnd_next(const BndInput& in, long long q, BndEntry& e) {
    if (++e.cyl < e.nc) return;
    e = bnd_entry(in, q);
}

// Is global cylinder c closer to plane `pl` than the cutoff?  Decided in single
// precision unless the distance lies within its rounding of the cutoff (then,
// and for values that compare with nothing, in FP64 as the reference's list
// test rounds it): the FP64 form alone takes ~20 instructions of the FP64 pipe
// and bound this list at 310 us for 6 planes x 1M cylinders; converting a
// plane's coefficients to float for each entry still bound it at 53 us; now 26 us.
__device__ __forceinline__ bool bnd_listed(const BndInput& in, int p, double cutoff, float cutoff_f, int c) {
    const float4 m = in.midf[c], pf = in.planes_f[p];
    const float ax = pf.x * m.x, by = pf.y * m.y, cz = pf.z * m.z;
    const float nrm = sqrtf(pf.x * pf.x + pf.y * pf.y + pf.z * pf.z);
    const float cut = cutoff_f * nrm;
    const float num = ax + by + cz + pf.w - cut;
    // 2 ulp of each midpoint component, 1 of each coefficient and of each operation, bounded by the magnitudes' sum
    const float err = 2e-6f * (fabsf(ax) + fabsf(by) + fabsf(cz) + fabsf(pf.w) + fabsf(cut));
    if (nrm > 1e-15f && nrm < 1e15f) {   // squares of the coefficients neither underflow nor overflow
        if (num > err) return false;
        if (num < -err) return true;
    }
    const double* pl = in.planes + 4 * (size_t)p;
    double x[3];
    exact_mid(in.x, in.mixed, in.cyl_b1[c], x);
    double num2 = __dmul_rn(pl[0], x[0]);
    num2 = __dadd_rn(num2, __dmul_rn(pl[1], x[1]));
    num2 = __dadd_rn(num2, __dmul_rn(pl[2], x[2]));
    num2 = __dadd_rn(num2, pl[3]);
    const double n2 = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(pl[0], pl[0]), __dmul_rn(pl[1], pl[1])), __dmul_rn(pl[2], pl[2])));
    return __ddiv_rn(num2, n2) < cutoff;
}

// Beads listed by each entry (0, 1, or 2 for a minus-end cylinder; one byte),
// the sum of each tile of kBndTile entries, and the number of listed entries.
__global__ void __launch_bounds__(kScanBlock) k_bnd_count(BndInput in, uint8_t* cnt, int* sums, int* ncyl) {
    __shared__ int sh[kScanBlock / 32];
    const long long q0 = (long long)blockIdx.x * kBndTile + 4 * threadIdx.x;
    int beads = 0, listed = 0;
    if (q0 < in.nq) {
        BndEntry e = bnd_entry(in, q0);
        unsigned packed = 0;
        const int m = (int)min(4LL, in.nq - q0);
        for (int k = 0; k < m; ++k) {
            if (k) bnd_next(in, q0 + k, e);
            const NLReplica& R = in.rep[e.r];
            const int c = R.cyl_begin + (int)e.cyl;
            if (bnd_listed(in, R.plane_begin + e.plane, R.bnd_cutoff, R.bnd_cutoff_f, c)) {
                const int nb = in.cyl_minus[c] ? 2 : 1;
                packed |= (unsigned)nb << (8 * k);
                beads += nb;
                ++listed;
            }
        }
        *reinterpret_cast<unsigned*>(cnt + q0) = packed;   // the array is padded to whole tiles
    }
    int total;
    block_scan_excl(beads, sh, &total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
    if (total == 0) return;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) listed += __shfl_down_sync(0xffffffffu, listed, o);
    if ((threadIdx.x & 31) == 0 && listed) atomicAdd(ncyl, listed);
}

// List offset of the first entry of each replica (and the total): the offset
// of its tile and the beads listed before it there.
__global__ void __launch_bounds__(kScanBlock) k_bnd_rep_offset(BndInput in, const uint8_t* cnt, const int* off,
                                                               long long* out) {
    __shared__ int sh[kScanBlock / 32];
    const long long q = (int)blockIdx.x < in.R ? in.rep[blockIdx.x].bnd_begin : in.nq;
    const long long t = q / kBndTile;
    int v = 0;
    for (long long i = t * kBndTile + threadIdx.x; i < q; i += blockDim.x) v += cnt[i];
    int total;
    block_scan_excl(v, sh, &total);
    if (threadIdx.x == 0) out[blockIdx.x] = off[t] + total;
}

__global__ void __launch_bounds__(kScanBlock) k_bnd_write(BndInput in, const uint8_t* cnt, const int* off, int* bb_bead,
                                                          int* bb_plane) {
    __shared__ int sh[kScanBlock / 32];
    if (off[blockIdx.x] == off[blockIdx.x + 1]) return;   // nothing listed in this tile
    const long long q0 = (long long)blockIdx.x * kBndTile + 4 * threadIdx.x;
    const unsigned packed = q0 < in.nq ? *reinterpret_cast<const unsigned*>(cnt + q0) : 0;
    const int beads = (packed & 255) + ((packed >> 8) & 255) + ((packed >> 16) & 255) + (packed >> 24);
    int total;
    int o = off[blockIdx.x] + block_scan_excl(beads, sh, &total);
    for (int k = 0; k < 4; ++k) {
        const int nb = (packed >> (8 * k)) & 255;
        if (!nb) continue;
        const BndEntry e = bnd_entry(in, q0 + k);
        const NLReplica& R = in.rep[e.r];
        const int b1 = in.cyl_b1[R.cyl_begin + (int)e.cyl], p = R.plane_begin + e.plane;
        if (nb == 2) {
            bb_bead[o] = b1;
            bb_plane[o++] = p;
        }
        bb_bead[o] = b1 + 1;
        bb_plane[o++] = p;
    }
}

cudaError_t count_boundary(const BndInput& in, BndBuild& bb, long long* rep_offset, cudaStream_t s) {
    cudaError_t e;
    const long long tiles = (in.nq + kBndTile - 1) / kBndTile;
    if ((e = bb.cnt.ensure((size_t)(tiles + 1) * kBndTile)) != cudaSuccess) return e;
    if ((e = bb.sums.ensure(sizeof(int) * (size_t)(tiles + 1))) != cudaSuccess) return e;
    if ((e = bb.off.ensure(sizeof(int) * (size_t)(tiles + 2))) != cudaSuccess) return e;
    if ((e = bb.ncyl.ensure(sizeof(int))) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(bb.ncyl.p, 0, sizeof(int), s)) != cudaSuccess) return e;
    if (tiles > 0)
        k_bnd_count<<<(unsigned)tiles, kScanBlock, 0, s>>>(in, bb.cnt.as<uint8_t>(), bb.sums.as<int>(), bb.ncyl.as<int>());
    if ((e = exclusive_scan_i32(bb.sums.as<int>(), bb.off.as<int>(), tiles, bb.scan_tmp, s)) != cudaSuccess) return e;
    k_bnd_rep_offset<<<in.R + 1, kScanBlock, 0, s>>>(in, bb.cnt.as<uint8_t>(), bb.off.as<int>(), rep_offset);
    return cudaGetLastError();
}

cudaError_t write_boundary(const BndInput& in, BndBuild& bb, long long total, cudaStream_t s) {
    cudaError_t e;
    if ((e = bb.bead.ensure(sizeof(int) * (size_t)(total > 0 ? total : 1))) != cudaSuccess) return e;
    if ((e = bb.plane.ensure(sizeof(int) * (size_t)(total > 0 ? total : 1))) != cudaSuccess) return e;
    if (total > 0)
        k_bnd_write<<<(unsigned)((in.nq + kBndTile - 1) / kBndTile), kScanBlock, 0, s>>>(
            in, bb.cnt.as<uint8_t>(), bb.off.as<int>(), bb.bead.as<int>(), bb.plane.as<int>());
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// CSR of sparse contribution slots per bead
// ---------------------------------------------------------------------------
__device__ __forceinline__ int slot_bead(const CsrInput& in, int s) {
    if (s < in.base[1]) { const int4 b = in.lk[(s - in.base[0]) >> 2]; const int q = (s - in.base[0]) & 3; return q == 0 ? b.x : q == 1 ? b.y : q == 2 ? b.z : b.w; }
    if (s < in.base[2]) { const int4 b = in.mt[(s - in.base[1]) >> 2]; const int q = (s - in.base[1]) & 3; return q == 0 ? b.x : q == 1 ? b.y : q == 2 ? b.z : b.w; }
    if (s < in.base[3]) { const int4 b = in.ev[(s - in.base[2]) >> 2]; const int q = (s - in.base[2]) & 3; return q == 0 ? b.x : q == 1 ? b.y : q == 2 ? b.z : b.w; }
    return in.bb[s - in.base[3]];
}

__global__ void k_csr_count(CsrInput in, int* cnt) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= in.base[4]) return;
    atomicAdd(cnt + slot_bead(in, s), 1);
}
__global__ void k_csr_fill(CsrInput in, const int* off, int* cursor, int* slots) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= in.base[4]) return;
    const int b = slot_bead(in, s);
    slots[off[b] + atomicAdd(cursor + b, 1)] = s;
}
__global__ void k_csr_sort(int nb, const int* off, int* slots) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    const int o = off[b], k = off[b + 1] - o;
    for (int i = 1; i < k; ++i) {
        const int v = slots[o + i];
        int j = i - 1;
        while (j >= 0 && slots[o + j] > v) {
            slots[o + j + 1] = slots[o + j];
            --j;
        }
        slots[o + j + 1] = v;
    }
}

// Position of every slot in the bead-ordered CSR sequence: the sparse force
// kernels write each contribution there, so a bead's contributions are
// contiguous, in the CSR order, for the filament force kernels to read.
__global__ void k_csr_inverse(int ns, const int* slots, int* pos) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= ns) return;
    pos[slots[c]] = c;
}

cudaError_t build_csr(const CsrInput& in, CsrBuild& cb, cudaStream_t s) {
    cudaError_t e;
    const int ns = in.base[4];
    if ((e = cb.cnt.ensure(sizeof(int) * (size_t)(in.nb + 1))) != cudaSuccess) return e;
    if ((e = cb.cursor.ensure(sizeof(int) * (size_t)(in.nb + 1))) != cudaSuccess) return e;
    // offsets padded for bulk copies that round their ranges up to 16 bytes
    if ((e = cb.off.ensure(sizeof(int) * (size_t)(in.nb + 1) + 64)) != cudaSuccess) return e;
    if ((e = cb.slots.ensure(sizeof(int) * (size_t)(ns > 0 ? ns : 1))) != cudaSuccess) return e;
    if ((e = cb.pos.ensure(sizeof(int) * (size_t)(ns > 0 ? ns : 1))) != cudaSuccess) return e;
    cudaMemsetAsync(cb.cnt.p, 0, sizeof(int) * (size_t)(in.nb + 1), s);
    cudaMemsetAsync(cb.cursor.p, 0, sizeof(int) * (size_t)(in.nb + 1), s);
    const int tb = 256;
    if (ns > 0) k_csr_count<<<(ns + tb - 1) / tb, tb, 0, s>>>(in, cb.cnt.as<int>());
    if ((e = exclusive_scan_i32(cb.cnt.as<int>(), cb.off.as<int>(), in.nb, cb.scan_tmp, s)) != cudaSuccess) return e;
    if (ns > 0) {
        k_csr_fill<<<(ns + tb - 1) / tb, tb, 0, s>>>(in, cb.off.as<int>(), cb.cursor.as<int>(), cb.slots.as<int>());
        k_csr_sort<<<(in.nb + tb - 1) / tb, tb, 0, s>>>(in.nb, cb.off.as<int>(), cb.slots.as<int>());
        k_csr_inverse<<<(ns + tb - 1) / tb, tb, 0, s>>>(ns, cb.slots.as<int>(), cb.pos.as<int>());
    }
    return cudaGetLastError();
}

}  // namespace mech
