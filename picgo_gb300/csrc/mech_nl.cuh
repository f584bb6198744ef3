// Inputs and scratch of the neighbor-list and CSR builds (mech_nl.cu).
#pragma once

#include "mech_internal.cuh"

namespace mech {

// What the list kernels need of a replica, uploaded in one copy per rebuild.
struct NLReplica {
    int4 dims;                 // bins along x, y, z; first bin
    float inv;                 // reciprocal of the bin edge (rounding slack included)
    float pre, sure;           // a single-precision squared distance above `pre` is out, one below `sure` is in
    double rmax2, rmin2;       // squared cutoffs rounded to float, held as double
    double bnd_cutoff;
    float bnd_cutoff_f;
    float reach;               // pre and sure hold up to this magnitude of a midpoint coordinate
    long long bnd_begin;       // first (plane, cylinder) entry
    int ncyl, cyl_begin, plane_begin;
};

struct NLInput {
    int ncyl;                  // all replicas
    const int* cyl_b1;         // internal index of the first bead (the second is +1)
    const int64_t* cyl_id;
    const int* cyl_fil;
    const int* cyl_pos;
    const int* cyl_rep;
    const void* x;             // current coordinates (engine format)
    int mixed;                 // 1: float hi/lo pairs, 0: doubles
    const NLReplica* rep;      // [R]
    int R;
    long long ncells;
};

struct PairBuild {
    DeviceBuffer cell_count, cell_start, sorted, midf, cell_of, keep, cnt, off, pairs, scan_tmp;
};

// Half pair list in two halves, with one read-back of the counts between them:
// count_pairs leaves the pair offset of every cylinder (and the total) in
// pb.off; write_pairs puts `total` (c, n) pairs into pb.pairs.
cudaError_t count_pairs(const NLInput& in, PairBuild& pb, cudaStream_t s);
cudaError_t write_pairs(const NLInput& in, PairBuild& pb, long long total, cudaStream_t s);

constexpr int kBndTile = 1024;   // entries per block of the boundary list kernels

struct BndInput {
    long long nq;              // sum over replicas of planes * cylinders
    int R;
    const NLReplica* rep;      // [R]
    const double* planes;      // [4 * planes]
    const float4* planes_f;    // [planes] the same in single precision
    const float4* midf;        // single-precision midpoints (count_pairs)
    const void* x;
    int mixed;
    const int* cyl_b1;
    const uint8_t* cyl_minus;  // filament minus-end cylinder
};

struct BndBuild {
    DeviceBuffer cnt, sums, off, bead, plane, scan_tmp, ncyl;
};

// cnt[q] (a byte, kept until the next rebuild) is 0 for an entry q = (plane,
// cylinder) outside the list, else the beads it contributes (2 for a minus-end
// cylinder); rep_offset[r] receives the list offset of replica r, [R] the
// total, and bb.ncyl the number of listed (plane, cylinder) entries.
cudaError_t count_boundary(const BndInput& in, BndBuild& bb, long long* rep_offset, cudaStream_t s);
cudaError_t write_boundary(const BndInput& in, BndBuild& bb, long long total, cudaStream_t s);

struct CsrInput {
    int nb;
    int base[5];               // slot ranges: linker, motor, exvol, boundary, end
    const int4* lk;
    const int4* mt;
    const int4* ev;
    const int* bb;
};

struct CsrBuild {
    DeviceBuffer cnt, cursor, off, slots, pos, scan_tmp;   // pos: slot -> its CSR position
};

cudaError_t build_csr(const CsrInput& in, CsrBuild& cb, cudaStream_t s);

}  // namespace mech
