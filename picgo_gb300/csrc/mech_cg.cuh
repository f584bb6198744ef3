// The per-replica reductions and CG step logic of the device-resident
// minimizer (CGMethod.hpp:238-373 and :826-1743, ForceFieldManager.cpp:96-290;
// paths relative to medyan-5.4.0/src), run by the finalizer kernels, one block
// per replica, behind an evaluation's last partial sums.
#pragma once

#include "mech_device.cuh"

namespace mech {

// whether a pass of mode `trial` evaluates a second trial for a replica in state S
__device__ __forceinline__ bool second_trial(int trial, int dual) {
    return trial == kTrialBoth || (trial == kTrialDual && dual);
}

__device__ __forceinline__ bool replica_selected(const CGState& S, int want) {
    return want < 0 ? (S.active != 0) : (S.phase == want);
}

// ---------------------------------------------------------------------------
// finalizers (run by the whole last block of a replica)
// ---------------------------------------------------------------------------
// Partial-sum slots of a replica's tile range [b, e): the FP64 kernels write
// one per tile (stride 1); the persistent mixed kernels write one per run of
// tiles, at b and at every multiple of their tiles-per-block inside (b, e).
__device__ __forceinline__ int run_slots(int b, int e, int stride) {
    const int m0 = (b / stride + 1) * stride;
    return 1 + (m0 < e ? (e - 1 - m0) / stride + 1 : 0);
}
__device__ __forceinline__ int run_slot(int b, int stride, int k) {
    return k == 0 ? b : (b / stride + 1) * stride + (k - 1) * stride;
}

// A thread's slots k = threadIdx.x, + kBlock, ... of `nslot`, in order: `load(k)`
// reads one without conditions (what a pass does not need is read and not added),
// `add` adds it.  Beyond kBlock slots the loads of kAhead slots are issued
// together, the first behind that of slot threadIdx.x; up to kBlock (4,000 to
// 60,000 cylinders) there is nothing to batch, and the guards cost 2 us.  1M
// cylinders: mixed energy loads 4.3 -> 2.2 us; FP64 reductions 14.0 and 15.0 ->
// 10.3 and 8.0 us.
template <int kAhead, typename Load, typename Add>
__device__ __forceinline__ void for_slots(int nslot, Load&& load, Add&& add) {
    const int t = threadIdx.x;
    decltype(load(0)) s0;
    if (t < nslot) s0 = load(t);
    if (nslot <= kBlock) {
        if (t < nslot) add(s0);
        return;
    }
    decltype(load(0)) s[kAhead];
    for (int k0 = kBlock; k0 < nslot; k0 += kAhead * kBlock) {
#pragma unroll
        for (int q = 0; q < kAhead; ++q)
            if (k0 + q * kBlock + t < nslot) s[q] = load(k0 + q * kBlock + t);
        if (k0 == kBlock) add(s0);
#pragma unroll
        for (int q = 0; q < kAhead; ++q)
            if (k0 + q * kBlock + t < nslot) add(s[q]);
    }
}

// The CG step logic of the finalizers runs in thread 0 on a register copy of
// its replica's state, loaded at the start so that the loads overlap the
// block's reduction, and stored back once: done field by field on global
// memory, the branchy logic waits on one dependent load after another.
// Per force field energies of one evaluation from the reduced partial sums
// `e`, with the numeric fallback energies of the replica's flagged pairs
// added in pair order (only entries recorded at step `lam` when `match_lam`).
// A failed pair makes the force field report -1 (CylinderExclVolRepulsion.cpp:442-481).
template <typename Real>
__device__ void add_fallback_energies(const DevNet<Real>& n, int r, int fb_count, bool match_lam, double lam,
                                      double* e) {
    const int cnt = min(fb_count, kExvolFallbackCap);
    int last = -1;
    bool ev_failed = false;
    for (;;) {
        int best = -1, bestPair = 0x7fffffff;
        for (int k = 0; k < cnt; ++k) {
            const int rep = __ldcg(n.ev_fb_list + 2 * k), pr = __ldcg(n.ev_fb_list + 2 * k + 1);
            if (rep != r || pr <= last || pr >= bestPair) continue;
            if (match_lam &&
                __longlong_as_double(__ldcg((const long long*)n.ev_fb_energy + kExvolFallbackCap + k)) != lam)
                continue;
            best = k;
            bestPair = pr;
        }
        if (best < 0) break;
        const double u = __ldcg(n.ev_fb_energy + best);
        if (u == -1.0) ev_failed = true;
        else e[MECH_FF_EXVOL] += u;
        last = bestPair;
    }
    if (ev_failed) e[MECH_FF_EXVOL] = -1.0;
}

// The evaluation's per force field energies into S.eval; returns the
// computeEnergy value (+inf when a force field failed).
__device__ __forceinline__ double record_energies(CGState& S, const double* e) {
    double tot = 0.0;
    bool failed = false;
    for (int k = 0; k < MECH_NUM_FF; ++k) {
        S.eval[k] = e[k];
        tot += e[k];
        if (e[k] <= -1) failed = true;
    }
    S.eval[MECH_NUM_FF] = tot;
    S.evalFailed = failed;
    S.numEnergyEval++;
    return failed ? (1.0 / 0.0) : tot;
}

// The finalizers take the replica's tile ranges and (thread 0) a register copy
// of its state, both loaded by the kernel at its start together with the
// phase it selects on: on this GPU every dependent round trip to L2 (partial
// slots written by the other die's SMs) costs about a microsecond, and a
// finalizer is a chain of them on the minimizer's critical path.
constexpr int kFinSums = 16;   // sums of the energy finalizer: two trials' six fields and d . F, to a power of two

template <typename Real>
__device__ void finalize_energy(const DevNet<Real>& n, int r, int trial, const RepTiles& rt, CGState& S, double* sh) {
    const int stride = sizeof(Real) == 4 ? n.ptiles[0] : 1;
    const int nslot = run_slots(rt.fil_begin, rt.fil_end, stride);
    const int ffk[K_NUM_SPARSE] = {MECH_FF_LINKER, MECH_FF_MOTOR, MECH_FF_EXVOL, MECH_FF_BOUNDARY};
    double e[MECH_NUM_FF], e2[MECH_NUM_FF], slope;
    const bool dual = sizeof(Real) == 4 && second_trial(trial, n.st[r].dual);
    const bool pend = trial && n.st[r].dPending;   // the pass formed a new direction
    // the fallback list's length, loaded now so that thread 0's step logic does
    // not wait on it at the end
    const int fb_count = threadIdx.x == 0 ? __ldcg(n.ev_fb_count) : 0;
    MECH_TRACE_STAMP(ts_load);
    if constexpr (sizeof(Real) == 4) {
        // mixed: (hi, lo) pair slots summed compensated in single precision;
        // the doubles are formed in warp 0 only.  acc[0, 6): the (first) trial,
        // acc[6, 12): the second trial, acc[12]: d . F of a new direction.
        FF acc[kFinSums];
        // each sparse kind's first slot of this thread, loaded with the first filament slots
        float2 sp0[K_NUM_SPARSE], sp1[K_NUM_SPARSE];
#pragma unroll
        for (int k = 0; k < K_NUM_SPARSE; ++k) {
            const int i = rt.sp_begin[k] + threadIdx.x;
            sp0[k] = sp1[k] = make_float2(0.f, 0.f);
            if (i < rt.sp_end[k]) {
                sp0[k] = load_pair(n.part_sp + i);
                if (dual) sp1[k] = load_pair(n.part_sp2 + i);
            }
        }
        struct Slot {
            float4 u, v;
            float2 w;
        };
        for_slots<3>(
            nslot,
            [&](int k) {
                const int i = run_slot(rt.fil_begin, stride, k);
                const float4* p = reinterpret_cast<const float4*>(n.part_fil + 4 * (size_t)i);
                return Slot{__ldcg(p), __ldcg(p + 1), load_pair(n.part_df + i)};
            },
            [&](const Slot& s) {
                add_pair(acc[MECH_FF_STRETCHING], make_float2(s.u.x, s.u.y));
                add_pair(acc[MECH_FF_BENDING], make_float2(s.u.z, s.u.w));
                if (dual) {
                    add_pair(acc[MECH_NUM_FF + MECH_FF_STRETCHING], make_float2(s.v.x, s.v.y));
                    add_pair(acc[MECH_NUM_FF + MECH_FF_BENDING], make_float2(s.v.z, s.v.w));
                }
                if (pend) add_pair(acc[2 * MECH_NUM_FF], s.w);
            });
#pragma unroll
        for (int k = 0; k < K_NUM_SPARSE; ++k) {
            const int i0 = rt.sp_begin[k] + threadIdx.x;
            if (i0 < rt.sp_end[k]) {
                add_pair(acc[ffk[k]], sp0[k]);
                if (dual) add_pair(acc[MECH_NUM_FF + ffk[k]], sp1[k]);
            }
#pragma unroll 4
            for (int i = i0 + blockDim.x; i < rt.sp_end[k]; i += blockDim.x) {
                add_pair(acc[ffk[k]], load_pair(n.part_sp + i));
                if (dual) add_pair(acc[MECH_NUM_FF + ffk[k]], load_pair(n.part_sp2 + i));
            }
        }
        MECH_TRACE_SECTION(n, TK_SEC_FE_LOAD, ts_load);
        MECH_TRACE_STAMP(ts_red);
        const FF sum = block_pair_sums<kFinSums>(acc, reinterpret_cast<float*>(sh));
        MECH_TRACE_SECTION(n, TK_SEC_FE_REDUCE, ts_red);
        if (threadIdx.x >= 32) return;
        // hi + lo in double, one pair per lane of warp 0: an FP64 warp
        // instruction costs the same with 1 or 13 active lanes
        const double v = (double)sum.h + (double)sum.l;
#pragma unroll
        for (int k = 0; k < MECH_NUM_FF; ++k) {
            e[k] = __shfl_sync(0xffffffffu, v, k);
            e2[k] = __shfl_sync(0xffffffffu, v, MECH_NUM_FF + k);
        }
        slope = __shfl_sync(0xffffffffu, v, 2 * MECH_NUM_FF);
        if (threadIdx.x != 0) return;
    } else {
        // every thread issues its loads back to back, then sums in a fixed order
        double acc[8] = {};   // the six fields, d . F of a new direction
        struct Slot {
            double2 v;
            double w;
        };
        for_slots<8>(
            nslot,
            [&](int k) {
                const size_t i = (size_t)(rt.fil_begin + k);
                return Slot{__ldcg(reinterpret_cast<const double2*>(n.part_fil + 4 * i)), __ldcg(n.part_df + i)};
            },
            [&](const Slot& s) {
                acc[MECH_FF_STRETCHING] += s.v.x;
                acc[MECH_FF_BENDING] += s.v.y;
                if (pend) acc[MECH_NUM_FF] += s.w;
            });
#pragma unroll
        for (int k = 0; k < K_NUM_SPARSE; ++k) {
#pragma unroll 8
            for (int i = rt.sp_begin[k] + threadIdx.x; i < rt.sp_end[k]; i += blockDim.x)
                acc[ffk[k]] += __ldcg(n.part_sp + i);
        }
        const double v = block_sums<8>(acc, sh);
        if (threadIdx.x >= 32) return;
#pragma unroll
        for (int k = 0; k < MECH_NUM_FF; ++k) e[k] = __shfl_sync(0xffffffffu, v, k);
        slope = __shfl_sync(0xffffffffu, v, MECH_NUM_FF);
        if (threadIdx.x != 0) return;
    }
    MECH_TRACE_STAMP(ts_tail);
    const double lam = S.lambda;   // the (first) trial's step, before the line search moves it
    const int xb = S.xbuf;
    add_fallback_energies(n, r, fb_count, dual, lam, e);
    const double E = record_energies(S, e);
    if (trial && S.phase == PH_LS_TRIAL && S.dPending) {
        if (S.backupPending) {
            S.backupValid = 1;
            S.backupPending = 0;
        }
        S.dPending = 0;
        if (slope <= 0) {
            // conjugacy lost (CGMethod.hpp:1553-1560): the search starts over
            // along F, at the same step; this pass's energies are not used
            S.dIsF = 1;
            S.slope = S.FdotF;
            S.lastFdotF = S.FdotF;
        } else {
            S.slope = slope;
            S.dIsF = 0;
            S.dbuf ^= 1;
            if (S.method >= 1) S.lastFdotF = S.newGrad;
        }
        S.reducedSlope = (S.safeMode ? 0.0 : kBacktrackSlope) * S.slope;
        if (S.dIsF) {
            n.st[r] = S;
            return;
        }
    }
    if (trial && S.phase == PH_LS_TRIAL) {
        S.Etrial = E;
        // the trial positions: the other buffer (FP64), or the next of three (mixed)
        line_search_step(S, E, sizeof(Real) == 4 ? (xb + 1) % 3 : xb ^ 1);
        if (dual && S.phase == PH_LS_TRIAL) {
            // rejected at lambda and halved: the reference's next trial, at
            // lambda / 2, was evaluated by the same pass (positions in the third buffer)
            add_fallback_energies(n, r, fb_count, true, S.lambda, e2);
            const double E2 = record_energies(S, e2);
            S.Etrial = E2;
            line_search_step(S, E2, (xb + 2) % 3);
        } else if (dual) {
            S.numEnergyEval++;   // the second trial was evaluated but not needed
        }
    } else if (S.phase == PH_RECOVER_ENERGY) {
        S.E0 = E;
        S.phase = PH_RESET;
    } else {
        S.E0 = E;
    }
    settle(S);
    n.st[r] = S;
    MECH_TRACE_SECTION(n, TK_SEC_FE_TAIL, ts_tail);
}

// Whether the direction F + beta F_prev, of a search that follows one along F_prev,
// has lost conjugacy for certain: its slope F.F + beta F.F_prev is negative by more
// than the pass that forms the direction can round it.  That pass adds rounded
// products, whose magnitudes' sum is at most |F|^2 + beta |F| |F_prev|, and that at
// most |F|^2 + beta (|F|^2 + |F_prev|^2) / 2 (no roots in thread 0): ten roundings of
// single precision at the most with compensated sums, and in FP64 as many as its
// longest chain of additions has (60 with 1M beads).  The bound is 40 and 4,500 of
// them.  Squares near underflow and an overflowing beta are left to the pass.
// A call: inlined, the iterations that never get here took 0.1 us longer.
template <typename Real>
__device__ __noinline__ bool conjugacy_lost(double ff, double ffp, double ff_prev, double beta) {
    constexpr double kRound = sizeof(Real) == 4 ? 2.4e-6 : 1e-12;
    return ff > 1e-30 && ff_prev > 1e-30 && beta < 1e30 &&
           ff + beta * ffp < -kRound * (ff + 0.5 * beta * (ff + ff_prev));
}

// CG bookkeeping after the forces (CGMethod.hpp:1540-1580): max |F|, beta.
template <typename Real>
__device__ __forceinline__ void force_step(CGState& S, double mx, double ff, double ffp) {
    const int ph = S.phase;
    const double ff_prev = S.FdotF;
    if (ph == PH_FORCE || ph == PH_RECOVER_FORCE) S.numForceCall++;
    S.maxF = mx;
    S.FdotF = ff;
    S.fbuf ^= 1;
    if (!isfinite(mx)) {   // CGMethod::maxF throws (CGMethod.hpp:207-210)
        S.status = MECH_ERR_NONFINITE;
        S.phase = PH_ERROR;
        return;
    }
    if (ph == PH_FORCE) {
        S.energyRelChange = fabs(S.newEnergy - S.prevEnergy) / fabs(S.prevEnergy);
        S.prevEnergy = S.newEnergy;
        double beta = 0.0;
        if (S.method == 1) {
            S.newGrad = ff;
            beta = S.newGrad / S.lastFdotF;
        } else if (S.method == 2) {
            S.newGrad = ff;
            S.prevGrad = ffp;
            beta = fmax(0.0, (S.newGrad - S.prevGrad) / S.lastFdotF);
        }
        S.beta = beta;
        // minimum-energy backup once past half the call limit (CGMethod.hpp:1564-1566)
        if (mx <= 10 * S.gradTol && S.numIter > S.forceCallLimit / 2 && S.totalEnergy <= S.minimumE) {
            S.minimumE = S.totalEnergy;
            S.backupPending = 1;
        }
        // The new direction F + beta d is formed by the first pass of the search,
        // which starts the search over along F where it finds conjugacy lost.  A
        // search along F is followed by such a loss in most iterations of a long
        // run (20,517 of 21,105 with 4,000 cylinders), and there d . F is known
        // already: no pass is spent on it (75.1 -> 47 us per iteration, FP64 92.5 -> 71.6).
        // A pending backup is written by the pass that forms the direction.
        if (S.dIsF && !S.backupPending && conjugacy_lost<Real>(ff, ffp, ff_prev, beta)) {
            S.slope = ff;
            S.lastFdotF = ff;
        } else {
            S.dPending = 1;
        }
        begin_iteration(S);
        settle(S);
    } else if (ph == PH_RECOVER_FORCE) {
        S.phase = PH_RECOVER_ENERGY;
    }
}

template <typename Real>
__device__ void finalize_force(const DevNet<Real>& n, int r, const RepTiles& rt, CGState& S, double* sh) {
    // k_force_gather writes one slot per tile, k_force_gather_mx one per run of
    // a replica's tiles in a block
    const int stride = sizeof(Real) == 4 ? n.gtiles : 1;
    const int nslot = run_slots(rt.fil_begin, rt.fil_end, stride);
    double mx, ff, ffp;
    MECH_TRACE_STAMP(ts_load);
    if constexpr (sizeof(Real) == 4) {
        // mixed slots hold float maxima and (hi, lo) pairs; sum them compensated
        // in single precision and form the doubles in thread 0 only
        FF a[2];
        float m = 0.f;
#pragma unroll 4
        for (int k = threadIdx.x; k < nslot; k += blockDim.x) {
            const float* p = reinterpret_cast<const float*>(n.part_fil + 4 * (size_t)run_slot(rt.fil_begin, stride, k));
            const float4 v = __ldcg(reinterpret_cast<const float4*>(p));
            const float w = __ldcg(p + 4);
            m = fmaxf(m, v.x);
            a[0].add(v.y);
            a[0].add(v.z);
            a[1].add(v.w);
            a[1].add(w);
        }
        MECH_TRACE_SECTION(n, TK_SEC_FF_LOAD, ts_load);
        MECH_TRACE_STAMP(ts_red);
        // the maxima, none negative, are ordered like their bits
        unsigned* s_mx = reinterpret_cast<unsigned*>(sh + 32);
        const unsigned wm = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
        if ((threadIdx.x & 31) == 0) s_mx[threadIdx.x >> 5] = wm;
        const FF s = block_pair_sums<2>(a, reinterpret_cast<float*>(sh));   // its barrier publishes s_mx
        const double sum = (double)s.h + (double)s.l;
        ff = sum;
        ffp = __shfl_sync(0xffffffffu, sum, 1);
        MECH_TRACE_SECTION(n, TK_SEC_FF_REDUCE, ts_red);
        if (threadIdx.x != 0) return;
        unsigned bm = 0;
#pragma unroll
        for (int k = 0; k < kBlock / 32; ++k) bm = max(bm, s_mx[k]);
        mx = (double)__uint_as_float(bm);
    } else {
        unsigned long long a_mx = 0;
        double a_ff = 0.0, a_ffp = 0.0;
        struct Slot {
            double2 v;
            double w;
        };
        for_slots<8>(
            nslot,
            [&](int k) {
                const double* p = n.part_fil + 4 * (size_t)(rt.fil_begin + k);
                return Slot{__ldcg(reinterpret_cast<const double2*>(p)), __ldcg(p + 2)};
            },
            [&](const Slot& s) {
                a_mx = max(a_mx, (unsigned long long)__double_as_longlong(s.v.x));
                a_ff += s.v.y;
                a_ffp += s.w;
            });
        // the maxima, none negative, are ordered like their bits, off the FP64 pipe
        unsigned long long m[1] = {a_mx};
        const unsigned long long bm = block_maxima<1>(m, reinterpret_cast<unsigned long long*>(sh));
        double v[2] = {a_ff, a_ffp};
        const double s = block_sums<2>(v, sh + 32);
        mx = __longlong_as_double((long long)bm);
        ff = s;
        ffp = __shfl_sync(0xffffffffu, s, 1);
        if (threadIdx.x != 0) return;
    }
    MECH_TRACE_STAMP(ts_tail);
    force_step<Real>(S, mx, ff, ffp);
    n.st[r] = S;
    MECH_TRACE_SECTION(n, TK_SEC_FF_TAIL, ts_tail);
}

}  // namespace mech
