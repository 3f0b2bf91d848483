// plan.cuh -- position ranks of the slots and the rows' crossover plans: device code of the
// plan kernels (k_prep.cu) and of the interval classifier (k_generation.cu).
#pragma once

#include "engine.cuh"

namespace clotho {

constexpr uint32_t kCmMaxEv = 16;     // chunk-mask build: breakpoints a row takes through the table
constexpr uint32_t kPlanSmemEv = 16;  // breakpoints of a row that are ranked in shared memory

// r(e) = #{slots with position < e} through the position buckets.
__device__ __forceinline__ uint32_t threshold_rank(const PopDev& P, double e) {
    const uint32_t b = pos_bucket(e, P.NB);
    const uint32_t k0 = P.boff[b], k1 = P.boff[b + 1u];
    uint32_t r = k0;
    for (uint32_t k = k0; k < k1; ++k) r += pos_lt(P.bpos[k], e) ? 1u : 0u;
    return r;
}
// Of two breakpoints, their chains of dependent loads side by side.
__device__ __forceinline__ uint2 threshold_ranks(const PopDev& P, double e0, double e1) {
    const uint32_t a = pos_bucket(e0, P.NB), b = pos_bucket(e1, P.NB);
    const uint32_t a0 = P.boff[a], a1 = P.boff[a + 1u], b0 = P.boff[b], b1 = P.boff[b + 1u];
    const uint32_t n = max(a1 - a0, b1 - b0);
    uint2 r = make_uint2(a0, b0);
    for (uint32_t k = 0; k < n; ++k) {
        if (a0 + k < a1) r.x += pos_lt(P.bpos[a0 + k], e0) ? 1u : 0u;
        if (b0 + k < b1) r.y += pos_lt(P.bpos[b0 + k], e1) ? 1u : 0u;
    }
    return r;
}

// Position as an integer of the same order (equal for both zeros).
__device__ __forceinline__ uint64_t pos_key(double x) {
    const uint64_t b = (uint64_t)__double_as_longlong(x);
    return b == 0x8000000000000000ull ? b : (b >> 63) ? ~b : b | 0x8000000000000000ull;
}
__device__ __forceinline__ double key_pos(uint64_t key) {   // both zeros: +0
    return __longlong_as_double((long long)((key >> 63) ? key & 0x7fffffffffffffffull : ~key));
}

// Nearest suffix-table row b (a multiple of 64) of rank threshold r and the
// ranks between them: [c0, c0 + n), n <= 32.
__device__ __forceinline__ uint32_t table_row(uint32_t r, uint32_t A, uint32_t& c0, uint32_t& n) {
    const uint32_t lo = r & ~63u;
    const uint32_t b = (r - lo <= 32u) ? lo : lo + 64u;
    c0 = min(r, b);
    n = min(max(r, b), A) - c0;
    return b;
}

// A slot's rank = slots in lower buckets + slots of its own bucket with a smaller position
// (or the same position and a lower slot index).  inv is the inverse map (rank -> slot).
__device__ __forceinline__ void slot_rank(const PopDev& P, uint32_t s) {
    const double x = P.pos[s];
    const uint32_t b = pos_bucket(x, P.NB);
    const uint32_t k0 = P.boff[b], k1 = P.boff[b + 1u];
    uint32_t r = k0;
    for (uint32_t k = k0; k < k1; ++k) {
        const double y = P.bpos[k];
        r += (y < x || (y == x && P.bslot[k] < s)) ? 1u : 0u;
    }
    P.rank[s] = r;
    if (P.inv) P.inv[r] = s;
}

// The plan of row v of the suffix-table classifier, one thread per row (whole warps call it): the top strand
// (parent individual and strand swap), the breakpoint count, and for every breakpoint its nearest table row and
// correction ranks; plus the direction of the phenotype gather.  Device-drawn breakpoints get their plan entries
// from a warp-aggregated counter; tape rows use the tape's own event offsets.  cdf: the population's Poisson(rho)
// table, searched with integer compares, so a breakpoint count costs no FP64 work.  own: kPlanSmemEv words of
// shared memory of this thread.
__device__ __forceinline__ void plan_row(const PopDev& P, const DevStatus& st, uint32_t v, const double* cdf,
                                         uint32_t* own) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t S = 2u * st.N, A = st.A, Se = (S + 1u) >> 1;
    const bool philox = P.mode == kModePhilox, q1 = (P.flags & 1u) != 0;
    const bool live = v < S;
    // even gametes on the first half of the threads, odd ones on the second:
    // under the reference's crossover rule odd gametes are copy rows, so a
    // warp holds one kind of row
    const uint32_t g = v < Se ? 2u * v : 2u * (v - Se) + 1u;
    uint32_t pind = 0, E = 0, base = 0, flags = 0;
    bool swap = false;
    if (live) {
        pind = P.pairs[g];
        if (pind >= st.pN) {
            atomicOr(&P.st->err, kErrParent);
            pind = 0;
        }
        if (philox) {
            const U4 x = philox4x32(g, 0u, st.gen, kStreamGamete, P.seed);
            E = (q1 && (g & 1u)) ? 0u : poisson_tab(u01(x.x, x.y), cdf, cdf[kPoisTab], P.rho);
            swap = lt_nonneg(u01(x.z, x.w), P.bias);
            if (E > kMaxEvDevice) {
                atomicOr(&P.st->err, kErrEvents);
                E = kMaxEvDevice;
            }
        } else {
            swap = P.swap[g] != 0;
            base = P.ev_off[g];
            E = (q1 && (g & 1u)) ? 0u : P.ev_off[g + 1u] - base;
        }
    }
    if (philox) {  // warp-aggregated allocation of the plan entries
        uint32_t incl = E;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += y;
        }
        const uint32_t tot = __shfl_sync(0xffffffffu, incl, 31);
        uint32_t b0 = 0;
        if (lane == 0 && tot) b0 = atomicAdd(&P.st->ev_used, tot);
        base = __shfl_sync(0xffffffffu, b0, 0) + incl - E;
        if (E && base + E > P.EVcap) {
            atomicOr(&P.st->err, kErrEvents);
            E = 0;
        }
    }
    if (!live) return;
    // what the plan entry needs besides the breakpoints, fetched before the breakpoint work so that
    // their round trips overlap it: the processing position, the new alleles' CSR range, and the
    // carried phenotypes of both parent strands (one 64-byte line; the gather direction picks one)
    const uint32_t at = P.ord_pos[g];
    const uint32_t mo = P.row_off[g], mend = P.row_off[g + 1u];
    const uint32_t topr = 2u * pind + (swap ? 1u : 0u);
    asm volatile("prefetch.global.L1 [%0];" ::"l"(P.zg[st.cur ^ 1u] + (size_t)(topr & ~1u) * 4u));
    if (E > kMaxEvDevice) {
        flags = kPlanLong;  // tape rows with very long event lists: direct compares
    } else if (E > 0) {
        uint32_t* cr = E <= kPlanSmemEv ? own : P.plan_cr + base;
        // the chunk-mask build classifies rows of more than kCmMaxEv breakpoints by direct compares
        // against their positions, which device-drawn rows keep in the event list for it (every
        // population's, to keep the plan kernel uniform; rare: E > 16)
        const bool keep_pos = philox && E > kCmMaxEv;
        for (uint32_t k = 0; k < E; k += 2u) {
            double e0, e1 = 0.0;
            if (philox) {
                const U4 a = philox4x32(g, 1u + (k >> 1), st.gen, kStreamGamete, P.seed);
                e0 = u01(a.x, a.y);
                e1 = u01(a.z, a.w);
                if (keep_pos) {
                    P.ev_pos[base + k] = e0;
                    if (k + 1u < E) P.ev_pos[base + k + 1u] = e1;
                }
            } else {
                e0 = P.ev_pos[base + k];
                if (k + 1u < E) e1 = P.ev_pos[base + k + 1u];
            }
            if (k + 1u < E) {
                const uint2 r = threshold_ranks(P, e0, e1);
                cr[k] = r.x;
                cr[k + 1u] = r.y;
            } else {
                cr[k] = threshold_rank(P, e0);
            }
        }
        // share of the rank space the breakpoints switch: sorted thresholds pair into intervals.  A threshold counts
        // by the parity of its place in the order (equal ones in list order); each pair is compared once.
        int64_t len = (E & 1u) ? (int64_t)A : 0;
        if (E <= kPlanSmemEv) {
            uint32_t odd = 0;
            for (uint32_t k = 1; k < E; ++k) {
                const uint32_t rk = cr[k];
                uint32_t here = 0;
                for (uint32_t j = 0; j < k; ++j) {
                    const uint32_t before = cr[j] <= rk ? 1u : 0u;
                    here ^= before;
                    odd ^= (before ^ 1u) << j;
                }
                odd |= here << k;
            }
            for (uint32_t k = 0; k < E; ++k) len += ((odd >> k) & 1u) ? (int64_t)cr[k] : -(int64_t)cr[k];
        } else {
            for (uint32_t k = 0; k < E; ++k) {
                const uint32_t rk = cr[k];
                uint32_t posn = 0;
                for (uint32_t j = 0; j < E; ++j) {
                    const uint32_t rj = cr[j];
                    posn += (rj < rk || (rj == rk && j < k)) ? 1u : 0u;
                }
                len += (posn & 1u) ? (int64_t)rk : -(int64_t)rk;
            }
        }
        if (2 * len > (int64_t)A) flags |= kPlanInv;
        for (uint32_t k = 0; k < E; ++k) {
            uint32_t c0, n;
            const uint32_t b = table_row(cr[k], A, c0, n);
            P.plan_go[base + k] = (b >> 6) * P.Wcap;
            P.plan_cr[base + k] = c0 | (n << 20);
        }
    }
    if (E > kPlanMaxEvents) {
        atomicOr(&P.st->err, kErrEvents);
        E = 0;
        flags = 0;
    }
    P.plan_row[at] = make_uint4(g, topr, base, E | (flags << kPlanFlagShift));
    // what the row's set-up would otherwise fetch after its plan: the new alleles' CSR
    // range and the carried phenotype's base strand value less the fixed effects (as good as always
    // zero, which subtracts to the bit: then the narrow FP64 pipe is left alone)
    P.plan_mut[at] = make_uint2(mo, mend - mo);
    const uint32_t zs = ((flags & kPlanInv) && st.nz_eff != 0) ? topr ^ 1u : topr;
    const double2* zp = reinterpret_cast<const double2*>(P.zg[st.cur ^ 1u] + (size_t)zs * 4u);
    double2 z0 = zp[0], z1 = zp[1];
    if (st.fixsum[0] != 0.0 || st.fixsum[1] != 0.0 || st.fixsum[2] != 0.0 || st.fixsum[3] != 0.0) {
        z0.x -= st.fixsum[0];
        z0.y -= st.fixsum[1];
        z1.x -= st.fixsum[2];
        z1.y -= st.fixsum[3];
    }
    double2* out = reinterpret_cast<double2*>(P.plan_z + (size_t)at * 4u);
    out[0] = z0;
    out[1] = z1;
}

}  // namespace clotho
