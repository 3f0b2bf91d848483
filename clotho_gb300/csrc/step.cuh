// step.cuh -- device code that the fused step's kernels (k_prep.cu) share with the
// staged API's stages (k_step.cu, k_freespace.cu).
#pragma once

#include "engine.cuh"

namespace clotho {

// ---------------------------------------------------------------------------
// The item prefix of the generation kernel: rows_per_item rows of one population an
// item, its counters at zero.  The whole block calls it; npops <= kMaxPops <= its threads.
// N of population p: from the header, at most the capacity.
__device__ inline void begin_items(const PopDev* pops, uint32_t npops, const uint32_t* hdr, WorkCtl* ctl) {
    __shared__ uint32_t s_items[kMaxPops / 32u];
    const uint32_t p = threadIdx.x, lane = p & 31u, warp = p >> 5;
    const uint32_t rpi = ctl->rows_per_item ? ctl->rows_per_item : kRowsPerItem;
    if (p == 0) ctl->sched_at += 1u;
    const uint32_t n = p < npops ? (2u * min(hdr[2u * p], pops[p].Ncap) + rpi - 1u) / rpi : 0u;
    uint32_t incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += y;
    }
    if (p < kMaxPops && lane == 31u) s_items[warp] = incl;
    __syncthreads();
    if (p < npops) {
        uint32_t base = 0;
        for (uint32_t i = 0; i < warp; ++i) base += s_items[i];
        ctl->item_base[p] = base + incl - n;
        if (p == npops - 1u) {
            ctl->item_base[npops] = base + incl;
            ctl->gen_items = base + incl;
            ctl->gen_counter = 0;
            ctl->gen_counter_iv = 0;
            ctl->gen_counter_cm = 0;
        }
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------
// Trait t of new allele i (and, with trait 0, its slot, position and age).  Returns the change of the number of
// nonzero effects.
__device__ inline int resolve_mutation(const PopDev& P, uint32_t i, uint32_t t, uint32_t gen, uint32_t fr, uint32_t pA,
                                       uint32_t Alim) {
    const uint32_t slot = (i < fr) ? P.free_list[i] : pA + (i - fr);
    if (slot >= Alim) {
        if (t == 0) {
            atomicOr(&P.st->err, kErrAlleles);
            P.mut_slot[i] = 0xffffffffu;
        }
        return 0;
    }
    const bool philox = P.mode == kModePhilox;
    if (t == 0) {
        P.mut_slot[i] = slot;
        double pos;
        if (philox) {
            const U4 x = philox4x32(i, 0u, gen, kStreamMutAllele, P.seed);
            pos = u01(x.x, x.y);
        } else {
            pos = P.mut_pos[i];
        }
        P.pos[slot] = pos;
        P.age[slot] = gen;
    }
    float w = 0.0f;
    if (philox) {
        const U4 a = philox4x32(i, 1u + t, gen, kStreamMutAllele, P.seed);
        if (!(u01(a.x, a.y) < P.p_neutral)) {
            // Box-Muller on two fresh uniforms, first in (0,1]
            const double u1 = 1.0 - u01(a.z, a.w);
            const U4 b = philox4x32(i, 1u + kMaxTraits + t, gen, kStreamMutAllele, P.seed);
            const double u2 = u01(b.x, b.y);
            const double n = sqrt(-2.0 * log(u1)) * cospi(2.0 * u2);
            w = (float)(P.eff_mean + P.eff_sigma * n);
        }
    } else {
        w = P.mut_eff[(size_t)i * P.T + t];
    }
    const float old = P.eff[(size_t)slot * 4u + t];
    P.eff[(size_t)slot * 4u + t] = w;
    return (w != 0.0f) - (old != 0.0f);
}

// ---------------------------------------------------------------------------
// Column state of word w of the parent after the reference's tail padding
// (free_space_mt_population_space_row_interlaced.hpp:52-81): F = fixed bits,
// L = lost bits; padding bits are neither.
__device__ inline void padded_word(const PopDev& P, uint32_t w, uint32_t W, uint32_t A, uint32_t S,
                                   uint64_t& F, uint64_t& L) {
    if (w >= W) { F = 0; L = 0; return; }
    if (S == 0) {  // no genomes: every bit of every word reads as lost (:52-56)
        F = 0;
        L = ~0ull;
        return;
    }
    uint64_t valid;
    const uint32_t b = w * 64u;
    if (b + 64u <= A) valid = ~0ull;
    else if (b >= A) valid = 0ull;
    else valid = (1ull << (A - b)) - 1ull;
    F = P.accF[w] & valid;
    L = ~(P.accV[w] | ~valid);
}

// Block-wide exclusive scan of two counts per thread (1024 threads), the second in the upper half.
__device__ inline uint64_t block_excl_scan_1024(uint64_t v, uint64_t* s_warp, uint64_t& total) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint64_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint64_t t = s_warp[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint64_t y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= (uint32_t)o) t += y;
        }
        s_warp[lane] = t;  // inclusive warp totals
    }
    __syncthreads();
    total = s_warp[31];
    const uint64_t excl = x - v + (warp ? s_warp[warp - 1] : 0ull);
    __syncthreads();
    return excl;
}

// Free-space analysis of the parent (pN individuals, pA alleles, pW words) from accF/accV, one block of 1024
// threads: ordered compaction (fixed indices ascending, then lost indices ascending), fixed-table append
// (engine_batched_task.hpp:303-345), the fixed alleles' effect sum; then the accumulators and, for a population
// that counts columns in its generation kernel, the counts are reset for the child.  Rows of up to 1,024 words
// take one scan; the FP64 reduction (5.4 us of a block's narrow FP64 pipe) runs only in generations that fix an
// allele: without one the sum is exactly zero.
__device__ inline void fs_finalize_block(const PopDev& P, uint32_t pN, uint32_t pA, uint32_t pW, bool count_on) {
    __shared__ uint64_t s_warp[32];
    __shared__ double s_fx[32][kMaxTraits];
    __shared__ uint32_t s_any;   // warps that hold a fixed allele
    DevStatus* st = P.st;
    const uint32_t pS = 2u * pN;
    const uint32_t fx_base = st->fixed_total;
    // column counts of this step's child rows, for the populations that asked: zeroed here, added by the
    // generation kernel's counting build (the bitmap builds count: capacity <= kSufMaxSlots)
    const bool counting = count_on && st->count_cols != 0u && P.suf != nullptr && P.Acap <= kSufMaxSlots;
    if (counting)
        for (uint32_t a = threadIdx.x; a < P.Acap; a += 1024u) P.colcnt[a] = 0u;
    uint32_t totF = 0, totL = 0;
    double fsum[kMaxTraits] = {0.0, 0.0, 0.0, 0.0};
    bool fixed_here = false;
    if (pA > 0) {
        if (pW > 1024u) {  // the lost list starts behind every fixed index
            uint32_t cf = 0;
            for (uint32_t w = threadIdx.x; w < pW; w += 1024u) {
                uint64_t F, L;
                padded_word(P, w, pW, pA, pS, F, L);
                cf += __popcll(F);
            }
            uint64_t t;
            block_excl_scan_1024(cf, s_warp, t);
            totF = (uint32_t)t;
        }
        uint32_t base_f = 0;
        for (uint32_t c = 0; c < pW; c += 1024u) {
            const uint32_t w = c + threadIdx.x;
            uint64_t F, L, t;
            padded_word(P, w, pW, pA, pS, F, L);
            const uint64_t o =
                block_excl_scan_1024((uint64_t)__popcll(F) | ((uint64_t)__popcll(L) << 32), s_warp, t);
            if (pW <= 1024u) totF = (uint32_t)t;
            if (w < pW) {
                uint32_t i = base_f + (uint32_t)o;
                fixed_here |= F != 0ull;
                for (uint64_t b = F; b; b &= b - 1ull) {
                    const uint32_t slot = w * 64u + (uint32_t)(__ffsll((long long)b) - 1);
                    P.free_list[i] = slot;
                    const uint32_t k = fx_base + i;
                    for (uint32_t q = 0; q < P.T; ++q) fsum[q] += (double)P.eff[(size_t)slot * 4u + q];
                    if (k < P.FXcap) {  // m_fixed.append / m_fixed_traits.append (:315-324)
                        P.fx_pos[k] = P.pos[slot];
                        P.fx_age[k] = P.age[slot];
                        for (uint32_t q = 0; q < P.T; ++q) P.fx_eff[(size_t)k * P.T + q] = P.eff[(size_t)slot * 4u + q];
                    }
                    ++i;
                }
                i = totF + totL + (uint32_t)(o >> 32);
                for (uint64_t b = L; b; b &= b - 1ull) P.free_list[i++] = w * 64u + (uint32_t)(__ffsll((long long)b) - 1);
                P.fixmask[w] = F;
            }
            base_f += (uint32_t)t;
            totL += (uint32_t)(t >> 32);
        }
    }
    // effect sum of the fixed alleles (every parent row carries them): the
    // generation pass subtracts it from the carried per-genome sums
    if (threadIdx.x == 0) s_any = 0u;
    __syncthreads();
    if (totF && __any_sync(0xffffffffu, fixed_here)) {
        for (uint32_t t = 0; t < P.T; ++t) {
            double v = t == 0 ? fsum[0] : t == 1 ? fsum[1] : t == 2 ? fsum[2] : fsum[3];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if ((threadIdx.x & 31u) == 0) s_fx[threadIdx.x >> 5][t] = v;
        }
        if ((threadIdx.x & 31u) == 0) atomicOr(&s_any, 1u << (threadIdx.x >> 5));
    }
    __syncthreads();
    if (threadIdx.x < kMaxTraits) {
        double v = 0.0;
        if (threadIdx.x < P.T)
            for (uint32_t m = s_any; m; m &= m - 1u) v += s_fx[__ffs((int)m) - 1][threadIdx.x];
        st->fixsum[threadIdx.x] = v;
    }
    // reset the accumulators for the child of this step
    for (uint32_t w = threadIdx.x; w < P.Wcap; w += 1024u) {
        P.accF[w] = ~0ull;
        P.accV[w] = 0ull;
    }
    if (threadIdx.x == 0) {
        if (pA > 0) {
            st->fixed_cnt = totF;
            st->lost_cnt = totL;
            st->free_cnt = totF + totL;
            if (fx_base + totF > P.FXcap) atomicOr(&st->err, kErrFixed);
            st->fixed_total = min(P.FXcap, fx_base + totF);
        }
        st->cols_valid = counting ? 1u : 0u;
    }
}

}  // namespace clotho
