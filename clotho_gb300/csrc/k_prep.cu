// k_prep.cu -- everything a generation needs before its rows are written, in seven
// kernels: step header, free space, mutation counts and slots, parents, the rows'
// processing order, the position buckets; then the slots' ranks with the rows'
// crossover plans, and the suffix tables.
//
// A small population's step is bound by its launches: every dependent launch costs
// 3 to 4 us however little it does.  So work that does not depend on each other
// shares a launch (free space beside the mutation counts and the parent draws; both
// prefix sums beside the new alleles; the rows' order beside the bucket counts), a
// scan is one kernel (each block sums what lies before its chunk itself, as long as
// that is at most kDirectScan counts; above, one more launch leaves chunk sums), and
// every kernel is launched with programmatic dependent launch.
//
// A block works on one population (block_part); sizes are read from the device status
// words.
#include "plan.cuh"
#include "step.cuh"

#include <algorithm>

namespace clotho {

namespace {

constexpr uint32_t kChunk = 1024;  // counts a scan chunk: 256 threads x 4, or one a thread of a 1,024-thread block

// The step's offspring count: from the header, or (staged calls, after k_begin) from the status.
__device__ __forceinline__ uint32_t step_N(const PopDev& P, const uint32_t* hdr, uint32_t p) {
    return hdr ? min(hdr[2u * p], P.Ncap) : P.st->N;
}

// The rows' ordering keys are parent individuals; rows of an empty parent generation all have key 0.
__device__ __forceinline__ uint32_t order_keys(uint32_t pN) { return max(pN, 1u); }

// Sum of v over a block of 256 threads, in every thread.
__device__ __forceinline__ uint32_t block_sum_256(uint32_t v, uint32_t* s8) {
    v = __reduce_add_sync(0xffffffffu, v);
    __syncthreads();
    if ((threadIdx.x & 31u) == 0u) s8[threadIdx.x >> 5] = v;
    __syncthreads();
    uint32_t t = 0;
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) t += s8[i];
    return t;
}

// One chunk of an exclusive prefix sum over cnt[0, L): off (and cur, when given: scatter cursors) of the
// chunk's elements.  What lies before the chunk is summed from the counts (direct) or from the chunk sums.
// Returns the inclusive total at the chunk's end, in every thread.
__device__ __forceinline__ uint32_t scan_chunk(const uint32_t* cnt, const uint32_t* part, bool direct, uint32_t L,
                                               uint32_t c, uint32_t* off, uint32_t* cur, uint32_t* s8) {
    uint32_t v = 0;
    if (direct) {
        const uint4* q = reinterpret_cast<const uint4*>(cnt);
        for (uint32_t i = threadIdx.x; i < c * (kChunk / 4u); i += 256u) {
            const uint4 x = q[i];
            v += (x.x + x.y) + (x.z + x.w);
        }
    } else {
        for (uint32_t i = threadIdx.x; i < c; i += 256u) v += part[i];
    }
    uint32_t run = block_sum_256(v, s8);
    const uint32_t b = c * kChunk + threadIdx.x * 4u;
    uint32_t x[4];
    if (b + 4u <= L) {
        const uint4 q = *reinterpret_cast<const uint4*>(cnt + b);
        x[0] = q.x; x[1] = q.y; x[2] = q.z; x[3] = q.w;
    } else {
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) x[k] = (b + k < L) ? cnt[b + k] : 0u;
    }
    const uint32_t s = (x[0] + x[1]) + (x[2] + x[3]);
    uint32_t incl = s;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += y;
    }
    __syncthreads();  // block_sum_256's reads of s8 are done
    if (lane == 31u) s8[warp] = incl;
    __syncthreads();
    uint32_t total = run;
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
        if (i < warp) run += s8[i];
        total += s8[i];
    }
    run += incl - s;
    const uint32_t o4[4] = {run, run + x[0], run + x[0] + x[1], run + x[0] + x[1] + x[2]};
    if (b + 4u <= L) {
        if (off) *reinterpret_cast<uint4*>(off + b) = make_uint4(o4[0], o4[1], o4[2], o4[3]);
        if (cur) *reinterpret_cast<uint4*>(cur + b) = make_uint4(o4[0], o4[1], o4[2], o4[3]);
    } else {
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k)
            if (b + k < L) {
                if (off) off[b + k] = o4[k];
                if (cur) cur[b + k] = o4[k];
            }
    }
    return total;
}

// Parents of individual k (SelectionGenerator::update, general_fitness_selection_generator.hpp:45-69): uniform
// when every fitness is equal, else the FP64 inclusive prefix sum and an upper_bound per draw.
__device__ __forceinline__ uint2 draw_parents(const PopDev& P, uint32_t k, uint32_t Np, uint32_t gen, bool uni,
                                              double total) {
    const U4 x = philox4x32(k, 0u, gen, kStreamSelect, P.seed);
    const double u[2] = {u01(x.x, x.y), u01(x.z, x.w)};
    uint32_t id[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        if (Np == 0) id[h] = 0;
        else if (uni) {
            id[h] = (uint32_t)(u[h] * (double)Np);
            if (id[h] >= Np) id[h] = Np - 1u;
        }
    }
    if (Np != 0 && !uni) {
        // first i with cdf[i] > target (both >= +0: integer compares); the two searches go side by side
        const double t0 = u[0] * total, t1 = u[1] * total;
        uint32_t lo0 = 0, hi0 = Np, lo1 = 0, hi1 = Np;
        while ((lo0 < hi0) | (lo1 < hi1)) {
            const uint32_t m0 = (lo0 + hi0) >> 1, m1 = (lo1 + hi1) >> 1;
            const double c0 = P.cdf[min(m0, Np - 1u)], c1 = P.cdf[min(m1, Np - 1u)];
            if (lo0 < hi0) {
                if (lt_nonneg(t0, c0)) hi0 = m0; else lo0 = m0 + 1u;
            }
            if (lo1 < hi1) {
                if (lt_nonneg(t1, c1)) hi1 = m1; else lo1 = m1 + 1u;
            }
        }
        id[0] = lo0 >= Np ? Np - 1u : lo0;
        id[1] = lo1 >= Np ? Np - 1u : lo1;
    }
    return make_uint2(id[0], id[1]);
}

// The first blocks of a population take the first of a kernel's two independent jobs, the rest the second; a single
// block takes both.
struct Share {
    uint32_t i, n;
    bool on;
};
__device__ __forceinline__ Share first_share(const BlockPart& b, uint32_t first) {
    return b.n == 1u ? Share{0u, 1u, true} : Share{b.i, first, b.i < first};
}
__device__ __forceinline__ Share second_share(const BlockPart& b, uint32_t first) {
    return b.n == 1u ? Share{0u, 1u, true} : Share{b.i - first, b.n - first, b.i >= first};
}

}  // namespace

// ---------------------------------------------------------------------------
// Stage 1.  Block 0 of a population: the step header (the child becomes the parent,
// engine_batched_task.hpp:164; the sizes of the parent move to pN, pA, pW here, those of
// the child are written by stage 2, so that nobody reads what another block writes) and
// the free-space analysis of the parent.  The other blocks: device-drawn mutation counts
// with their chunk sums, or the tape's counted per row; parents, counted per parent for
// the rows' processing order.
//
// Device-drawn mutation counts are Poisson(mu) per offspring row.  The sum over
// rows is Poisson(2N mu) and, given the total, the rows are uniform -- the
// same law as M ~ Poisson(mu * 2N) with uniform target rows
// (mutation_allocator.hpp:41-47, batch_mutation_task_population_space_row.hpp:77).
template <bool ONE>
__global__ void __launch_bounds__(1024) k_stage1(const __grid_constant__ PopDev one, const PopDev* __restrict__ pops,
                                                 const BlockPart* __restrict__ map, uint32_t npops,
                                                 const uint32_t* __restrict__ hdr, WorkCtl* ctl, uint32_t what,
                                                 uint32_t count_on) {
    __shared__ uint32_t s_u32[33];
    const BlockPart part = block_part<ONE>(map);
    const PopDev& P = ONE ? one : pops[part.pop];
    pdl_wait();
    DevStatus* st = P.st;
    const bool philox = P.mode == kModePhilox;
    const uint32_t N = step_N(P, hdr, part.pop), S = 2u * N;
    if (part.i == 0) {
        if (!(what & kStepBegin)) return;
        const uint32_t pN = st->N, pA = st->A, pW = st->W;
        fs_finalize_block(P, pN, pA, pW, count_on != 0u);
        if (threadIdx.x == 0) {
            uint32_t err = 0, M = hdr[2u * part.pop + 1u];
            if (hdr[2u * part.pop] > P.Ncap) err |= kErrAlleles;
            if (M > P.Mcap) { err |= kErrMut; M = P.Mcap; }
            if (err) atomicOr(&st->err, err);
            st->pN = pN;
            st->pA = pA;
            st->pW = pW;
            st->M = M;
            st->ev_used = 0;
        }
        return;
    }
    const uint32_t bx = part.i - 1u, nb = part.n - 1u, p = part.pop;
    if (p == 0 && bx == 0 && (what & kStepBegin)) begin_items(pops, npops, hdr, ctl);
    if (what & kStepMut) {
        if (philox) {
            const uint32_t gen = st->gen;
            const double* cdf = P.pois_mu;
            for (uint32_t c = bx; c * kChunk < S; c += nb) {
                const uint32_t r = c * kChunk + threadIdx.x;
                uint32_t n = 0;
                if (r < S) {
                    const U4 x = philox4x32(r, 0u, gen, kStreamMutCount, P.seed);
                    n = poisson_tab(u01(x.x, x.y), cdf, cdf[kPoisTab], P.mu);
                    P.row_cnt[r] = n;
                }
                n = __reduce_add_sync(0xffffffffu, n);
                if ((threadIdx.x & 31u) == 0u) s_u32[threadIdx.x >> 5] = n;
                __syncthreads();
                if (threadIdx.x < 32u) {
                    n = __reduce_add_sync(0xffffffffu, s_u32[threadIdx.x]);
                    if (threadIdx.x == 0) P.scan_upart[c] = n;
                }
                __syncthreads();
            }
        } else {
            const uint32_t M = min(hdr[2u * p + 1u], P.Mcap);
            for (uint32_t i = bx * 1024u + threadIdx.x; i < M; i += nb * 1024u) {
                const uint32_t s = P.mut_seq[i];
                if (s >= S) { atomicOr(&st->err, kErrSeq); continue; }
                atomicAdd(&P.row_cnt[s], 1u);
            }
        }
    }
    if (what & kStepOrder) {
        const uint32_t Np = hdr ? st->N : st->pN;  // staged calls have moved the sizes already
        uint32_t* const cnt = P.plan_row ? P.ord_cnt : nullptr;
        if (philox && (what & kStepSelect)) {
            const bool uni = st->fit_const != 0u || !(st->fit_total > 0.0);
            const double total = st->fit_total;
            const uint32_t gen = st->gen;
            for (uint32_t k = bx * 1024u + threadIdx.x; k < N; k += nb * 1024u) {
                const uint2 id = draw_parents(P, k, Np, gen, uni, total);
                *reinterpret_cast<uint2*>(P.pairs + 2u * k) = id;
                if (cnt) {
                    atomicAdd(cnt + id.x, 1u);
                    atomicAdd(cnt + id.y, 1u);
                }
            }
        } else if (cnt) {
            for (uint32_t g = bx * 1024u + threadIdx.x; g < S; g += nb * 1024u) {
                const uint32_t id = P.pairs[g];
                atomicAdd(cnt + (id < Np ? id : 0u), 1u);
            }
        }
    }
}

// Chunk sums of the counts that a scan cannot sum by itself (which == 0: new alleles per row, 1: rows per
// parent, 2: positions per bucket).
template <bool ONE>
__global__ void __launch_bounds__(256) k_chunk_sums(const __grid_constant__ PopDev one,
                                                    const PopDev* __restrict__ pops,
                                                    const BlockPart* __restrict__ map,
                                                    const uint32_t* __restrict__ hdr, uint32_t which) {
    __shared__ uint32_t s8[8];
    const BlockPart part = block_part<ONE>(map);
    const PopDev& P = ONE ? one : pops[part.pop];
    pdl_wait();
    const uint32_t L = which == 0 ? 2u * step_N(P, hdr, part.pop) : which == 1 ? order_keys(P.st->pN) : P.NB;
    const uint32_t* cnt = which == 0 ? P.row_cnt : which == 1 ? P.ord_cnt : P.bcnt;
    uint32_t* sums = which == 1 ? P.scan_opart : P.scan_upart;
    if (!cnt) return;
    for (uint32_t c = part.i; c * kChunk < L; c += part.n) {
        uint32_t v = 0;
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
            const uint32_t i = c * kChunk + 256u * k + threadIdx.x;
            if (i < L) v += cnt[i];
        }
        v = block_sum_256(v, s8);
        if (threadIdx.x == 0) sums[c] = v;
    }
}

// ---------------------------------------------------------------------------
// Stage 2.  The prefix sums of the new alleles per row and of the rows per parent, and
// the new alleles themselves: mutation i takes free_indices[i]; beyond the free list new
// slots are appended at the parent allele count (batch_mutation_mt.hpp:69-80).  Writes
// the allele table (AlleleGenerator, allele_generator_vector.hpp:76-83) and the trait
// table (TraitSpaceGenerator2, trait_space_generator.hpp:118-129).  One thread per new
// allele and trait, neighbours in different blocks: a drawn effect is about a hundred
// operations of the narrow FP64 pipe, so they are spread over all SMs.
template <bool ONE>
__global__ void __launch_bounds__(256) k_stage2(const __grid_constant__ PopDev one, const PopDev* __restrict__ pops,
                                                const BlockPart* __restrict__ map, const uint32_t* __restrict__ hdr,
                                                uint32_t what, uint32_t direct_max) {
    __shared__ uint32_t s8[8];
    const BlockPart part = block_part<ONE>(map);
    const PopDev& P = ONE ? one : pops[part.pop];
    pdl_wait();
    DevStatus* st = P.st;
    const bool philox = P.mode == kModePhilox;
    const uint32_t N = step_N(P, hdr, part.pop), S = 2u * N;
    const uint32_t a = max(1u, part.n / 3u);
    const Share res = first_share(part, a), scan = second_share(part, a);
    if (res.on && (what & kStepMut)) {
        uint32_t M = 0;
        if (philox) {  // stage 1 left the chunk sums
            for (uint32_t i = threadIdx.x; i * kChunk < S; i += 256u) M += P.scan_upart[i];
            M = block_sum_256(M, s8);
        } else {
            M = st->M;
        }
        const uint32_t Mraw = M;
        M = min(M, P.Mcap);
        const uint32_t fr = st->free_cnt, pA = st->pA, gen = st->gen, T = P.T;
        const uint32_t Ac = pA + (M > fr ? M - fr : 0u), A = min(Ac, P.Acap);
        if (res.i == 0 && threadIdx.x == 0) {
            if (Ac > P.Acap) atomicOr(&st->err, kErrAlleles);
            if (Mraw > P.Mcap) atomicOr(&st->err, kErrMut);
            st->N = N;
            st->A = A;
            st->W = ref_width(A);
            st->cur ^= 1u;
            if (philox) st->M = M;
        }
        int nz_delta = 0;
        for (uint64_t q = (uint64_t)threadIdx.x * res.n + res.i; q < (uint64_t)M * T; q += 256ull * res.n) {
            const uint32_t i = (uint32_t)(q / T), t = (uint32_t)(q % T);
            nz_delta += resolve_mutation(P, i, t, gen, fr, pA, A);
        }
        if (nz_delta) atomicAdd(&st->nz_eff, nz_delta);
        __syncthreads();
    }
    if (!scan.on) return;
    // units: the row chunks, then the parent chunks
    const uint32_t keys = order_keys(st->pN);
    const uint32_t nr = (what & kStepMut) ? S / kChunk + 1u : 0u;
    const uint32_t no = ((what & kStepOrder) && P.plan_row) ? (keys + kChunk - 1u) / kChunk : 0u;
    for (uint32_t u = scan.i; u < nr + no; u += scan.n) {
        if (u < nr) {
            const uint32_t total = scan_chunk(P.row_cnt, P.scan_upart, !philox && S <= direct_max, S, u, P.row_off,
                                              philox ? nullptr : P.row_cur, s8);
            if (u == nr - 1u && threadIdx.x == 0) P.row_off[S] = total;
        } else {
            scan_chunk(P.ord_cnt, P.scan_opart, keys <= direct_max, keys, u - nr, nullptr, P.ord_cur, s8);
        }
    }
}

// ---------------------------------------------------------------------------
// Stage 3.  The first step of the slots' ranks, the rows' processing
// positions (parent-major order: rows sorted by parent individual, so rows reading the
// same parent strands run side by side and the second read of a strand is an L2 hit;
// the order inside one parent does not matter), the tape's new alleles grouped by row;
// the counts of stage 1 go back to zero.
//
// Ranks of many slots: positions per bucket here, grouped by stages 4 and 5, ranked beside the plans.  Of few
// (DIRECT, at most kDirectRanks slots of capacity): all of it here, by one or eight blocks in shared memory, which saves three
// launches.
struct RankSmem {   // dynamic shared memory of the DIRECT form
    uint64_t key[kDirectRanks];       // positions grouped by bucket, as integers of the same order
    uint32_t off[kDirectRanks + 4];   // counts, then offsets, per bucket
    uint16_t slot[kDirectRanks];
    uint16_t inv[kDirectRanks];
    uint32_t s32[32];
};

// Block c of n: the ranks of the slots in its share of the buckets (all count them, which spares a launch or a wait
// between blocks).  One block is bound by its SM's instruction issue: 2,700 slots 7.7 us by one block, 6.8 by four, 6.5
// by eight; a generation of 10,000 individuals 40.3, 38.7, 38.3.
__device__ __forceinline__ void rank_block(const PopDev& P, uint32_t A, RankSmem& z, uint32_t c, uint32_t n) {
    constexpr uint32_t kItems = kDirectRanks / 1024u;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, NB = P.NB, per = NB >> 10;
    for (uint32_t i = tid; i < NB; i += 1024u) z.off[i] = 0u;
    double x[kItems];
#pragma unroll
    for (uint32_t j = 0; j < kItems; ++j) x[j] = tid + 1024u * j < A ? P.pos[tid + 1024u * j] : 0.0;
    __syncthreads();
    uint32_t at[kItems];   // bucket, and the place in it
#pragma unroll
    for (uint32_t j = 0; j < kItems; ++j)
        if (tid + 1024u * j < A) {
            const uint32_t b = pos_bucket(x[j], NB);
            at[j] = b | atomicAdd(&z.off[b], 1u) << 16;
        }
    __syncthreads();
    // exclusive prefix of the counts: four or eight buckets a thread (capacities come in steps of 4,096 slots)
    uint4* const off4 = reinterpret_cast<uint4*>(z.off) + tid * (per >> 2);
    uint4 n0 = off4[0], n1 = per > 4u ? off4[1] : make_uint4(0, 0, 0, 0);
    const uint32_t s = n0.x + n0.y + n0.z + n0.w + n1.x + n1.y + n1.z + n1.w;
    uint32_t incl = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += y;
    }
    if (lane == 31u) z.s32[warp] = incl;
    __syncthreads();
    uint32_t t = z.s32[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, t, o);
        if (lane >= (uint32_t)o) t += y;
    }
    const uint32_t before = __shfl_sync(0xffffffffu, t, warp ? warp - 1u : 0u);
    uint32_t run = (warp ? before : 0u) + incl - s;
    auto advance = [&run](uint4& q) {
        const uint4 c = q;
        q = make_uint4(run, run + c.x, run + c.x + c.y, run + c.x + c.y + c.z);
        run = q.w + c.w;
    };
    advance(n0);
    advance(n1);
    off4[0] = n0;
    if (per > 4u) off4[1] = n1;
    if (tid == 1023u) z.off[NB] = A;
    __syncthreads();
    const uint32_t b0 = NB / n * c, b1 = c + 1u < n ? b0 + NB / n : NB, k0 = z.off[b0], ke = z.off[b1];
    for (uint32_t i = b0 + tid; i <= b1; i += 1024u) P.boff[i] = z.off[i];
    uint32_t mine = 0;
#pragma unroll
    for (uint32_t j = 0; j < kItems; ++j)
        if (tid + 1024u * j < A && (at[j] & 0xffffu) - b0 < b1 - b0) {
            mine |= 1u << j;
            const uint32_t k = z.off[at[j] & 0xffffu] + (at[j] >> 16);
            z.key[k] = pos_key(x[j]);
            z.slot[k] = (uint16_t)(tid + 1024u * j);
        }
    __syncthreads();
    // what is in bucket or rank order leaves from shared memory, neighbours by neighbouring threads: stored as each
    // thread came to it, every lane's store was a wavefront of its own (neutral run of 10,000: the stage 10.6 us, so 9.0)
    for (uint32_t k = k0 + tid; k < ke; k += 1024u) P.bpos[k] = key_pos(z.key[k]);
#pragma unroll
    for (uint32_t j = 0; j < kItems; ++j) {
        if (!((mine >> j) & 1u)) continue;
        const uint32_t me = tid + 1024u * j;
        const uint64_t key = pos_key(x[j]);
        const uint32_t b = at[j] & 0xffffu, k1 = z.off[b + 1u];
        uint32_t r = z.off[b];
        for (uint32_t k = r; k < k1; ++k) r += (z.key[k] < key || (z.key[k] == key && z.slot[k] < me)) ? 1u : 0u;
        P.rank[me] = r;
        z.inv[r] = (uint16_t)me;
    }
    __syncthreads();
    for (uint32_t r = k0 + tid; r < ke; r += 1024u) P.inv[r] = z.inv[r];
}

template <bool ONE, bool DIRECT>
__global__ void __launch_bounds__(DIRECT ? 1024 : 256)
k_stage3(const __grid_constant__ PopDev one, const PopDev* __restrict__ pops, const BlockPart* __restrict__ map,
         uint32_t what, uint32_t rankers) {
    extern __shared__ __align__(16) uint8_t s_raw[];
    constexpr uint32_t kThreads = DIRECT ? 1024u : 256u;
    const BlockPart part = block_part<ONE>(map);
    const PopDev& P = ONE ? one : pops[part.pop];
    pdl_wait();
    const DevStatus* st = P.st;
    const uint32_t A = st->A;
    // DIRECT: the first blocks rank the slots, the others do the rest
    if (DIRECT && part.i < rankers) {
        rank_block(P, A, *reinterpret_cast<RankSmem*>(s_raw), part.i, rankers);
        return;
    }
    const uint32_t at = (part.i - (DIRECT ? rankers : 0u)) * kThreads + threadIdx.x;
    const uint32_t step = (part.n - (DIRECT ? rankers : 0u)) * kThreads;
    const uint32_t N = st->N, pN = st->pN, S = 2u * N;
    if (!DIRECT)
        for (uint32_t s = at; s < A; s += step) atomicAdd(&P.bcnt[pos_bucket(P.pos[s], P.NB)], 1u);
    if ((what & kStepOrder) && P.plan_row) {
        for (uint32_t g = at; g < S; g += step) {
            const uint32_t id = P.pairs[g];
            P.ord_pos[g] = atomicAdd(&P.ord_cur[id < pN ? id : 0u], 1u);
        }
        for (uint32_t k = at; k < order_keys(pN); k += step) P.ord_cnt[k] = 0u;
    }
    if (what & kStepMut) {
        if (P.mode != kModePhilox) {
            const uint32_t M = st->M;
            for (uint32_t i = at; i < M; i += step) {
                const uint32_t s = P.mut_seq[i];
                if (s < S) P.row_mut[atomicAdd(&P.row_cur[s], 1u)] = i;
            }
        }
        for (uint32_t r = at; r < S; r += step) P.row_cnt[r] = 0u;
    }
}

// Ascending order of a[0..n): insertion sort for short lists, heapsort beyond
// (a tape may send many mutations to one row).
static __device__ void sort_ascending(uint32_t* a, uint32_t n) {
    if (n <= 16u) {
        for (uint32_t i = 1; i < n; ++i) {
            const uint32_t x = a[i];
            uint32_t j = i;
            for (; j > 0 && a[j - 1] > x; --j) a[j] = a[j - 1];
            a[j] = x;
        }
        return;
    }
    auto sift = [a](uint32_t r, uint32_t end) {
        const uint32_t x = a[r];
        for (uint32_t c = 2u * r + 1u; c < end; c = 2u * r + 1u) {
            if (c + 1u < end && a[c + 1u] > a[c]) ++c;
            if (a[c] <= x) break;
            a[r] = a[c];
            r = c;
        }
        a[r] = x;
    };
    for (uint32_t r = n / 2u; r-- > 0;) sift(r, n);
    for (uint32_t end = n - 1u; end > 0; --end) {
        const uint32_t x = a[0];
        a[0] = a[end];
        a[end] = x;
        sift(0, end);
    }
}

// Each tape row's new alleles in ascending mutation index (the list order is the order in which their FP32 effects
// enter the row's carried phenotype, so it must not depend on the order of the scatter's atomics).  One thread per
// list position; the thread at a row's first position sorts the row's list: ownership is decided by position, which
// never moves, and every entry of a row's segment names that row, so no other thread acts on it.
__device__ __forceinline__ void sort_tape_lists(const PopDev& P, uint32_t at, uint32_t step) {
    const uint32_t listed = P.row_off[2u * P.st->N];
    for (uint32_t t = at; t < listed; t += step) {
        const uint32_t s = P.mut_seq[P.row_mut[t]];
        const uint32_t off = P.row_off[s], n = P.row_off[s + 1u] - off;
        if (t == off && n >= 2u) sort_ascending(P.row_mut + off, n);
    }
}

// ---------------------------------------------------------------------------
// Stage 4.  The prefix sum of the positions per bucket, and the tape rows' lists in order.
template <bool ONE>
__global__ void __launch_bounds__(256) k_stage4(const __grid_constant__ PopDev one, const PopDev* __restrict__ pops,
                                                const BlockPart* __restrict__ map, uint32_t what,
                                                uint32_t direct_max) {
    __shared__ uint32_t s8[8];
    const BlockPart part = block_part<ONE>(map);
    const PopDev& P = ONE ? one : pops[part.pop];
    pdl_wait();
    for (uint32_t c = part.i; c * kChunk < P.NB; c += part.n) {
        const uint32_t total = scan_chunk(P.bcnt, P.scan_upart, P.NB <= direct_max, P.NB, c, P.boff, P.bcur, s8);
        if ((c + 1u) * kChunk >= P.NB && threadIdx.x == 0) P.boff[P.NB] = total;
    }
    if ((what & kStepMut) && P.mode != kModePhilox)
        sort_tape_lists(P, part.i * 256u + threadIdx.x, part.n * 256u);
}

// Stage 5.  Positions and slots grouped by bucket; the bucket counts go back to zero.
template <bool ONE>
__global__ void __launch_bounds__(256) k_stage5(const __grid_constant__ PopDev one, const PopDev* __restrict__ pops,
                                                const BlockPart* __restrict__ map) {
    const BlockPart part = block_part<ONE>(map);
    const PopDev& P = ONE ? one : pops[part.pop];
    pdl_wait();
    const uint32_t at = part.i * 256u + threadIdx.x, step = part.n * 256u;
    const uint32_t A = P.st->A;
    for (uint32_t s = at; s < A; s += step) {
        const double x = P.pos[s];
        const uint32_t k = atomicAdd(&P.bcur[pos_bucket(x, P.NB)], 1u);
        P.bpos[k] = x;
        P.bslot[k] = s;
    }
    for (uint32_t b = at; b < P.NB; b += step) P.bcnt[b] = 0u;
}

// ---------------------------------------------------------------------------
// The rows' plans, and beside them what does not depend on them: the slots' ranks (both need only the position
// buckets), or, with DIRECT ranks, the suffix table and the tape rows' lists.

// suf[g * Wcap + w] = bits of word w whose slot has rank >= 64 g, for
// g = 0 .. ceil(A/64) (the last row is empty).  A unit of work is 32 words and
// every kSufSlices-th table row; the units are spread over the blocks from
// the current width, so the blocks are busy however wide the capacity is.
constexpr uint32_t kSufSlices = 16;
__device__ __forceinline__ void build_suffix_table(const PopDev& P, uint32_t block, uint32_t blocks,
                                                   uint32_t (*s_grp)[65]) {   // (rank >> 6) + 1 per slot, 0 beyond A
    const uint32_t tx = threadIdx.x & 31u, ty = threadIdx.x >> 5;
    const uint32_t A = P.st->A, W = P.st->W;
    const uint32_t Gt = (A + 63u) >> 6;
    const uint32_t wblocks = (W + 31u) / 32u;
    for (uint32_t u = block; u < wblocks * kSufSlices; u += blocks) {
        const uint32_t wb = (u % wblocks) * 32u, slice = u / wblocks;
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < 2048u; i += 256u) {
            const uint32_t s = wb * 64u + i;
            s_grp[i >> 6][i & 63u] = (s < A) ? (P.rank[s] >> 6) + 1u : 0u;
        }
        __syncthreads();
        const uint32_t w = wb + tx;
        if (w >= W) continue;
        for (uint32_t g = slice * 8u + ty; g <= Gt; g += kSufSlices * 8u) {
            uint64_t m = 0;
#pragma unroll 16
            for (uint32_t b = 0; b < 64u; ++b) m |= (uint64_t)(s_grp[tx][b] > g) << b;
            P.suf[(size_t)g * P.Wcap + w] = m;
        }
    }
}

template <bool ONE, bool DIRECT>
__global__ void __launch_bounds__(256, 4) k_plan(const __grid_constant__ PopDev one, const PopDev* __restrict__ pops,
                                                 const BlockPart* __restrict__ map, uint32_t what, uint32_t first) {
    __shared__ uint32_t s_cr[256][kPlanSmemEv + 1];
    __shared__ double s_cdf[kPoisTab + 1];
    __shared__ uint32_t s_grp[DIRECT ? 32 : 1][65];
    const BlockPart part = block_part<ONE>(map);
    const PopDev& P = ONE ? one : pops[part.pop];
    pdl_wait();
    const DevStatus st = *P.st;
    const uint32_t a = ONE ? first : max(1u, part.n / first);
    const Share side = first_share(part, a), plan = second_share(part, a);
    if (side.on) {
        if (DIRECT) {
            if ((what & kStepMut) && P.mode != kModePhilox)
                sort_tape_lists(P, side.i * 256u + threadIdx.x, side.n * 256u);
            build_suffix_table(P, side.i, side.n, s_grp);
        } else {
            for (uint32_t s = side.i * 256u + threadIdx.x; s < st.A; s += side.n * 256u) slot_rank(P, s);
        }
    }
    if (!P.plan_row || !plan.on) return;
    if (threadIdx.x <= kPoisTab) s_cdf[threadIdx.x] = P.pois_rho[threadIdx.x];
    __syncthreads();
    for (uint32_t v0 = plan.i * 256u; v0 < 2u * st.N; v0 += plan.n * 256u) {
        plan_row(P, st, v0 + threadIdx.x, s_cdf, s_cr[threadIdx.x]);
    }
}

// The suffix tables of populations whose ranks k_plan has made.
template <bool ONE>
__global__ void __launch_bounds__(256) k_suf_build(const __grid_constant__ PopDev one,
                                                   const PopDev* __restrict__ pops,
                                                   const BlockPart* __restrict__ map) {
    __shared__ uint32_t s_grp[32][65];
    const BlockPart part = block_part<ONE>(map);
    const PopDev& P = ONE ? one : pops[part.pop];
    pdl_wait();
    if (P.suf) build_suffix_table(P, part.i, part.n, s_grp);
}

uint32_t launch_plan(const LaunchCfg& L, const PopDev* pops, uint32_t npops, const PrepSizes& z, uint32_t maxW,
                     uint32_t what) {
    const uint32_t np = z.tables ? blocks_for(z.maxS, 256) : 0u, units = (maxW + 31u) / 32u * kSufSlices;
    // Blocks for the tables: as many as there are units, at most half as many as for the rows, but eight (a unit is a
    // dependent chain of its own: 16 of them in one block made a generation of 100 individuals 29.7 us, in eight
    // 25.7); in a batch an eighth of each population's.
    if (direct_ranks(z)) {
        const uint32_t ns = std::min(units, std::max(np / 2u, 8u)), g = blocks_of(L, ns + np, 8);
        launch_pops(L, kTablePlan, k_plan<true, true>, k_plan<false, true>, g, pops, npops, what,
                    npops == 1u ? ns : 8u);
        return 1u;
    }
    const uint32_t nr = blocks_for(z.maxA, 256), g = blocks_of(L, nr + np, 8);
    const uint32_t ns = npops > 1u ? (z.tables ? 4u : 1u) : (z.tables ? std::max(1u, g / 4u) : g);
    launch_pops(L, kTablePlan, k_plan<true, false>, k_plan<false, false>, g, pops, npops, what, ns);
    if (!z.tables) return 1u;
    launch_pops(L, kTable256, k_suf_build<true>, k_suf_build<false>, blocks_of(L, units, 4), pops, npops);
    return 2u;
}

uint32_t launch_prep(const LaunchCfg& L, const PopDev* pops, uint32_t npops, const PrepSizes& z, const uint32_t* hdr,
                     WorkCtl* ctl, uint32_t what, bool count_on) {
    // up to this many counts a scan block sums what lies before its chunk by itself: at 32,768 counts the last
    // block reads 128 KB of L2, about as long as the extra launch that it saves
    constexpr uint32_t kDirectScan = 32768;
    uint32_t n = 0;
    auto sums = [&](uint32_t most, uint32_t which) {
        launch_pops(L, kTable256, k_chunk_sums<true>, k_chunk_sums<false>, blocks_of(L, blocks_for(most, kChunk), 4), pops, npops,
                    hdr, which);
        ++n;
    };
    if (what & (kStepBegin | kStepMut | kStepOrder)) {
        launch_pops(L, kTable1024, k_stage1<true>, k_stage1<false>,
                    1u + blocks_of(L, blocks_for(z.maxS, kChunk), std::max(1u, L.ind_per_sm / 4u)), pops, npops, npops,
                    hdr, ctl, what, count_on ? 1u : 0u);
        ++n;
        // chunk sums: of the tape's counts (device draws leave their own in stage 1), of the rows per parent
        if ((what & kStepMut) && (what & kStepTape) && z.maxS > kDirectScan) sums(z.maxS, 0u);
        if ((what & kStepOrder) && z.tables && z.maxN > kDirectScan) sums(z.maxN, 1u);
        const uint32_t units = blocks_for(z.maxS + 1u, kChunk) + blocks_for(z.maxN, kChunk);
        launch_pops(L, kTable256, k_stage2<true>, k_stage2<false>, blocks_of(L, units + (uint32_t)L.num_sms, 6), pops, npops, hdr,
                    what, kDirectScan);
        ++n;
    }
    const uint32_t rest = blocks_for(z.maxS, 256);
    if (direct_ranks(z)) {
        const uint32_t rankers = npops == 1u ? 8u : 1u;   // a batch's populations have two blocks at least
        launch_pops_smem(L, kTable1024, k_stage3<true, true>, k_stage3<false, true>,
                         rankers + blocks_of(L, blocks_for(z.maxS, 1024), 2), sizeof(RankSmem), pops, npops, what, rankers);
        return n + 1u;
    }
    launch_pops(L, kTable256, k_stage3<true, false>, k_stage3<false, false>,
                blocks_of(L, std::max(rest, blocks_for(z.maxA, 256)), 8), pops, npops, what, 0u);
    if (z.maxNB > kDirectScan) sums(z.maxNB, 2u);
    launch_pops(L, kTable256, k_stage4<true>, k_stage4<false>, blocks_of(L, blocks_for(z.maxNB, kChunk), 4), pops, npops, what,
                kDirectScan);
    launch_pops(L, kTable256, k_stage5<true>, k_stage5<false>, blocks_of(L, blocks_for(std::max(z.maxNB, z.maxA), 256), 8), pops,
                npops);
    return n + 3u;
}

// ---------------------------------------------------------------------------
// A small tape's arrays in one launch: the host has packed them into one pinned block, which the threads read over
// the chip-to-chip link, 16 bytes each.  (Seven copies from pageable memory cost 10 us each on the host, 88 us a
// call at 10,007 individuals, where the bytes take 3.)
__global__ void __launch_bounds__(256) k_tape_upload(const TapePieces z, uint32_t* __restrict__ hdr) {
    pdl_wait();
    const uint32_t at = blockIdx.x * 256u + threadIdx.x, step = gridDim.x * 256u;
    if (at == 0) {
        hdr[0] = z.N;
        hdr[1] = z.M;
    }
    for (uint32_t i = at; i < z.end[6]; i += step) {
        uint32_t begin = 0;
#pragma unroll
        for (uint32_t k = 0; k < 7; ++k) {
            if (i >= begin && i < z.end[k])
                static_cast<uint4*>(z.dst[k])[i - begin] = __ldcv(static_cast<const uint4*>(z.src[k]) + (i - begin));
            begin = z.end[k];
        }
    }
}
void launch_tape_upload(const LaunchCfg& L, const TapePieces& z, uint32_t* hdr) {
    const uint32_t g = std::min(blocks_for(z.end[6], 256), (uint32_t)L.num_sms * 2u);
    launch_k(L, k_tape_upload, dim3(g), dim3(256), z, hdr);
}

__global__ void __launch_bounds__(256) k_pack_traits(const double* __restrict__ src, double* __restrict__ dst, uint32_t n,
                                                     uint32_t T) {
    for (uint32_t i = blockIdx.x * 256u + threadIdx.x; i < n; i += gridDim.x * 256u)
        for (uint32_t t = 0; t < T; ++t) dst[(size_t)i * T + t] = src[(size_t)i * 4u + t];
}
void launch_pack_traits(const LaunchCfg& L, const double* src, double* dst, uint32_t n, uint32_t T) {
    k_pack_traits<<<std::min(blocks_for(n, 256), (uint32_t)L.num_sms * 8u), 256, 0, L.stream>>>(src, dst, n, T);
}

// ---------------------------------------------------------------------------
// A population's Poisson CDF tables, made once with it (thread 0: breakpoints per gamete, thread 1: new alleles
// per row): 64 dependent FP64 steps, 10 us, that a block of the plan kernel would otherwise spend each generation.
__global__ void k_pois_tables(PopDev P) {
    if (threadIdx.x > 1u) return;
    const double lambda = threadIdx.x ? P.mu : P.rho;
    double* t = threadIdx.x ? P.pois_mu : P.pois_rho;
    double pk = threadIdx.x ? P.exp_neg_mu : P.exp_neg_rho, F = pk;
    t[0] = F;
    for (uint32_t k = 1; k < kPoisTab; ++k) {
        poisson_step(pk, F, lambda, k);
        t[k] = F;
    }
    t[kPoisTab] = pk;
}
void launch_pois_tables(cudaStream_t s, const PopDev& P) { k_pois_tables<<<1, 32, 0, s>>>(P); }

int init_recip_prep() { return fill_recip_table(); }

// ---------------------------------------------------------------------------
// Parent sampling on its own (staged API).
__global__ void k_select_philox(const PopDev* __restrict__ pops, uint32_t npops) {
    for (uint32_t p = blockIdx.z; p < npops; p += gridDim.z) {
        const PopDev& P = pops[p];
        const DevStatus* st = P.st;
        const bool uni = st->fit_const != 0u || !(st->fit_total > 0.0);
        for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < st->N; k += gridDim.x * blockDim.x)
            *reinterpret_cast<uint2*>(P.pairs + 2u * k) = draw_parents(P, k, st->pN, st->gen, uni, st->fit_total);
    }
}
void launch_select_philox(const LaunchCfg& L, const PopDev* pops, uint32_t npops) {
    k_select_philox<<<pop_grid(npops, L.num_sms * 2u, L.num_sms, L.ind_per_sm), 256, 0, L.stream>>>(pops, npops);
}

}  // namespace clotho
