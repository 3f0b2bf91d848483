// k_analysis.cu -- pairwise differences between sampled sequences.
//
// The reference's statistic (association_matrix_pairwise_difference.hpp:75-120
// on the CPU, cuda/analysis/pairwise_difference_kernel.hpp:56-339 on its GPU
// path): for every pair i < j of a sample of rows, the number of allele slots
// where the two sequences differ, popcount(row_i XOR row_j); summarised by
// count, total, min, max, mean and variance (and, from the distances, the
// median).
//
// popcount(a XOR b) = |a| + |b| - 2 |a AND b|, and |a AND b| over all pairs is the product of the
// sample's 0/1 matrix with its transpose: a contraction, so it runs on the tensor cores.
#include "engine.cuh"

#include <algorithm>

namespace clotho {

namespace {
constexpr uint32_t kTM = 128, kTN = 256;        // pairs a CTA takes: rows i of the tile, rows j
constexpr uint32_t kRowWarps = (kTM + kTN) / 32u;             // warps that expand rows, 32 each
constexpr uint32_t kPairThreads = (kRowWarps + 1u) * 32u;     // and one that issues the multiplications
constexpr uint32_t kRing = 4;                   // stages of 128 slots in shared memory
constexpr uint32_t kRound = 8;                  // stages from one load of the rows: 128 bytes of each
constexpr uint32_t kStageBytes = (kTM + kTN) * 128u;
constexpr uint32_t kMaxSlots = 1u << 19;        // slots a CTA sums up: counts stay far below 2^24 units
constexpr uint32_t kTileSums = kTM * kTN + kTM + kTN;   // counts of a tile whose slots several CTAs share
constexpr uint32_t kSplitTiles = 1024;          // tiles whose slots are shared at a time: 136 MB of counts
constexpr uint32_t kPairWait = 1u << 20;        // try_wait rounds before a CTA gives up

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// false: given up, by this warp or (fail) by another one of the CTA
__device__ __forceinline__ bool wait_parity(uint32_t bar, uint32_t parity, volatile uint32_t* fail) {
    for (uint32_t it = 0; it < kPairWait && !*fail; ++it) {
        uint32_t ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    *fail = 1u;
    return false;
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

// Shared-memory operand of K-major rows of 128 bytes in the 128-byte swizzle: groups of eight rows 1,024 bytes apart.
__device__ __forceinline__ uint64_t operand(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(1024u >> 4) << 32) | (1ull << 46) | (2ull << 61);
}

__device__ __forceinline__ void mma_f8(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)accumulate)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void load_32_columns(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
}  // namespace

// One CTA takes a 128 x 256 tile of the pair matrix (tiles with a pair i < j only) and a range of the slots.
// A warp loads 128 bytes of each of its 32 rows, eight lanes a row, for eight stages; in a stage every lane turns 16
// of a row's slots into 16 bytes of 0 or 1: bit k of each byte of a 32-bit word becomes a byte (two operations for
// four slots; which slots make up a stage is the same for all rows, which is all a sum needs), in the
// 128-byte swizzle that the tensor core reads.  A byte of 1 is the e4m3 value 2^-9, so products are 2^-18
// and sums are whole multiples of it, exact in FP32.  A warp of its own issues the four K = 32 steps of a stage when
// the twelve others have arrived on its barrier; a stage is filled again when its multiplications have ended, so warps
// run up to four stages apart (a block barrier a stage: 4,001 rows of 320 words 226 us, this 187).  Bound by
// shared memory: 48 KB written and 48 KB read, 768 clocks, for a stage's 512 of multiplication; a stage takes 985.
// splits > 1 (few tiles): the CTAs of a tile add their counts into tile_sum, the last one to come finishes the
// tile; no CTA waits for another.  (popcount of 64 x 64 tiles: 1.1 ms for 4,001 rows of 320 words, the popcount
// unit's 16 words a clock and SM.)
__global__ void __launch_bounds__(kPairThreads, 1)
k_pairwise(const PopDev* __restrict__ pops, uint32_t p, const uint32_t* __restrict__ sample, uint32_t n,
           uint32_t tile0, uint32_t splits, uint32_t per, uint32_t* __restrict__ tile_sum,
           uint32_t* __restrict__ tile_done, uint32_t* __restrict__ dist, PairwiseOut* __restrict__ out) {
    extern __shared__ uint8_t s_raw[];
    __shared__ __align__(8) unsigned long long s_full[kRing], s_free[kRing], s_end;
    __shared__ uint32_t s_tmem, s_last, s_fail, s_issued;
    __shared__ uint32_t s_ones[kTM + kTN];
    __shared__ unsigned long long s_sum[kRowWarps], s_sq[kRowWarps], s_cnt[kRowWarps];
    __shared__ uint32_t s_min[kRowWarps], s_max[kRowWarps];
    const PopDev& P = pops[p];
    const uint64_t* rows = P.rows[P.st->cur];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    // tile (ti, tj): of tile row ti, the tile columns from its first row on; tile0: the launch's first
    const uint32_t tile = blockIdx.x / splits, split = blockIdx.x % splits;
    const uint32_t TJ = (n + kTN - 1u) / kTN;
    uint32_t ti = 0, left = tile0 + tile;
    while (left >= TJ - ti * kTM / kTN) {
        left -= TJ - ti * kTM / kTN;
        ++ti;
    }
    const uint32_t tj = ti * kTM / kTN + left;
    const uint32_t quads = P.st->W / 2u;   // 16-byte pieces of a row
    const uint32_t nr = (quads + kRound - 1u) / kRound, r0 = min(nr, split * per), cnt = min(nr, r0 + per) - r0;
    uint8_t* const ring = s_raw + ((1024u - (smem_addr(s_raw) & 1023u)) & 1023u);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&s_tmem)),
                     "r"(kTN)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        for (uint32_t i = 0; i < kRing; ++i) {
            mbar_init(smem_addr(&s_full[i]), kRowWarps);
            mbar_init(smem_addr(&s_free[i]), 1u);
        }
        mbar_init(smem_addr(&s_end), 1u);
        s_fail = s_issued = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;
    // e4m3 x e4m3 -> f32, K-major operands; columns up to the sample's end
    const uint32_t ncol = min(kTN, (n - tj * kTN + 15u) & ~15u);
    const uint32_t idesc = (1u << 4) | ((ncol >> 3) << 17) | ((kTM >> 4) << 24);
    if (warp < kRowWarps) {
        // the thread's rows: warp's first + 4 j + lane / 8, of each the piece lane % 8 of a round
        const uint32_t first = warp * 32u + (lane >> 3), piece = lane & 7u;
        const ulonglong2* const base = reinterpret_cast<const ulonglong2*>(rows) + piece;
        uint32_t at[8];   // row of the population; ~0 past the sample
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) {
            const uint32_t r = first + 4u * j, row = r < kTM ? ti * kTM + r : tj * kTN + (r - kTM);
            at[j] = row < n ? sample[row] : ~0u;
        }
        auto load = [&](uint32_t r, ulonglong2 (&x)[8]) {
            const uint32_t quad = r * kRound;
#pragma unroll
            for (uint32_t j = 0; j < 8; ++j)
                x[j] = at[j] != ~0u && quad + piece < quads ? __ldg(base + (size_t)at[j] * (P.Wcap / 2u) + quad)
                                                            : make_ulonglong2(0, 0);
        };
        ulonglong2 x[8], next[8];
        if (cnt) load(r0, next);
        bool ok = true;
        uint32_t ones[8] = {0, 0, 0, 0, 0, 0, 0, 0};   // the rows' alleles in this lane's slots
        for (uint32_t r = 0; r < cnt && ok; ++r) {
#pragma unroll
            for (uint32_t j = 0; j < 8; ++j) {
                x[j] = next[j];
                ones[j] += (uint32_t)(__popcll(x[j].x) + __popcll(x[j].y));
            }
            if (r + 1u < cnt) load(r0 + r + 1u, next);
#pragma unroll
            for (uint32_t t = 0; t < kRound; ++t) {
                const uint32_t it = r * kRound + t, s = t % kRing;
                if (it >= kRing) ok = wait_parity(smem_addr(&s_free[s]), (it / kRing - 1u) & 1u, &s_fail);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                uint8_t* const dst = ring + s * kStageBytes + first * 128u;
#pragma unroll
                for (uint32_t j = 0; j < 8; ++j) {
                    const uint64_t half = (t & 4u) ? x[j].y : x[j].x;
                    const uint32_t v = (uint32_t)(half >> (32u * ((t >> 1) & 1u))) >> (4u * (t & 1u));
                    const uint4 b = make_uint4(v & 0x01010101u, (v >> 1) & 0x01010101u, (v >> 2) & 0x01010101u,
                                               (v >> 3) & 0x01010101u);
                    if (at[j] != ~0u || it < kRing)   // rows past the sample stay zero
                        *reinterpret_cast<uint4*>(dst + j * 512u + ((piece ^ ((first + 4u * j) & 7u)) << 4)) = b;
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0)
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(&s_full[s])) : "memory");
            }
        }
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) {
            uint32_t v = ones[j];
            v += __shfl_xor_sync(0xffffffffu, v, 1);
            v += __shfl_xor_sync(0xffffffffu, v, 2);
            v += __shfl_xor_sync(0xffffffffu, v, 4);
            if (piece == 0) s_ones[first + 4u * j] = v;
        }
    } else if (lane == 0) {
        uint32_t it = 0;
        for (; it < cnt * kRound; ++it) {
            const uint32_t s = it % kRing;
            if (!wait_parity(smem_addr(&s_full[s]), (it / kRing) & 1u, &s_fail)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t a = smem_addr(ring + s * kStageBytes), b = a + kTM * 128u;
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k)
                mma_f8(tmem, operand(a + 32u * k), operand(b + 32u * k), idesc, (it | k) != 0u);
            mma_commit(smem_addr(&s_free[s]));
        }
        s_issued = it;
        if (it) mma_commit(smem_addr(&s_end));
    }
    __syncthreads();
    bool ok = !s_fail;
    if (s_issued) {   // everything issued has ended, whether the loops ran through or not
        uint32_t never = 0;
        ok = __syncthreads_and(wait_parity(smem_addr(&s_end), 0u, &never)) && ok;
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // TMEM lanes are the tile's rows: a warp reads the 32 of its place in its warpgroup, a third of the columns (the
    // issuing warp none)
    const uint32_t i_tile = (warp & 3u) * 32u + lane, i = ti * kTM + i_tile;
    const uint32_t taddr = tmem + (((warp & 3u) * 32u) << 16), col0 = warp < kRowWarps ? (warp >> 2) * 32u : ncol;
    uint32_t* const sums = tile_sum ? tile_sum + (size_t)tile * kTileSums : nullptr;   // [column][row], then the rows' alleles
    bool finish = ok;
    if (splits > 1u) {
        for (uint32_t c0 = col0; c0 < ncol; c0 += 96u) {
            uint32_t v[32];
            load_32_columns(taddr + c0, v);
            if (ok && cnt)
#pragma unroll
                for (uint32_t k = 0; k < 32; ++k) {
                    const uint32_t x = __float2uint_rn(__uint_as_float(v[k]) * 262144.0f);
                    if (x && c0 + k < ncol) atomicAdd(sums + (c0 + k) * kTM + i_tile, x);
                }
        }
        if (tid < kTM + kTN && s_ones[tid]) atomicAdd(sums + kTM * kTN + tid, s_ones[tid]);
        __threadfence();
        __syncthreads();
        if (tid == 0) s_last = atomicAdd(tile_done + tile, 1u) == splits - 1u;
        __syncthreads();
        finish = ok && s_last;
        __threadfence();
        if (finish && tid < kTM + kTN) s_ones[tid] = __ldcg(sums + kTM * kTN + tid);
        __syncthreads();
    }
    unsigned long long sum = 0, sq = 0, pairs = 0;
    uint32_t mn = 0xffffffffu, mx = 0;
    if (finish) {
        for (uint32_t c0 = col0; c0 < ncol; c0 += 96u) {
            uint32_t v[32];
            if (splits > 1u) {
#pragma unroll
                for (uint32_t k = 0; k < 32; ++k) v[k] = c0 + k < ncol ? __ldcg(sums + (c0 + k) * kTM + i_tile) : 0u;
            } else {
                load_32_columns(taddr + c0, v);
#pragma unroll
                for (uint32_t k = 0; k < 32; ++k)
                    v[k] = cnt ? __float2uint_rn(__uint_as_float(v[k]) * 262144.0f) : 0u;
            }
#pragma unroll
            for (uint32_t k = 0; k < 32; ++k) {
                const uint32_t j = tj * kTN + c0 + k;
                if (i < j && j < n) {
                    const uint32_t d = s_ones[i_tile] + s_ones[kTM + c0 + k] - 2u * v[k];
                    if (dist) dist[(uint64_t)i * n - (uint64_t)i * (i + 1) / 2 + (j - i - 1)] = d;
                    sum += d;
                    sq += (unsigned long long)d * d;
                    pairs += 1;
                    mn = min(mn, d);
                    mx = max(mx, d);
                }
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
        sq += __shfl_xor_sync(0xffffffffu, sq, o);
        pairs += __shfl_xor_sync(0xffffffffu, pairs, o);
    }
    mn = __reduce_min_sync(0xffffffffu, mn);
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0 && warp < kRowWarps) {
        s_sum[warp] = sum;
        s_sq[warp] = sq;
        s_cnt[warp] = pairs;
        s_min[warp] = mn;
        s_max[warp] = mx;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTN) : "memory");
    if (tid == 0) {
        for (uint32_t k = 1; k < kRowWarps; ++k) {
            sum += s_sum[k];
            sq += s_sq[k];
            pairs += s_cnt[k];
            mn = min(mn, s_min[k]);
            mx = max(mx, s_max[k]);
        }
        if (!ok) atomicOr(&out->err, 1u);
        if (pairs) {
            atomicAdd(&out->count, pairs);
            atomicAdd(&out->total, sum);
            atomicAdd(&out->sumsq, sq);
            atomicMin(&out->min, mn);
            atomicMax(&out->max, mx);
        }
    }
}

PairwisePlan pairwise_plan(const LaunchCfg& L, uint32_t n, uint32_t W) {
    PairwisePlan z{};
    const uint32_t TI = (n + kTM - 1u) / kTM, TJ = (n + kTN - 1u) / kTN, nr = (W / 2u + kRound - 1u) / kRound;
    for (uint32_t ti = 0; ti < TI; ++ti) z.tiles += TJ - ti * kTM / kTN;
    // Slots over several CTAs where the tiles alone leave SMs idle: the count with the least work on the busiest SM
    // (tiles x splits over the SMs, each with its share of the rounds plus about six stages' time to start and
    // to add up), and as many as keep a CTA's sums in range.  Above kSplitTiles tiles the counts would take more
    // memory (133 KB a tile, 8.7 GB for 65,536 rows) than the last wave's idle SMs are worth: one CTA a tile, or, where
    // the sums' range asks for more, a launch for every kSplitTiles of them.
    const uint32_t least = std::max(1u, (nr * kRound * 128u + kMaxSlots - 1u) / kMaxSlots);
    const bool many = z.tiles > kSplitTiles;
    z.group = many && least > 1u ? kSplitTiles : z.tiles;
    double best = 1e30;
    z.splits = least;
    for (uint32_t s = least; s <= std::max(least, many && least == 1u ? 1u : std::min(nr, 64u)); ++s) {
        const double waves = (double)((z.group * (uint64_t)s + L.num_sms - 1u) / L.num_sms);
        const double cost = waves * ((double)((nr + s - 1u) / s * kRound) + 6.0 + (s > 1u ? 6.0 : 0.0));
        if (cost < best * 0.98) {
            best = cost;
            z.splits = s;
        }
    }
    z.per = (nr + z.splits - 1u) / z.splits;
    z.sum_bytes = z.splits > 1u ? (size_t)z.group * (kTileSums + 1u) * 4 : 0;
    return z;
}

// scratch: sum_bytes.
cudaError_t launch_pairwise(const LaunchCfg& L, const PopDev* pops, uint32_t p, const uint32_t* sample, uint32_t n,
                            const PairwisePlan& z, void* scratch, uint32_t* dist, PairwiseOut* out) {
    uint32_t* sums = z.sum_bytes ? static_cast<uint32_t*>(scratch) : nullptr;
    uint32_t* done = z.sum_bytes ? sums + (size_t)z.group * kTileSums : nullptr;
    const size_t smem = kRing * kStageBytes + 1024u;
    // a property of the function on the current device; setting it again is harmless
    cudaError_t e =
        cudaFuncSetAttribute((const void*)k_pairwise, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    for (uint32_t t = 0; t < z.tiles && e == cudaSuccess; t += z.group) {
        if (sums) e = cudaMemsetAsync(sums, 0, z.sum_bytes, L.stream);
        if (e != cudaSuccess) break;
        k_pairwise<<<std::min(z.group, z.tiles - t) * z.splits, kPairThreads, smem, L.stream>>>(
            pops, p, sample, n, t, z.splits, z.per, sums, done, dist, out);
        e = cudaPeekAtLastError();
    }
    return e;
}

}  // namespace clotho
