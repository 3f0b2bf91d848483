// k_step.cu -- the kernels after the generation pass (individual phenotypes, fitness and
// its FP64 prefix sum), the staged API's own stages, seeding and column statistics.
//
// All kernels walk every population of the batch; sizes are read from the
// device status words so a step needs no host synchronisation and can be
// captured in a CUDA graph.
#include "step.cuh"

#include <algorithm>

namespace clotho {

namespace {
constexpr uint32_t kScanChunk = 4096;  // individuals a chunk of the fitness sum: 32 warps of 128

__device__ inline double warp_incl_f64(double x) {
    const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        double y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    return x;
}
}  // namespace

// ---------------------------------------------------------------------------
// Step begin (staged API): the child becomes the parent (engine_batched_task.hpp:164), the
// offspring count comes from the header, and the item prefix of the generation kernel is
// rebuilt.
__global__ void k_begin(const PopDev* __restrict__ pops, uint32_t npops, const uint32_t* __restrict__ hdr,
                        WorkCtl* ctl) {
    const uint32_t p = threadIdx.x;
    begin_items(pops, npops, hdr, ctl);
    if (p < npops) {
        const PopDev& P = pops[p];
        DevStatus* st = P.st;
        uint32_t N = hdr[2 * p], M = hdr[2 * p + 1];
        if (N > P.Ncap) { st->err |= kErrAlleles; N = P.Ncap; }
        if (M > P.Mcap) { st->err |= kErrMut; M = P.Mcap; }
        st->pN = st->N;
        st->pA = st->A;
        st->pW = st->W;
        st->N = N;
        st->M = M;
        st->ev_used = 0;
        st->cur ^= 1u;
    }
}

void launch_begin(const LaunchCfg& L, const PopDev* pops, uint32_t npops, const uint32_t* hdr, WorkCtl* ctl) {
    k_begin<<<1, kMaxPops, 0, L.stream>>>(pops, npops, hdr, ctl);
}

__global__ void k_end(const PopDev* __restrict__ pops, uint32_t npops) {
    const uint32_t p = threadIdx.x;
    if (p < npops) {
        DevStatus* st = pops[p].st;
        st->last_M = st->M;
        st->gen += 1u;  // ++m_generation (engine_batched_task.hpp:222)
    }
}
void launch_end(const LaunchCfg& L, const PopDev* pops, uint32_t npops) {
    k_end<<<1, kMaxPops, 0, L.stream>>>(pops, npops);
}

// ---------------------------------------------------------------------------
// The new alleles of a staged generation, one thread per allele and trait.
__global__ void k_mut_resolve(const PopDev* __restrict__ pops, uint32_t npops) {
    for (uint32_t p = blockIdx.z; p < npops; p += gridDim.z) {
        const PopDev& P = pops[p];
        DevStatus* st = P.st;
        const uint64_t M = st->M, T = P.T;
        int nz_delta = 0;
        for (uint64_t q = blockIdx.x * blockDim.x + threadIdx.x; q < M * T; q += gridDim.x * blockDim.x)
            nz_delta += resolve_mutation(P, (uint32_t)(q / T), (uint32_t)(q % T), st->gen, st->free_cnt, st->pA, st->A);
        if (nz_delta) atomicAdd(&st->nz_eff, nz_delta);
    }
}
void launch_mut_resolve(const LaunchCfg& L, const PopDev* pops, uint32_t npops) {
    k_mut_resolve<<<pop_grid(npops, L.num_sms * 2u, L.num_sms, 2), 256, 0, L.stream>>>(pops, npops);
}

// Standalone mutation scatter (staged API): child->mutate(seq, slot) is a
// single-bit XOR (population_space_row_block.hpp:111-125).
__global__ void k_mut_scatter(const PopDev* __restrict__ pops, uint32_t npops) {
    for (uint32_t p = blockIdx.z; p < npops; p += gridDim.z) {
        const PopDev& P = pops[p];
        const DevStatus* st = P.st;
        const uint32_t M = st->M, S = 2u * st->N;
        uint64_t* rows = P.rows[st->cur];
        for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < M; i += gridDim.x * blockDim.x) {
            const uint32_t slot = P.mut_slot[i], s = P.mut_seq[i];
            if (slot == 0xffffffffu || s >= S) continue;
            atomicXor((unsigned long long*)&rows[(size_t)s * P.Wcap + (slot >> 6)], 1ull << (slot & 63u));
        }
    }
}
void launch_mut_scatter(const LaunchCfg& L, const PopDev* pops, uint32_t npops) {
    k_mut_scatter<<<pop_grid(npops, L.num_sms * 2u, L.num_sms, 2), 256, 0, L.stream>>>(pops, npops);
}

// ---------------------------------------------------------------------------
// Individual phenotype = genome 0 + genome 1 (individual_reducer_task_population_space_row.hpp:51-79),
// or the constant 1.0 when every trait weight is zero (engine_batched_task.hpp:207-211);
// then the fitness metric (GeneralFitness::operator(), general_fitness.hpp:101-119) and the first level of its
// prefix sum: four individuals a lane, 128 a warp.
//
// Bound by the FP64 pipe (about two operations a clock and SM): the exponential and the sum's adds.  So every
// warp of the GPU takes 128 individuals, and what is the same for all of them (the root, the quotients) is
// computed once a block.
//
// CONSTANT (no population of the launch has a metric): every fitness is 1, so the prefix sum of individual i is i + 1
// in any order of additions; it is written here and the step ends here, without k_cdf.
__device__ __forceinline__ void end_step(const StepEnd& end, uint32_t pop, DevStatus* st) {
    if (end.mode == StepEnd::kNone) return;
    st->last_M = st->M;
    st->gen += 1u;  // ++m_generation (engine_batched_task.hpp:222)
    if (end.mode == StepEnd::kSchedule) {
        const uint32_t* next = end.ctl->sched + (size_t)end.ctl->sched_at * 2u * end.npops + 2u * pop;
        end.hdr[2u * pop] = next[0];
        end.hdr[2u * pop + 1u] = next[1];
    }
}

template <bool ONE, bool CONSTANT>
__global__ void __launch_bounds__(256) k_individuals(const __grid_constant__ PopDev one,
                                                     const PopDev* __restrict__ pops,
                                                     const BlockPart* __restrict__ map, const StepEnd end) {
    __shared__ double s_k[4];
    __shared__ double s_f[8][128];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const BlockPart part = block_part<ONE>(map);
    const PopDev& P = ONE ? one : pops[part.pop];
    pdl_wait();
    DevStatus* st = P.st;
    const uint32_t N = st->N, T = P.T;
    const uint32_t nw = (N + kScanChunk - 1u) / kScanChunk * 32u;  // whole chunks: empty warps sum to zero
    if (part.i >= nw && part.i) return;
    const bool neutral = st->nz_eff == 0;
    const int fitness = P.fitness;
    __syncthreads();
    if (threadIdx.x == 0) {
        if (part.i == 0) {
            st->all_neutral = neutral ? 1u : 0u;
            st->fit_const = 1u;  // k_cdf clears it
            if (CONSTANT) {
                st->fit_total = (double)N;
                end_step(end, part.pop, st);
            }
        }
        if (fitness == 1 || fitness == 2) {
            const double sig = sqrt(4.0 * (double)N * P.mu);  // normal/quadratic generators
            s_k[0] = (1.0 / sig) * 0.398942280401432677939946059934;
            s_k[1] = 2.0 * sig * sig;
            s_k[2] = P.fit_param * sig;
        }
    }
    __syncthreads();
    const double* zg = P.zg[st->cur];
    // neighbouring units in different blocks: as even a share of the FP64 pipes as there are units
    for (uint32_t w = warp * part.n + part.i; w < nw; w += part.n * 8u) {
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
            const uint32_t i = w * 128u + 32u * k + lane;
            double f = 0.0;
            if (i < N) {
                const double2* a = reinterpret_cast<const double2*>(zg + (size_t)i * 8u);  // genomes 2i, 2i + 1
                double z[4] = {1.0, 1.0, 1.0, 1.0};
                if (!neutral) {
                    const double2 a0 = a[0], b0 = a[2];
                    z[0] = a0.x + b0.x;
                    if (T > 1) z[1] = a0.y + b0.y;
                    if (T > 2) {
                        const double2 a1 = a[1], b1 = a[3];
                        z[2] = a1.x + b1.x;
                        z[3] = a1.y + b1.y;
                    }
                }
                for (uint32_t t = 1; t < 4; ++t)
                    if (t >= T) z[t] = 0.0;
                double2* zi = reinterpret_cast<double2*>(P.zi + (size_t)i * 4u);
                zi[0] = make_double2(z[0], z[1]);
                zi[1] = make_double2(z[2], z[3]);
                f = 1.0;
                const double z0 = z[0];
                if (!CONSTANT) switch (fitness) {
                    case 1:  // gaussian (normal_fitness_metric.cpp:25-31)
                        f = s_k[0] * exp(-(z0 * z0) / s_k[1]);
                        break;
                    case 2: {  // quadratic (quadratic_fitness_metric.cpp:23-28)
                        double r = z0 / s_k[2];
                        r *= r;
                        f = (r >= 1.0) ? 0.0 : 1.0 - r;
                    } break;
                    case 3: {  // gaussian_vs
                        const double ss = z[0] * z[0] + z[1] * z[1] + z[2] * z[2] + z[3] * z[3];
                        f = exp(-ss / (2.0 * P.fit_param));
                    } break;
                    default: f = 1.0;
                }
                P.fit[i] = f;
                if (CONSTANT) P.cdf[i] = (double)(i + 1u);
            }
            s_f[warp][32u * k + lane] = f;
        }
        if (CONSTANT) continue;
        __syncwarp();
        const double* v = &s_f[warp][4u * lane];
        const double s = warp_incl_f64(((v[0] + v[1]) + v[2]) + v[3]);
        if (lane == 31u) P.scan_wsum[w] = s;
        __syncwarp();
    }
}

// Deterministic FP64 inclusive prefix sum of fitness with a fixed association order (four individuals a lane,
// a shuffle scan over the warp, the 32 warps of a chunk and the chunks one after another), the total and the
// all-equal check; then the step's end.
constexpr uint32_t kInlineChunks = 64;   // up to here a block adds up the chunks before its own by itself

__device__ __forceinline__ double chunk_total(const double* wsum, uint32_t c) {
    double t = 0.0;
#pragma unroll 8
    for (uint32_t i = 0; i < 32u; ++i) t += wsum[32u * c + i];
    return t;
}

// Chunk offsets of populations of more than kInlineChunks chunks.
__global__ void __launch_bounds__(256) k_cdf_offsets(const PopDev* __restrict__ pops) {
    __shared__ double s_t[256];
    __shared__ double s_acc;
    const PopDev& P = pops[blockIdx.x];
    pdl_wait();
    const uint32_t nch = (P.st->N + kScanChunk - 1u) / kScanChunk;
    if (nch <= kInlineChunks) return;
    if (threadIdx.x == 0) s_acc = 0.0;
    for (uint32_t c0 = 0; c0 < nch; c0 += 256u) {
        __syncthreads();
        if (c0 + threadIdx.x < nch) s_t[threadIdx.x] = chunk_total(P.scan_wsum, c0 + threadIdx.x);
        __syncthreads();
        if (threadIdx.x == 0) {
            double acc = s_acc;
            for (uint32_t j = 0; j < min(256u, nch - c0); ++j) {
                const double t = s_t[j];
                s_t[j] = acc;
                acc += t;
            }
            s_acc = acc;
        }
        __syncthreads();
        if (c0 + threadIdx.x < nch) P.scan_part[c0 + threadIdx.x] = s_t[threadIdx.x];
    }
}

// A unit is 8 warps of 128 individuals: a quarter of a chunk.
template <bool ONE>
__global__ void __launch_bounds__(256) k_cdf(const __grid_constant__ PopDev one, const PopDev* __restrict__ pops,
                                             const BlockPart* __restrict__ map, const StepEnd end) {
    __shared__ double s_tot[kInlineChunks];
    __shared__ double s_woff[32];
    __shared__ double s_part, s_last;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const BlockPart part = block_part<ONE>(map);
    const PopDev& P = ONE ? one : pops[part.pop];
    pdl_wait();
    DevStatus* st = P.st;
    const uint32_t N = st->N;
    const uint32_t nch = (N + kScanChunk - 1u) / kScanChunk;
    if (part.i == 0 && threadIdx.x == 0) {
        end_step(end, part.pop, st);
        if (N == 0) st->fit_total = 0.0;
    }
    const double f0 = N ? P.fit[0] : 0.0;
    for (uint32_t u = part.i; u < nch * 4u; u += part.n) {
        const uint32_t c = u >> 2, w = u * 8u + warp;
        const bool last = u == nch * 4u - 1u;
        const uint32_t b = w * 128u + lane * 4u;
        double v[4], s = 0.0;
        bool same = true;
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
            v[k] = (b + k < N) ? P.fit[b + k] : 0.0;
            if (b + k < N && v[k] != f0) same = false;
            s += v[k];
        }
        if (!__all_sync(0xffffffffu, same) && lane == 0u) atomicAnd(&st->fit_const, 0u);
        __syncthreads();  // the previous unit's offsets are read
        if (nch <= kInlineChunks) {
            if (threadIdx.x < c) s_tot[threadIdx.x] = chunk_total(P.scan_wsum, threadIdx.x);
            __syncthreads();
        }
        if (threadIdx.x == 0) {
            double acc = 0.0;
            if (nch <= kInlineChunks)
                for (uint32_t j = 0; j < c; ++j) acc += s_tot[j];
            else
                acc = P.scan_part[c];
            s_part = acc;
        }
        if (warp == 1u) {  // offsets of the chunk's warps: lane i adds the i before it one after another
            const double ws = P.scan_wsum[32u * c + lane];
            double acc = 0.0;
            for (uint32_t j = 0; j < 31u; ++j) {
                const double x = __shfl_sync(0xffffffffu, ws, j);
                if (j < lane) acc += x;
            }
            s_woff[lane] = acc;
            if (lane == 31u) s_last = acc + ws;  // the chunk's total
        }
        const double incl = warp_incl_f64(s);
        __syncthreads();
        // exclusive prefix inside the warp = inclusive value of the previous lane
        const double prev = __shfl_up_sync(0xffffffffu, incl, 1);
        const double excl_w = lane ? prev : 0.0;
        double r = s_part + (s_woff[w & 31u] + excl_w);
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
            r += v[k];
            if (b + k < N) P.cdf[b + k] = r;
        }
        if (last && threadIdx.x == 0) {
            const double total = s_part + s_last;
            st->fit_total = total;
            if (!(total > 0.0)) atomicOr(&st->err, kErrFitness);
        }
    }
}
uint32_t launch_fitness(const LaunchCfg& L, const PopDev* pops, uint32_t npops, uint32_t maxN, bool constant, StepEnd end) {
    const uint32_t units = std::max(1u, (maxN + kScanChunk - 1u) / kScanChunk * 4u);
    // Few individuals: a warp of 128 to an SM (blocks of which one warp works) before a second one, for the FP64 pipe.
    // Eight to a block left most of the pipes idle: 10,000 individuals 11.9 -> 9.4 us, 50,000 14.3 -> 11.6.
    const uint32_t warps = std::max(1u, (maxN + 127u) / 128u);
    const uint32_t ind = std::max(blocks_of(L, units, L.ind_per_sm), std::min(warps, (uint32_t)L.num_sms));
    if (constant) {
        launch_pops(L, kTable256, k_individuals<true, true>, k_individuals<false, true>, ind, pops, npops, end);
        return 1u;
    }
    launch_pops(L, kTable256, k_individuals<true, false>, k_individuals<false, false>, ind, pops, npops, StepEnd{});
    const bool offsets = maxN > kInlineChunks * kScanChunk;
    if (offsets) launch_k(L, k_cdf_offsets, dim3(npops), dim3(256), pops);
    launch_pops(L, kTable256, k_cdf<true>, k_cdf<false>, blocks_of(L, units, 8), pops, npops, end);
    return offsets ? 3u : 2u;
}

// ---------------------------------------------------------------------------
// Pre-seeded rows: bit (row, slot) iff seed_hash(seed,row,slot) < thr[slot].
__global__ void k_seed_rows(const PopDev* __restrict__ pops, uint32_t p, const uint32_t* __restrict__ thr,
                            uint64_t seed, uint32_t A) {
    const PopDev& P = pops[p];
    const DevStatus* st = P.st;
    const uint32_t S = 2u * st->N, W = st->W;
    uint64_t* rows = P.rows[st->cur];
    const size_t total = (size_t)S * W;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const uint32_t r = (uint32_t)(i / W), w = (uint32_t)(i % W);
        uint64_t x = 0;
        for (uint32_t j = 0; j < 64; ++j) {
            const uint32_t a = w * 64u + j;
            if (a < A && seed_hash(seed, r, a) < thr[a]) x |= 1ull << j;
        }
        rows[(size_t)r * P.Wcap + w] = x;
    }
}
void launch_seed_rows(const LaunchCfg& L, const PopDev* pops, uint32_t p, const uint32_t* thr, uint64_t seed,
                      uint32_t A) {
    k_seed_rows<<<L.num_sms * 8, 256, 0, L.stream>>>(pops, p, thr, seed, A);
}

// ---------------------------------------------------------------------------
// Margins of the current child rows in one pass: carriers per allele slot (count_alleles,
// cuda/analysis/allele_frequency_kernels.hpp:20-73) and alleles per sequence (the column and row margins of
// population_space_row_frequency_evaluator.hpp:37-62).
//
// Bound by the one read of the rows.  A lane holds two words (one 16-byte load a row) and counts their 128
// columns bit-sliced: eight rows are loaded together and added through a tree of carry-save adders, about 12
// logic operations a row and lane, into eight planes of binary digits (at most kMarginRows rows a lane).  The
// planes are transposed to bytes once per block and summed over its warps in shared memory, so a column costs one
// global addition per block.  Rows narrower than a warp's 64 words share it: lpr lanes a row, 32 / lpr rows a load.
// A warp's next eight rows are prefetched into L2, one instruction for each, while it counts these: both margins of
// 2e5 rows of 912 words 388 -> 356 us a call, the columns alone 350 -> 296 (two or three rounds ahead 368, 406; the
// registers hold three blocks an SM: two 399, four spill, 407).
// (One thread a column, a bit a step: 10.07 ms for 2e5 rows of 2,288 words, where the one read takes 0.54 ms at
// the copy rate.)
constexpr uint32_t kMarginRows = 248;   // rows a lane adds up (eight binary digits hold 255)

__device__ __forceinline__ void csa(uint64_t& h, uint64_t& l, uint64_t a, uint64_t b, uint64_t c) {
    h = (a & b) | (a & c) | (b & c);
    l = a ^ b ^ c;
}

// One column group's planes of a lane: digit i of the counts of the 64 columns of one word.
struct Planes {
    uint64_t d[8];
    __device__ __forceinline__ void add8(const uint64_t (&x)[8]) {
        uint64_t a, b, fa, fb, c;
        csa(a, d[0], d[0], x[0], x[1]);
        csa(b, d[0], d[0], x[2], x[3]);
        csa(fa, d[1], d[1], a, b);
        csa(a, d[0], d[0], x[4], x[5]);
        csa(b, d[0], d[0], x[6], x[7]);
        csa(fb, d[1], d[1], a, b);
        csa(c, d[2], d[2], fa, fb);
#pragma unroll
        for (int i = 3; i < 8; ++i) {
            const uint64_t t = d[i] & c;
            d[i] ^= c;
            c = t;
        }
    }
    // cnt[j * 65] += count of column j.  The lanes of one word (rows that share a warp) go through its columns eight
    // apart: side by side they would add to the same counts.
    __device__ __forceinline__ void flush(uint32_t* cnt, uint32_t sub) const {
#pragma unroll 1
        for (uint32_t k0 = 0; k0 < 8; ++k0) {
            const uint32_t k = (k0 + sub) & 7u;
            uint64_t x = 0;  // byte i: digit i of columns 8k .. 8k + 7
#pragma unroll
            for (int i = 0; i < 8; ++i) x |= ((d[i] >> (8u * k)) & 0xffull) << (8 * i);
            uint64_t t = (x ^ (x >> 7)) & 0x00AA00AA00AA00AAull;  // 8 x 8 bit transpose: byte j = column 8k + j
            x ^= t ^ (t << 7);
            t = (x ^ (x >> 14)) & 0x0000CCCC0000CCCCull;
            x ^= t ^ (t << 14);
            t = (x ^ (x >> 28)) & 0x00000000F0F0F0F0ull;
            x ^= t ^ (t << 28);
#pragma unroll
            for (uint32_t j = 0; j < 8; ++j) {
                const uint32_t c = (uint32_t)(x >> (8u * j)) & 0xffu;
                if (c) atomicAdd(cnt + (8u * k + j) * 65u, c);
            }
        }
    }
};

template <bool COL, bool ROW>
__global__ void __launch_bounds__(256, 3) k_margins(const PopDev* __restrict__ pops, uint32_t p,
                                                 uint32_t* __restrict__ colc, uint32_t* __restrict__ rowc,
                                                 uint32_t lpr, uint32_t strip, uint32_t groups) {
    __shared__ uint32_t s_cnt[COL ? 64 * 65 : 1];   // [column of the word][word]
    const PopDev& P = pops[p];
    const DevStatus* st = P.st;
    const uint32_t S = 2u * st->N, W = st->W;
    const uint64_t* rows = P.rows[st->cur];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t rpl = 32u / lpr, sub = lane / lpr;       // rows a load, this lane's row among them
    // a block's 64-word group and strip of rows: in one grid dimension, which takes more strips than the others'
    // 65,535 (130 million rows)
    const uint32_t g = blockIdx.x % groups, wi = 2u * (lane & (lpr - 1u)), w = g * 64u + wi;
    const uint32_t r0 = blockIdx.x / groups * strip, r1 = min(S, r0 + strip);
    if (COL) {
        for (uint32_t i = threadIdx.x; i < 64u * 65u; i += 256u) s_cnt[i] = 0u;
        __syncthreads();
    }
    Planes c0{}, c1{};
    for (uint32_t b = r0 + warp * 8u * rpl; b < r1; b += 64u * rpl) {
        uint64_t x[8], y[8];
        if (lpr == 32u && lane < 8u) {   // the warp's next eight rows
            const uint32_t r = b + 64u + lane, w0 = g * 64u;
            if (r < r1)
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(rows + (size_t)r * P.Wcap + w0),
                             "r"(min(64u, W - w0) * 8u)
                             : "memory");
        }
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
            const uint32_t r = b + k * rpl + sub;
            const ulonglong2 v = (r < r1 && w < W)
                                     ? __ldg(reinterpret_cast<const ulonglong2*>(rows + (size_t)r * P.Wcap + w))
                                     : make_ulonglong2(0, 0);
            x[k] = v.x;
            y[k] = v.y;
        }
        if (COL) {
            c0.add8(x);
            c1.add8(y);
        }
        if (ROW) {
            // two rows' counts (at most 4,096 each) share a word; lane j < 4 of a row's lanes keeps rows 2j, 2j + 1
            uint32_t mine = 0;
            const uint32_t j = lane & (lpr - 1u);
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) {
                uint32_t n = (uint32_t)(__popcll(x[2 * k]) + __popcll(y[2 * k])) |
                             (uint32_t)(__popcll(x[2 * k + 1]) + __popcll(y[2 * k + 1])) << 16;
                if (lpr == 32u) n = __reduce_add_sync(0xffffffffu, n);
                else
                    for (uint32_t o = lpr >> 1; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
                if (j == k) mine = n;
            }
            if (j < 4u) {
#pragma unroll
                for (uint32_t k = 0; k < 2; ++k) {
                    const uint32_t r = b + (2u * j + k) * rpl + sub, n = (mine >> (16u * k)) & 0xffffu;
                    if (r < r1) {
                        if (groups == 1u) rowc[r] = n;
                        else if (n) atomicAdd(rowc + r, n);
                    }
                }
            }
        }
    }
    if (COL) {
        if (w < W && r0 + warp * 8u * rpl < r1) {   // (warps that had rows)
            c0.flush(s_cnt + wi, sub);
            c1.flush(s_cnt + wi + 1u, sub);
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < 4096u; i += 256u) {
            const uint32_t j = i & 63u, ww = i >> 6;
            const uint32_t c = s_cnt[j * 65u + ww];
            if (c) atomicAdd(colc + (size_t)g * 4096u + i, c);
        }
    }
}
// colc (W * 64 counts) and rowc (S counts), either null, both zero on entry; S and W are the current child's.
void launch_margins(const LaunchCfg& L, const PopDev* pops, uint32_t p, uint32_t S, uint32_t W, uint32_t* colc,
                    uint32_t* rowc) {
    if (S == 0 || W == 0 || (!colc && !rowc)) return;
    uint32_t lpr = 4;  // a row is at least 8 words
    while (lpr < 32u && 2u * lpr < W) lpr <<= 1;
    const uint32_t rpl = 32u / lpr, unit = 64u * rpl;       // rows that a block's warps load together
    const uint32_t groups = (W + 63u) / 64u;
    // about four blocks an SM: three are resident (their loads in flight cover the DRAM latency), the rest
    // even out the end; narrow populations take fewer rows a block
    const uint32_t want = std::max(1u, (uint32_t)L.num_sms * 4u / groups);
    uint32_t strip = (blocks_for(S, want) + unit - 1u) / unit * unit;
    strip = std::min(strip, kMarginRows * 8u * rpl);
    const uint32_t grid = groups * blocks_for(S, strip);
    if (colc && rowc) k_margins<true, true><<<grid, 256, 0, L.stream>>>(pops, p, colc, rowc, lpr, strip, groups);
    else if (colc) k_margins<true, false><<<grid, 256, 0, L.stream>>>(pops, p, colc, nullptr, lpr, strip, groups);
    else k_margins<false, true><<<grid, 256, 0, L.stream>>>(pops, p, nullptr, rowc, lpr, strip, groups);
}


// ---------------------------------------------------------------------------
// Summary statistics from the column counts and the individual phenotypes: segregating and fixed sites, the
// spectrum, and per block the sums of 2 f (1 - f) and of each trait (fixed order in a block; the host adds the
// blocks in order, so the sums do not depend on timing).  FP64 adds and quotients, spread over the GPU; on the
// host these were 4 N dependent adds behind a copy of the phenotypes (0.6 ms of a 1.0 ms call at N = 1e5).
constexpr uint32_t kStatBins = 2048;   // spectrum bins counted in shared memory

__global__ void __launch_bounds__(256) k_stats(const PopDev* __restrict__ pops, uint32_t p,
                                               const uint32_t* __restrict__ counts, uint32_t sfs_len,
                                               StatsOut* __restrict__ out, uint32_t* __restrict__ sfs) {
    __shared__ uint32_t s_bin[kStatBins];
    __shared__ double s_sum[8][5];
    const uint32_t bins = min(sfs_len, kStatBins);
    for (uint32_t i = threadIdx.x; i < bins; i += 256u) s_bin[i] = 0u;
    pdl_wait();
    const PopDev& P = pops[p];
    const DevStatus* st = P.st;
    const uint32_t A = st->A, N = st->N, S = 2u * N;
    __syncthreads();
    double v[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    uint32_t seg = 0, fix = 0;
    for (uint32_t a = blockIdx.x * 256u + threadIdx.x; a < A; a += gridDim.x * 256u) {
        const uint32_t c = counts[a];
        seg += (c > 0u && c < S) ? 1u : 0u;
        fix += (S && c == S) ? 1u : 0u;
        if (S && c) {
            const double f = (double)c / (double)S;
            v[4] += 2.0 * f * (1.0 - f);
        }
        if (sfs_len) {
            const uint32_t b = min(c, sfs_len - 1u);
            if (b < kStatBins) atomicAdd(&s_bin[b], 1u);
            else atomicAdd(sfs + b, 1u);
        }
    }
    for (uint32_t i = blockIdx.x * 256u + threadIdx.x; i < N; i += gridDim.x * 256u) {
        const double2* z = reinterpret_cast<const double2*>(P.zi + (size_t)i * 4u);
        const double2 a = z[0], b = z[1];
        v[0] += a.x;
        v[1] += a.y;
        v[2] += b.x;
        v[3] += b.y;
    }
    seg = __reduce_add_sync(0xffffffffu, seg);
    fix = __reduce_add_sync(0xffffffffu, fix);
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (lane == 0) {
        if (seg) atomicAdd(&out->segregating, seg);
        if (fix) atomicAdd(&out->fixed_now, fix);
    }
#pragma unroll
    for (uint32_t t = 0; t < 5; ++t) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[t] += __shfl_xor_sync(0xffffffffu, v[t], o);
        if (lane == 0) s_sum[warp][t] = v[t];
    }
    __syncthreads();
    if (threadIdx.x < 5u) {
        double x = 0.0;
        for (uint32_t i = 0; i < 8; ++i) x += s_sum[i][threadIdx.x];
        out->part[blockIdx.x][threadIdx.x] = x;
    }
    for (uint32_t i = threadIdx.x; i < bins; i += 256u)
        if (s_bin[i]) atomicAdd(sfs + i, s_bin[i]);
}
void launch_stats(const LaunchCfg& L, const PopDev* pops, uint32_t p, const uint32_t* counts, uint32_t sfs_len,
                  StatsOut* out, uint32_t* sfs) {
    launch_k(L, k_stats, dim3(kStatBlocks), dim3(256), pops, p, counts, sfs_len, out, sfs);
}

}  // namespace clotho
