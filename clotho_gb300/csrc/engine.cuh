// engine.cuh -- device data layout and shared device helpers of the GB300
// engine for Clotho's per-generation hot path.
//
// One PopDev describes one resident population.  Every kernel takes an array
// of PopDev and walks all of them, so the plain engine is a batch of one and
// the batched/served forms reuse the same launches.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace clotho {

constexpr uint32_t kMaxTraits = 4;
#ifndef CLOTHO_GEN_THREADS
#define CLOTHO_GEN_THREADS 512
#endif
constexpr uint32_t kGenThreads = CLOTHO_GEN_THREADS;  // one CTA per SM in the generation kernel
constexpr uint32_t kRowsPerItem = 512;     // default child rows per scheduling item (tunable)
constexpr uint32_t kMaxEvReg = 16;         // events held in registers
constexpr uint32_t kMaxEvDevice = 128;     // device-drawn events per gamete
constexpr uint32_t kMaxMutReg = 32;        // mutations per row held in registers
constexpr uint32_t kWordAlign = 64;        // row stride granularity (words)
constexpr uint32_t kSufMaxSlots = 65536;   // allele capacity up to which suffix-table masks are built in per-warp bitmaps
#ifndef CLOTHO_TABLE_MAX_SLOTS
#define CLOTHO_TABLE_MAX_SLOTS (1u << 19)
#endif
// allele capacity up to which a population has a suffix table (above kSufMaxSlots its masks are XORed chunk
// by chunk); at least kSufMaxSlots
constexpr uint32_t kTableMaxSlots = CLOTHO_TABLE_MAX_SLOTS;

// sticky device error bits (CLOTHO_DEVERR_* in clotho_gpu.h)
constexpr uint32_t kErrAlleles = 1u, kErrFixed = 2u, kErrEvents = 4u, kErrParent = 8u,
                   kErrSeq = 16u, kErrMut = 32u, kErrFitness = 64u, kErrStall = 128u, kErrAbandon = 256u;

enum Mode : uint32_t { kModeTape = 0, kModePhilox = 1 };

// Philox counter streams
enum Stream : uint32_t {
    kStreamGamete = 1, kStreamSelect = 2, kStreamMutCount = 3, kStreamMutAllele = 4
};

struct DevStatus {
    uint32_t gen;          // generation number of the step in progress / next step
    uint32_t cur;          // rows buffer holding the current child
    uint32_t N, A, W;      // current child: individuals, alleles, reference width
    uint32_t pN, pA, pW;   // parent of the step in progress
    uint32_t M;            // mutations of the step in progress
    uint32_t fixed_cnt, lost_cnt, free_cnt;
    uint32_t fixed_total;
    int32_t  nz_eff;       // nonzero effect entries in eff[0, A*T)
    uint32_t fs_valid;     // accF/accV hold AND/OR over the current child rows
    uint32_t err;
    uint32_t fit_const;    // every fitness value equal (selection is uniform)
    uint32_t all_neutral;  // phenotype took the constant path
    uint32_t last_M;
    uint32_t ev_used;      // crossover-plan event entries allocated in the step in progress
    uint32_t count_cols;   // the host asked for per-column counts of every fused step's child rows
    uint32_t cols_valid;   // colcnt holds the column counts of the current child rows
    double   fit_total;    // sum of fitness of the current population
    double   fixsum[4];    // effect sums of the alleles fixed in this step's parent
};

struct PopDev {
    uint64_t* rows[2];     // [Scap * Wcap] each
    uint64_t* fixmask;     // [Wcap] fixed columns of the parent
    uint64_t* accF;        // [Wcap] AND over current child rows
    uint64_t* accV;        // [Wcap] OR over current child rows
    uint32_t* free_list;   // [Acap]
    double*   pos;         // [Acap] allele positions (non-negative: ordered as u64)
    uint32_t* age;         // [Acap]
    float*    eff;         // [Acap * 4] effects, traits padded to 4 (unused traits 0)
    double*   fx_pos;      // [FXcap]
    uint32_t* fx_age;      // [FXcap]
    float*    fx_eff;      // [FXcap * T]
    double*   zg[2];       // [Scap * 4] per-genome trait sums, one array per rows buffer
    double*   zi;          // [Ncap * 4] per-individual phenotypes
    double*   fit;         // [Ncap]
    double*   cdf;         // [Ncap]
    double*   scan_part;   // [Ncap / 4096 + 2] offsets of the fitness sum's 4,096-individual chunks
    double*   scan_wsum;   // [Ncap / 128 + 64] fitness sums of 128 individuals
    double*   pois_mu;     // [kPoisTab + 1] Poisson(mu) CDF F_0 .. F_{kPoisTab-1}, then p_{kPoisTab-1}
    double*   pois_rho;    // [kPoisTab + 1] the same of Poisson(rho)
    uint32_t* scan_upart;  // [max(Scap, NB) / 1024 + 32] chunk sums
    uint32_t* scan_opart;  // [Ncap / 1024 + 32] the row-ordering scan's own chunk sums (it runs beside the others)
    uint32_t* pairs;       // [2 * Ncap]
    uint8_t*  swap;        // [Scap]
    uint32_t* ev_off;      // [Scap + 1]
    double*   ev_pos;      // [EVcap]
    uint32_t* mut_seq;     // [Mcap]
    double*   mut_pos;     // [Mcap]
    float*    mut_eff;     // [Mcap * T]
    uint32_t* mut_slot;    // [Mcap]
    uint32_t* row_cnt;     // [Scap + 1] per-row mutation counts (zero between steps)
    uint32_t* row_off;     // [Scap + 1] exclusive prefix of row_cnt
    uint32_t* row_cur;     // [Scap] scatter cursors of the tape's new alleles
    uint32_t* row_mut;     // [Mcap] mutation indices grouped by row
    uint32_t* bcnt;        // [NB + 1] positions per bucket (zero between steps)
    uint32_t* boff;        // [NB + 1] exclusive prefix of bcnt
    uint32_t* bcur;        // [NB] bucket scatter cursors
    double*   bpos;        // [Acap] positions grouped by bucket
    uint32_t* bslot;       // [Acap] slot of each bpos entry
    uint32_t* rank;        // [Acap] rank of each slot (position, then slot index) among the A slots
    uint32_t* inv;         // [Acap] slot of each rank (Acap <= kTableMaxSlots, else null)
    uint64_t* suf;         // [(Acap/64 + 1) * Wcap] suffix table of the crossover classifier (Acap <= kTableMaxSlots, else null)
    uint4*    plan_row;    // [Scap] crossover plans in processing order: row, top strand, event base, events | flags << 30
    uint32_t* ord_cnt;     // [Ncap] rows per parent individual (zero between steps)
    uint32_t* ord_cur;     // [Ncap] scatter cursors: the exclusive prefix of ord_cnt
    uint32_t* ord_pos;     // [Scap] processing position of each row
    uint32_t* plan_go;     // [EVcap] table row offset per planned event (with suf)
    uint32_t* plan_cr;     // [EVcap] correction ranks per planned event: first | count << 20 (with suf)
    uint2*    plan_mut;    // [Scap] new alleles of the planned row (processing order): CSR offset, count
    double*   plan_z;      // [Scap * 4] phenotype base of the planned row: z(base strand) - sum(fixed)
    uint32_t* colcnt;      // [Acap] per-column counts of the child rows (counting steps)
    DevStatus* st;
    uint32_t Scap, Ncap, Wcap, Acap, Mcap, EVcap, FXcap, T;
    uint32_t NB, pad2;     // position buckets (power of two)
    double mu, rho, bias, p_neutral, eff_mean, eff_sigma, fit_param;
    double exp_neg_rho, exp_neg_mu;   // Poisson inversion seeds, computed on the host
    uint64_t seed;
    int32_t fitness;
    uint32_t flags;
    uint32_t mode;
    uint32_t pad1;
};

// Work control shared by the persistent kernels of one step.
struct WorkCtl {
    uint32_t gen_counter;           // dynamic item counter of k_generation
    uint32_t gen_items;             // total items
    uint32_t rows_per_item;         // scheduling granularity (set by the host)
    uint32_t wait_limit;            // try_wait rounds before a bulk copy is flagged late (0: default)
    uint32_t item_base[257];        // item prefix per population (<= 256 pops)
    uint32_t gen_counter_iv;        // item counter of the interval-classifier pass of a mixed batch
    uint32_t gen_counter_cm;        // item counter of the chunk-mask pass of a mixed batch
    const uint32_t* sched;          // step headers of a size schedule
    uint32_t sched_at;              // steps begun since the host set it
    uint64_t rows_done;             // profiling: rows processed
    uint64_t words_done;            // profiling: words written
    uint64_t phase[16];             // profiling: k_generation phase cycles (kPh*)
};

// Phase counters of the profiling build of k_generation (suffix-table rows):
// SM cycles summed over warps, per kind of row, and the rows of each kind.
enum : uint32_t {
    kPhCopyRows = 0, kPhCopySetup, kPhCopyBody, kPhCopyPheno,
    kPhXoRows, kPhXoSetup, kPhXoMask, kPhXoBody, kPhXoGather, kPhXoPheno,
    kPhLongRows, kPhLongCyc, kPhWarpCyc, kPhWarps, kPhCount
};

constexpr uint32_t kMaxPops = 256;

// ---------------------------------------------------------------------------
// small helpers

__host__ __device__ inline uint32_t ref_width(uint32_t A) {
    // population_space_row::setMaxAlleles (population_space_row_block.hpp:94-101)
    return ((A + 511u) / 512u) * 8u;
}

__device__ inline uint64_t dkey(double d) { return (uint64_t)__double_as_longlong(d); }

// seed rule shared with the oracle (orc_seed_hash)
__host__ __device__ inline uint32_t seed_hash(uint64_t seed, uint32_t row, uint32_t slot) {
    uint64_t x = seed + 0x9E3779B97F4A7C15ull * ((((uint64_t)row) << 32) + (uint64_t)slot + 1ull);
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    x ^= x >> 31;
    return (uint32_t)(x >> 32);
}

// Philox-4x32-10 counter-based generator, written from the published
// description (Salmon, Moraes, Dror, Shaw: "Parallel random numbers: as easy
// as 1, 2, 3", SC'11): multipliers 0xD2511F53/0xCD9E8D57, Weyl key increments
// 0x9E3779B9/0xBB67AE85, ten rounds.
struct U4 { uint32_t x, y, z, w; };

__device__ inline U4 philox4x32(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3, uint64_t key) {
    uint32_t k0 = (uint32_t)key, k1 = (uint32_t)(key >> 32);
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        uint32_t hi0 = __umulhi(0xD2511F53u, c0), lo0 = 0xD2511F53u * c0;
        uint32_t hi1 = __umulhi(0xCD9E8D57u, c2), lo1 = 0xCD9E8D57u * c2;
        uint32_t n0 = hi1 ^ c1 ^ k0, n2 = hi0 ^ c3 ^ k1;
        c0 = n0; c1 = lo1; c2 = n2; c3 = lo0;
        k0 += 0x9E3779B9u; k1 += 0xBB67AE85u;
    }
    return U4{c0, c1, c2, c3};
}

// [0,1) double from 53 random bits: v * 2^-53, assembled as IEEE-754 bits with
// integer operations (exactly the value of the FP64 conversion and scaling, which
// would occupy GB300's narrow FP64 pipe).
__device__ inline double u01(uint32_t hi, uint32_t lo) {
    const uint64_t v = ((((uint64_t)hi) << 32) | lo) >> 11;
    const int msb = 63 - __clzll((long long)(v | 1ull));          // highest set bit, 0..52
    const uint64_t frac = (v << (52 - msb)) & 0x000FFFFFFFFFFFFFull;
    const uint64_t bits = ((uint64_t)(1023 - 53 + msb) << 52) | frac;
    return __longlong_as_double((long long)(v ? bits : 0ull));
}

// x < y for non-negative, non-NaN doubles, as an integer compare of their bit
// patterns (IEEE-754 order); exact, and off the FP64 pipe.
__device__ inline bool lt_nonneg(double x, double y) {
    return (unsigned long long)__double_as_longlong(x) < (unsigned long long)__double_as_longlong(y);
}

// 1/k for the Poisson inversion (k = 1..kRecip-1); multiplying by it avoids
// FP64 divisions, which are slow on this part.  Every translation unit that
// draws Poisson numbers has its own copy (no relocatable device code), filled
// on the current device by that unit's init_recip_* function.
constexpr uint32_t kRecip = 256;
static __constant__ double c_recip[kRecip];
static inline int fill_recip_table() {
    double h[kRecip];
    h[0] = 0.0;
    for (uint32_t k = 1; k < kRecip; ++k) h[k] = 1.0 / (double)k;
    return cudaMemcpyToSymbol(c_recip, h, sizeof(h)) == cudaSuccess ? 0 : -1;
}

// Poisson draw by sequential inversion of the CDF; e = exp(-lambda) from the
// host.  Used only for small means (per-gamete events, per-row mutations).
// One step of the Poisson CDF recurrence p_k = p_{k-1} lambda / k, F_k = F_{k-1} + p_k, with
// explicitly rounded operations (never contracted into FMAs), so every copy of it -- the inversion
// loop and the plan kernel's table -- gives the same bits.
__device__ inline void poisson_step(double& p, double& F, double lambda, uint32_t k) {
    p = __dmul_rn(p, __dmul_rn(lambda, k < kRecip ? c_recip[k] : 1.0 / (double)k));
    F = __dadd_rn(F, p);
}

__device__ inline uint32_t poisson_inv(double u, double lambda, double e) {
    double p = e, F = e;
    uint32_t k = 0;
    while (u > F && k < 4096u) {
        ++k;
        poisson_step(p, F, lambda, k);
    }
    return k;
}

constexpr uint32_t kPoisTab = 64;     // entries of a population's Poisson CDF tables (made with it)

// poisson_inv(u, lambda, exp(-lambda)) from the table cdf[k] = F_k of the same recurrence: the first k with
// u <= F_k (u and F_k are non-negative, so their bit patterns compare as integers); past the table the
// recurrence goes on from (p, F) at k = kPoisTab - 1, as poisson_inv would.
__device__ __forceinline__ uint32_t poisson_tab(double u, const double* cdf, double plast, double lambda) {
    uint32_t k = 0;
    while (k < kPoisTab && lt_nonneg(cdf[k], u)) ++k;
    if (k < kPoisTab) return k;
    k = kPoisTab - 1u;
    double pk = plast, F = cdf[k];
    while (u > F && k < 4096u) {
        ++k;
        poisson_step(pk, F, lambda, k);
    }
    return k;
}

// Programmatic dependent launch: a kernel launched with launch_k is set up while its predecessor in the stream ends.
// pdl_wait returns when the predecessor has ended and its writes are visible; every block of every such kernel
// calls it before it touches memory (so a predecessor's end means that all before it ended, too).  No kernel
// triggers its successor early (griddepcontrol.launch_dependents): blocks that are resident and wait cost the running
// ones more than their start (a generation of 10,000 individuals 67.6 us with early triggers, 61.5 without; without
// the programmatic dependency 65.6, and 84 against 71 us launched one by one).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Monotone bucket of a position in [0,1) (values outside are clamped).
// floor(x * NB) for x in (0, 1), from the bits with integer operations: 0 for
// x <= 0 (and subnormals), NB - 1 for x >= 1.  Monotone, which is all the
// bucket index needs (the rank kernels and the threshold search use this one
// function; ranks are exact within a bucket), and off the FP64 pipe.
__device__ inline uint32_t pos_bucket(double x, uint32_t NB) {
    const uint64_t b = (uint64_t)__double_as_longlong(x);
    if ((b >> 63) || b == 0ull) return 0u;
    const int ex = (int)((b >> 52) & 0x7FFu) - 1023;                     // x = 1.f * 2^ex
    if (ex >= 0) return NB - 1u;
    const uint64_t m = (b & 0x000FFFFFFFFFFFFFull) | (1ull << 52);      // 53-bit significand
    const int sh = -ex - 1;                                              // x * 2^53 = m >> sh
    const uint64_t v = sh >= 64 ? 0ull : (m >> sh);
    const uint32_t k = (uint32_t)__umul64hi(v << 11, (uint64_t)NB);     // floor(v * NB / 2^53)
    return k < NB - 1u ? k : NB - 1u;
}

// x < y for positions (doubles >= 0, -0.0 included) as an integer compare of
// the bit patterns with the sign cleared.
__device__ inline bool pos_lt(double x, double y) {
    return ((unsigned long long)__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFull) <
           ((unsigned long long)__double_as_longlong(y) & 0x7FFFFFFFFFFFFFFFull);
}

}  // namespace clotho

// ---------------------------------------------------------------------------
// Host-side launch wrappers (defined in the kernel translation units).
namespace clotho {
struct LaunchCfg {
    cudaStream_t stream;
    int num_sms;
    uint32_t ind_per_sm = 16;     // blocks per SM of the per-individual kernels (selection, fitness)
    bool narrow_ok = true;        // the narrow build of k_generation may run when every row fits it
    const PopDev* one = nullptr;  // host copy of the descriptor of a launch's only population
    // which block works on which population of a batch (device tables, by BlockTable)
    const struct BlockPart* parts[3] = {nullptr, nullptr, nullptr};
    uint32_t blocks[3] = {0, 0, 0};
};
// Kernels of 256 threads, of 1,024 (every population has at least two blocks), and the row plans, whose work goes with
// the breakpoints as well.
enum BlockTable : uint32_t { kTable256 = 0, kTable1024 = 1, kTablePlan = 2 };
// A block's population and its place among that population's blocks.  A batch's blocks are dealt out in proportion to
// the populations' work by their capacities: with as many for each, the largest population's blocks ran when the
// others' were done (64 populations of 1,000 to 20,000 individuals, a generation: plans 119 -> 64 us, fitness
// 73 -> 62, first stage 47 -> 36).
struct BlockPart {
    uint32_t pop, i, n, pad;
};

// Population-parallel launches: blockIdx.z walks the populations, so small
// populations of a batch run side by side; blockIdx.x (and .y) stride inside
// one population.  per_pop bounds the useful blocks of one population.
inline dim3 pop_grid(uint32_t npops, uint32_t per_pop, int num_sms, uint32_t per_sm = 4) {
    const uint32_t gz = npops < 1u ? 1u : (npops > 65535u ? 65535u : npops);
    uint32_t gx = (uint32_t)num_sms * per_sm / gz;
    if (gx > per_pop) gx = per_pop;
    if (gx < 1u) gx = 1u;
    return dim3(gx, 1u, gz);
}
inline uint32_t blocks_for(uint64_t n, uint32_t per_block) {
    const uint64_t b = (n + per_block - 1) / per_block;
    return b < 1 ? 1u : (b > 0x7fffffffull ? 0x7fffffffu : (uint32_t)b);
}
template <bool ONE>
__device__ __forceinline__ BlockPart block_part(const BlockPart* map) {
    return ONE ? BlockPart{0u, blockIdx.x, gridDim.x, 0u} : map[blockIdx.x];
}

// Launch with the programmatic dependency of pdl_wait.
template <class... P, class... A>
inline cudaError_t launch_smem_k(const LaunchCfg& L, void (*k)(P...), dim3 grid, dim3 block, size_t smem, A... a) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = L.stream;
    c.attrs = &at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, k, static_cast<P>(a)...);
}
template <class... P, class... A>
inline cudaError_t launch_k(const LaunchCfg& L, void (*k)(P...), dim3 grid, dim3 block, A... a) {
    return launch_smem_k(L, k, grid, block, 0, a...);
}

// The kernels of a step are templates over ONE: with one population its descriptor comes in the kernel's parameters
// (the constant bank) instead of an array in memory, which takes a round trip to L2 off each kernel's chain of
// dependent loads.
// grid: blocks for one population; a batch takes its table's.
template <class K, class... A>
inline cudaError_t launch_pops_smem(const LaunchCfg& L, BlockTable table, K one, K all, uint32_t grid, size_t smem,
                                    const PopDev* pops, uint32_t npops, A... a) {
    if (npops == 0u) return cudaErrorInvalidValue;   // the tables may hold an earlier batch's blocks
    const bool single = npops == 1u;
    const K k = single ? one : all;
    if (smem > 48u * 1024u) {  // a property of the function on the current device; setting it again is harmless
        const cudaError_t e =
            cudaFuncSetAttribute((const void*)k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    return launch_smem_k(L, k, dim3(single ? grid : L.blocks[table]), dim3(table == kTable1024 ? 1024u : 256u), smem,
                         single ? *L.one : PopDev{}, pops, single ? nullptr : L.parts[table], a...);
}
template <class K, class... A>
inline cudaError_t launch_pops(const LaunchCfg& L, BlockTable table, K one, K all, uint32_t grid, const PopDev* pops,
                               uint32_t npops, A... a) {
    return launch_pops_smem(L, table, one, all, grid, 0, pops, npops, a...);
}
// Blocks of one population's launch: per_pop useful ones, at most per_sm an SM.
inline uint32_t blocks_of(const LaunchCfg& L, uint32_t per_pop, uint32_t per_sm) {
    const uint32_t most = (uint32_t)L.num_sms * per_sm;
    return per_pop < 1u ? 1u : per_pop < most ? per_pop : most;
}

// which: 0 = current child rows, 1 = parent rows of the step in progress
void launch_fs_reduce(const LaunchCfg&, const PopDev* pops, uint32_t npops, uint32_t maxW, uint32_t which);
// staged API: the step header; the free-space analysis and the child's allele count
void launch_begin(const LaunchCfg&, const PopDev* pops, uint32_t npops, const uint32_t* hdr, WorkCtl* ctl);
void launch_fs_finalize(const LaunchCfg&, const PopDev* pops, uint32_t npops);

// What launch_prep does.  Begin: header and free space; Mut: mutation counts and slots (Tape: of tapes);
// Order: the rows' processing order (Select: with parents drawn on the device); position buckets always.
constexpr uint32_t kStepBegin = 1u, kStepMut = 2u, kStepOrder = 4u, kStepSelect = 8u, kStepTape = 16u;
struct PrepSizes {
    uint32_t maxS, maxN, maxNB, maxA;   // largest capacities of the batch
    bool tables;                        // some population has a suffix table
};
// hdr: null in the staged API, where k_begin has set the sizes.  count_on: the step's generation kernel counts
// columns for the populations that asked (see generation_counts_fit); their counts are zeroed here and marked
// valid.  Returns the launches made.
uint32_t launch_prep(const LaunchCfg&, const PopDev* pops, uint32_t npops, const PrepSizes&, const uint32_t* hdr,
                     WorkCtl* ctl, uint32_t what, bool count_on);
// Allele capacity up to which a population's slots are ranked in shared memory: by eight blocks, each its share of the
// buckets, or in a batch by one (k_prep.cu).  Against global buckets, a generation of
// 300 individuals 24.4 / 28.4 us, of 100,000 99 / 107, of 1,000,000 809 / 814 (rho = 0.1, 1,250 slots in use).
constexpr uint32_t kDirectRanks = 8192;
inline bool direct_ranks(const PrepSizes& z) { return z.maxA <= kDirectRanks && z.tables; }
// One generation's tape from a pinned staging block into a population's tape arrays, and the step's header: seven pieces
// of whole 16-byte words (their ends padded; arrays and staging start on 16-byte boundaries).
struct TapePieces {
    const void* src[7];
    void* dst[7];
    uint32_t end[7];      // 16-byte words up to and with this piece
    uint32_t N, M;
};
void launch_tape_upload(const LaunchCfg&, const TapePieces&, uint32_t* hdr);
// dst[i * T + t] = src[i * 4 + t]
void launch_pack_traits(const LaunchCfg&, const double* src, double* dst, uint32_t n, uint32_t T);
// Poisson tables of one population (the device copy of its descriptor)
void launch_pois_tables(cudaStream_t s, const PopDev& P);
void launch_mut_resolve(const LaunchCfg&, const PopDev* pops, uint32_t npops);
void launch_select_philox(const LaunchCfg&, const PopDev* pops, uint32_t npops);
// Generation-kernel builds: suffix-table masks in per-warp bitmaps (capacity <= kSufMaxSlots), chunk by
// chunk from the table (populations with a table above that), interval classifier (populations without a
// table).  mixed: the batch holds populations of more than one kind; this launch runs only the populations
// of its own kind (build; maxW, maxA are theirs) and skips the others' items, so each population keeps the
// build it runs alone whatever it is batched with
enum GenBuild : int { kBuildInterval = 0, kBuildBitmap = 1, kBuildChunk = 2 };
cudaError_t launch_generation(const LaunchCfg&, const PopDev* pops, uint32_t npops, WorkCtl* ctl,
                              uint32_t maxW, uint32_t maxA, uint32_t fuse, int profile, GenBuild build,
                              bool count_on = false, bool mixed = false);
// whether the generation kernel's counting build fits this launch (suffix-table rows, counters in shared memory)
bool generation_counts_fit(uint32_t maxW, uint32_t maxA);
void launch_mut_scatter(const LaunchCfg&, const PopDev* pops, uint32_t npops);
void launch_phenotype(const LaunchCfg&, const PopDev* pops, uint32_t npops);
// How a step ends after the fitness: not here (a staged generation), with ++m_generation, or with that and the next
// header of a schedule (2 * npops words a step) copied to where the next step reads it.
struct StepEnd {
    enum Mode : uint32_t { kNone = 0, kStep = 1, kSchedule = 2 };
    uint32_t mode, npops;
    uint32_t* hdr;
    const WorkCtl* ctl;
};
// individual phenotypes, fitness (constant: no population has a metric) and its prefix sum, then the step's end.
// Returns the launches made.
uint32_t launch_fitness(const LaunchCfg&, const PopDev* pops, uint32_t npops, uint32_t maxN, bool constant, StepEnd end);
void launch_end(const LaunchCfg&, const PopDev* pops, uint32_t npops);
void launch_seed_rows(const LaunchCfg&, const PopDev* pops, uint32_t npops, const uint32_t* thr,
                      uint64_t seed, uint32_t A);
void launch_margins(const LaunchCfg&, const PopDev* pops, uint32_t p, uint32_t S, uint32_t W, uint32_t* colc,
                    uint32_t* rowc);
// sums over the current child for clotho_stats_compute, per block: traits 0..3, heterozygosity
constexpr uint32_t kStatBlocks = 128;
struct StatsOut {
    uint32_t segregating, fixed_now;
    double part[kStatBlocks][5];
};
// out and sfs (sfs_len counts) zero on entry; counts: carriers of every slot
void launch_stats(const LaunchCfg&, const PopDev* pops, uint32_t p, const uint32_t* counts, uint32_t sfs_len,
                  StatsOut* out, uint32_t* sfs);
// device accumulators of the pairwise-difference kernel
struct PairwiseOut {
    unsigned long long count, total, sumsq;
    unsigned int min, max;
    unsigned int err;   // a CTA gave up waiting for its multiplications
};
// how the pairs of n rows of W words are cut into CTAs, and the scratch that takes
struct PairwisePlan {
    uint32_t tiles, splits, per;       // per: rounds of eight 128-slot stages a CTA
    uint32_t group;                    // tiles a launch
    size_t sum_bytes;
};
PairwisePlan pairwise_plan(const LaunchCfg&, uint32_t n, uint32_t W);
cudaError_t launch_pairwise(const LaunchCfg&, const PopDev* pops, uint32_t p, const uint32_t* sample, uint32_t n,
                            const PairwisePlan&, void* scratch, uint32_t* dist, PairwiseOut* out);
// After launch_prep: the slots' ranks, the suffix tables and (tables: some population has one) the rows' plans.
// Returns the launches made.
uint32_t launch_plan(const LaunchCfg&, const PopDev* pops, uint32_t npops, const PrepSizes&, uint32_t maxW,
                     uint32_t what);
int init_recip_prep();  // k_prep.cu's copy of the reciprocal table
int init_recip_gen();   // k_generation.cu's copy

// crossover-plan row flags
constexpr uint32_t kPlanInv = 1u, kPlanLong = 2u, kPlanFlagShift = 30u;
constexpr uint32_t kPlanMaxEvents = (1u << kPlanFlagShift) - 1u;

// fuse flags of k_generation
constexpr uint32_t kFuseMut = 1u, kFusePheno = 2u, kFuseFs = 4u;
}  // namespace clotho
