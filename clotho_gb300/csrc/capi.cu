// capi.cu -- host side of the C-ABI (include/clotho_gpu.h).
//
// A context owns a set of resident populations (one for the plain engine) and
// two CUDA streams: a compute stream for every kernel and a copy stream for
// the uploads of large tapes.  Tape buffers are double-buffered, so that the
// host->device copies of generation g+1 overlap the kernels of generation g.
// Tapes of at most 1 MB are packed into a pinned block (one a buffer) and
// uploaded by a kernel on the compute stream.
#include "engine.cuh"
#include "../../include/clotho_gpu.h"

#include <sys/mman.h>
#include <unistd.h>

#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

using namespace clotho;

namespace {

struct PopHost {
    clotho_desc desc{};
    bool counting = false;    // asked for fused column counts (clotho_pop_count_columns)
    PopDev dev[3]{};          // tape set 0, tape set 1, device-drawn (Philox)
    void* arena = nullptr;          // every device table of the population, one pool block
    size_t bytes = 0;
    bool acc_valid = false;   // accF/accV hold AND/OR of the current child rows
    bool ready = false;       // init/seed done
    uint32_t hostN = 0;       // host view of N, while n_known
    bool n_known = false;     // false from a step's enqueuing to its call's success: a call that fails leaves the size open
};

struct Geometry {
    uint32_t Ncap, Scap, Wcap, Aslots, Mcap, EVcap, FXcap, T, NB;
    bool table;  // the population has a suffix table (its crossover classifier)
};

// Suffix tables above kSufMaxSlots slots (masks chunk by chunk) pay for themselves at low recombination: on
// GB300 at 2,352-word rows and rho = 1 the chunk-mask kernel took 2.65 against the interval classifier's
// 3.20 ms, while at 472-word rows it took 0.44 / 0.59 / 0.82 ms a generation against 0.45 / 0.51 / 0.60 ms at
// rho = 0.5 / 2 / 5 (each row's breakpoints cost a table load per chunk).
constexpr double kChunkMaxRho = 1.0;

Geometry geometry(const clotho_desc& d) {
    Geometry g{};
    g.Ncap = d.max_individuals ? d.max_individuals : 1;
    g.Scap = 2 * g.Ncap;
    uint32_t w = ref_width(d.max_alleles ? d.max_alleles : 1);
    g.Wcap = (w + kWordAlign - 1) / kWordAlign * kWordAlign;
    g.Aslots = g.Wcap * 64u;
    g.Mcap = d.max_mutations ? d.max_mutations : 1;
    g.EVcap = d.max_events ? d.max_events : 1;
    g.FXcap = d.max_fixed ? d.max_fixed : 1;
    g.T = d.traits;
    g.NB = 1024;
    while (g.NB < g.Aslots) g.NB <<= 1;
    g.table = g.Aslots <= kSufMaxSlots || (g.Aslots <= kTableMaxSlots && d.rho <= kChunkMaxRho);
    return g;
}

size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

// Byte sizes of every device array of one population, in allocation order.
std::vector<size_t> sizes_of(const Geometry& g) {
    const size_t S = g.Scap, N = g.Ncap, W = g.Wcap, A = g.Aslots, T = g.T;
    return {
        S * W * 8, S * W * 8,            // rows[0], rows[1]
        W * 8, W * 8, W * 8,             // fixmask, accF, accV
        A * 4, A * 8, A * 4, A * 16,     // free_list, pos, age, eff (traits padded to 4)
        g.FXcap * 8ull, g.FXcap * 4ull, g.FXcap * T * 4ull,
        S * 32, S * 32, N * 32, N * 8, N * 8,    // zg[0], zg[1], zi, fit, cdf
        (N / 1024 + 8) * 8, (N / 128 + 64) * 8, (kPoisTab + 1) * 8, (kPoisTab + 1) * 8, ((S > g.NB ? S : g.NB) / 1024 + 32) * 4ull, (N / 1024 + 32) * 4ull,
        (S + 1) * 4, (S + 1) * 4,        // row_cnt, row_off
        S * 4, g.Mcap * 4ull, g.Mcap * 4ull,  // row_cur, row_mut, mut_slot
        (g.NB + 1ull) * 4, (g.NB + 1ull) * 4, g.NB * 4ull, A * 8, A * 4, A * 4,  // bcnt, boff, bcur, bpos, bslot, rank
        g.table ? A * 4 : 0,                            // inv
        g.table ? (A / 64 + 1) * W * 8 : 0,             // suf
        g.table ? S * 16 : 0,                           // plan_row
        g.table ? N * 4 : 0,                            // ord_cnt
        g.table ? N * 4 : 0,                            // ord_cur
        g.table ? S * 4 : 0,                            // ord_pos
        g.table ? g.EVcap * 4ull : 0,                   // plan_go
        g.table ? g.EVcap * 4ull : 0,                   // plan_cr
        g.table ? S * 8 : 0,                            // plan_mut
        g.table ? S * 32 : 0,                           // plan_z
        A * 4,                                                    // colcnt
        sizeof(DevStatus),
        // two tape sets: pairs, swap, ev_off, ev_pos, mut_seq, mut_pos, mut_eff
        S * 4, S, (S + 1) * 4, g.EVcap * 8ull, g.Mcap * 4ull, g.Mcap * 8ull, g.Mcap * T * 4ull,
        S * 4, S, (S + 1) * 4, g.EVcap * 8ull, g.Mcap * 4ull, g.Mcap * 8ull, g.Mcap * T * 4ull,
    };
}

}  // namespace

struct clotho_ctx {
    int device = 0;
    int num_sms = 152;
    cudaStream_t stream = nullptr, copy_stream = nullptr;
    cudaStream_t own_stream = nullptr;  // the context's own compute stream (stream may be the caller's)
    // populations' device tables come from the context's own stream-ordered pool, which keeps freed
    // blocks for the next population (a serving loop adds and removes populations every few steps)
    cudaMemPool_t pool = nullptr;
    std::vector<PopHost*> pops;
    PopDev* d_pops[3] = {nullptr, nullptr, nullptr};  // per set: npops contiguous PopDev
    WorkCtl* d_ctl = nullptr;
    BlockPart* d_parts = nullptr;      // a batch's block tables (BlockTable), kMaxParts entries each
    uint32_t n_parts[3] = {0, 0, 0};
    bool parts_stale = true;
    bool parts_captured = false;             // a caller's graph may read d_parts
    std::vector<BlockPart*> parts_kept;      // tables that such graphs read, superseded
    uint32_t* d_hdr[3] = {nullptr, nullptr, nullptr}; // per set: [2*npops]
    // step headers (N, M per population) are staged in a ring of pinned slots:
    // a slot is reused only after the copy that read it has completed
    uint32_t* h_ring = nullptr;                         // [kHdrRing][2 * kMaxPops]
    // asynchronous status read-back: a pinned ring of status copies, each behind an event
    DevStatus* h_stat = nullptr;                        // [kStatRing]
    cudaEvent_t stat_ev[8]{};
    uint32_t stat_next = 0;                             // tickets issued so far
    cudaEvent_t ring_ev[64]{};
    bool ring_used[64]{};
    uint32_t ring_next = 0;
    char* h_tape[2] = {nullptr, nullptr};                // pinned staging of small tapes, one a tape set
    uint32_t set = 0;                                    // next tape set
    uint32_t pairs_set = 0;                              // the set whose pairs the last generation used
    cudaEvent_t copy_done[2]{}, kern_done[2]{};
    bool captured = false;   // a step went into a graph of the caller's: replays run steps that no call here tells of
    bool drawn = false;   // device-drawn steps, which share set 0's buffers, enqueued since kern_done[0] was recorded
    std::string err;
    bool profiling = false;
    bool phase_clocks = false;      // profiling with the phase-clock build of k_generation
    std::vector<cudaEvent_t> prof_ev;  // pairs around each k_generation launch
    size_t prof_used = 0;
    double prof_ms = 0.0;
    uint32_t prof_launches = 0;
    cudaEvent_t t0 = nullptr, t1 = nullptr;
    uint64_t launches = 0;
    cudaGraphExec_t graph = nullptr;        // one device-drawn generation
    cudaGraphExec_t graph_long = nullptr;   // kLongGraph of them, made when the key's replays pay for it
    uint64_t graph_launches = 0;  // kernels per generation of the graphs
    uint64_t replayed = 0;        // generations replayed under graph_key
    std::vector<uint32_t> graph_key;
    bool in_step = false;
    uint32_t maxW = 0, maxS = 0, maxN = 0, maxNB = 0, maxA = 0;
    // per generation-kernel build: suffix-table masks in bitmaps (bm, at most kSufMaxSlots slots) or chunk by
    // chunk (cm, the other populations with a table), interval classifier (iv, no table); suf = bm + cm
    uint32_t n_suf = 0, n_iv = 0, maxW_suf = 0, maxW_iv = 0, maxA_suf = 0, maxA_iv = 0;
    uint32_t n_bm = 0, n_cm = 0, maxW_bm = 0, maxW_cm = 0, maxA_bm = 0, maxA_cm = 0;
    cudaError_t launch_err = cudaSuccess;  // a launch set-up failure, reported by the next check_launch
    uint32_t ind_per_sm = 16;               // tuning (clotho_set_tuning)
    bool narrow_ok = true;
    uint32_t tuning_epoch = 0;              // part of every graph's key: a new tuning re-captures
    uint32_t counting = 0;                  // populations that asked for fused column counts
};

namespace {

constexpr uint32_t kHdrRing = 64;
constexpr uint32_t kMaxParts = 4096;   // blocks of a batch's launch at most
constexpr uint32_t kStatRing = 8;   // outstanding asynchronous status reads (clotho_info_request)
static_assert(sizeof(((clotho_ctx*)nullptr)->ring_ev) / sizeof(cudaEvent_t) == kHdrRing, "header ring size");
static_assert(sizeof(((clotho_ctx*)nullptr)->stat_ev) / sizeof(cudaEvent_t) == kStatRing, "status ring size");

int fail(clotho_ctx* c, int code, const std::string& m) {
    if (c) c->err = m;
    return code;
}

// The runtime's record of the error goes with its report: left there, the next call that checks its launches would
// report it again.
#define CK(call)                                                                                      \
    do {                                                                                              \
        cudaError_t e_ = (call);                                                                      \
        if (e_ != cudaSuccess) {                                                                      \
            cudaGetLastError();                                                                       \
            return fail(ctx, CLOTHO_E_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_));      \
        }                                                                                             \
    } while (0)

// set: the descriptors that the launch takes (tape set 0 or 1, or 2 for device draws)
LaunchCfg cfg(clotho_ctx* ctx, uint32_t set = 0) {
    LaunchCfg L{ctx->stream, ctx->num_sms};
    if (!ctx->pops.empty()) L.one = &ctx->pops[0]->dev[set];  // taken by launches over the first population alone
    for (uint32_t k = 0; k < 3; ++k) {
        L.parts[k] = ctx->d_parts ? ctx->d_parts + k * kMaxParts : nullptr;
        L.blocks[k] = ctx->n_parts[k];
    }
    L.ind_per_sm = ctx->ind_per_sm;
    L.narrow_ok = ctx->narrow_ok;
    return L;
}

// The context's stream is inside a graph capture of the caller's (false for the library's own: they end in their call).
bool capturing(clotho_ctx* ctx) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(ctx->stream, &st) != cudaSuccess) cudaGetLastError();
    return st != cudaStreamCaptureStatusNone;
}

// A pinned slot for one step header; nullptr if pinned memory is unavailable.
uint32_t* hdr_stage(clotho_ctx* ctx, uint32_t* slot) {
    if (!ctx->h_ring) {
        if (cudaMallocHost(&ctx->h_ring, sizeof(uint32_t) * 2 * kMaxPops * kHdrRing) != cudaSuccess) {
            cudaGetLastError();
            ctx->h_ring = nullptr;
            return nullptr;
        }
        for (uint32_t k = 0; k < kHdrRing; ++k) cudaEventCreateWithFlags(&ctx->ring_ev[k], cudaEventDisableTiming);
    }
    const uint32_t k = ctx->ring_next;
    ctx->ring_next = (k + 1) % kHdrRing;
    if (ctx->ring_used[k]) cudaEventSynchronize(ctx->ring_ev[k]);
    *slot = k;
    return ctx->h_ring + (size_t)k * 2 * kMaxPops;
}

// Copy n headers from slot into dst on stream s and mark the slot busy until then.
int hdr_copy(clotho_ctx* ctx, uint32_t slot, uint32_t* dst, uint32_t n, cudaStream_t s) {
    if (s == ctx->stream) ctx->captured |= capturing(ctx);
    CK(cudaMemcpyAsync(dst, ctx->h_ring + (size_t)slot * 2 * kMaxPops, 8ull * n, cudaMemcpyHostToDevice, s));
    CK(cudaEventRecord(ctx->ring_ev[slot], s));
    ctx->ring_used[slot] = true;
    return 0;
}

// Scratch device memory for a call, from the context's stream-ordered pool (freed with cudaFreeAsync on
// the context's stream): no device-wide synchronisation, unlike cudaMalloc / cudaFree.
template <class T>
cudaError_t pool_alloc(clotho_ctx* ctx, T** p, size_t bytes) {
    return cudaMallocFromPoolAsync(reinterpret_cast<void**>(p), bytes, ctx->pool, ctx->stream);
}

int check_launch(clotho_ctx* ctx, const char* what) {
    cudaError_t e = cudaGetLastError();
    if (ctx->launch_err != cudaSuccess) {
        e = ctx->launch_err;
        ctx->launch_err = cudaSuccess;
    }
    if (e != cudaSuccess) return fail(ctx, CLOTHO_E_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
    return 0;
}

// The caller has synchronized the context's streams: nothing reads the tables any more.
void free_pop(clotho_ctx* ctx, PopHost* p) {
    if (p->arena) cudaFreeAsync(p->arena, ctx->own_stream);
    p->arena = nullptr;
    delete p;
}

int alloc_pop(clotho_ctx* ctx, const clotho_desc& d, PopHost** out) {
    if (d.traits < 1 || d.traits > kMaxTraits) return fail(ctx, CLOTHO_E_ARG, "traits must be 1..4");
    if (d.max_individuals == 0 || d.max_alleles == 0) return fail(ctx, CLOTHO_E_ARG, "zero capacity");
    const Geometry g = geometry(d);
    PopHost* p = new PopHost();
    p->desc = d;
    std::vector<size_t> sz = sizes_of(g);
    std::vector<void*> ptr(sz.size(), nullptr);
    // one block for all tables, each at a 256-byte aligned offset (optional tables of size 0 stay null)
    size_t total = 0;
    for (size_t x : sz) total += align256(x);
    cudaError_t e = cudaMallocFromPoolAsync(&p->arena, total, ctx->pool, ctx->own_stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->own_stream);  // ready before other streams use it
    if (e != cudaSuccess) {
        cudaGetLastError();
        p->arena = nullptr;
        delete p;
        return fail(ctx, CLOTHO_E_NOMEM, "device allocation refused (" + std::to_string(total) + " bytes)");
    }
    p->bytes = total;
    for (size_t i = 0, off = 0; i < sz.size(); off += align256(sz[i]), ++i)
        if (sz[i]) ptr[i] = static_cast<char*>(p->arena) + off;
    // zero the tables and the status: everything after the two row sets, in one call
    const size_t rows_bytes = align256(sz[0]) + align256(sz[1]);
    if (total > rows_bytes) cudaMemsetAsync(static_cast<char*>(p->arena) + rows_bytes, 0, total - rows_bytes, ctx->stream);
    PopDev b{};
    size_t k = 0;
    b.rows[0] = (uint64_t*)ptr[k++]; b.rows[1] = (uint64_t*)ptr[k++];
    b.fixmask = (uint64_t*)ptr[k++]; b.accF = (uint64_t*)ptr[k++]; b.accV = (uint64_t*)ptr[k++];
    b.free_list = (uint32_t*)ptr[k++]; b.pos = (double*)ptr[k++]; b.age = (uint32_t*)ptr[k++]; b.eff = (float*)ptr[k++];
    b.fx_pos = (double*)ptr[k++]; b.fx_age = (uint32_t*)ptr[k++]; b.fx_eff = (float*)ptr[k++];
    b.zg[0] = (double*)ptr[k++]; b.zg[1] = (double*)ptr[k++];
    b.zi = (double*)ptr[k++]; b.fit = (double*)ptr[k++]; b.cdf = (double*)ptr[k++];
    b.scan_part = (double*)ptr[k++]; b.scan_wsum = (double*)ptr[k++];
    b.pois_mu = (double*)ptr[k++]; b.pois_rho = (double*)ptr[k++];
    b.scan_upart = (uint32_t*)ptr[k++]; b.scan_opart = (uint32_t*)ptr[k++];
    b.row_cnt = (uint32_t*)ptr[k++]; b.row_off = (uint32_t*)ptr[k++];
    b.row_cur = (uint32_t*)ptr[k++]; b.row_mut = (uint32_t*)ptr[k++]; b.mut_slot = (uint32_t*)ptr[k++];
    b.bcnt = (uint32_t*)ptr[k++]; b.boff = (uint32_t*)ptr[k++];
    b.bcur = (uint32_t*)ptr[k++]; b.bpos = (double*)ptr[k++]; b.bslot = (uint32_t*)ptr[k++];
    b.rank = (uint32_t*)ptr[k++]; b.inv = (uint32_t*)ptr[k++]; b.suf = (uint64_t*)ptr[k++];
    b.plan_row = (uint4*)ptr[k++];
    b.ord_cnt = (uint32_t*)ptr[k++]; b.ord_cur = (uint32_t*)ptr[k++]; b.ord_pos = (uint32_t*)ptr[k++];
    b.plan_go = (uint32_t*)ptr[k++]; b.plan_cr = (uint32_t*)ptr[k++];
    b.plan_mut = (uint2*)ptr[k++]; b.plan_z = (double*)ptr[k++];
    b.colcnt = (uint32_t*)ptr[k++];
    b.st = (DevStatus*)ptr[k++];
    b.Scap = g.Scap; b.Ncap = g.Ncap; b.Wcap = g.Wcap; b.Acap = g.Aslots; b.Mcap = g.Mcap;
    b.EVcap = g.EVcap; b.FXcap = g.FXcap; b.T = g.T; b.NB = g.NB;
    b.mu = d.mu; b.rho = d.rho; b.bias = d.bias; b.p_neutral = d.p_neutral;
    b.eff_mean = d.eff_mean; b.eff_sigma = d.eff_sigma; b.fit_param = d.fit_param;
    b.exp_neg_rho = std::exp(-d.rho);
    b.exp_neg_mu = std::exp(-d.mu);
    b.seed = d.seed; b.fitness = d.fitness; b.flags = d.flags;
    for (int s = 0; s < 2; ++s) {
        PopDev t = b;
        t.mode = kModeTape;
        t.pairs = (uint32_t*)ptr[k++]; t.swap = (uint8_t*)ptr[k++]; t.ev_off = (uint32_t*)ptr[k++];
        t.ev_pos = (double*)ptr[k++]; t.mut_seq = (uint32_t*)ptr[k++]; t.mut_pos = (double*)ptr[k++];
        t.mut_eff = (float*)ptr[k++];
        p->dev[s] = t;
    }
    p->dev[2] = p->dev[0];
    p->dev[2].mode = kModePhilox;
    launch_pois_tables(ctx->stream, b);
    *out = p;
    return 0;
}

// Steps were enqueued, and a call has succeeded: N(i) individuals in population i.
void sizes_open(clotho_ctx* ctx) {
    for (PopHost* p : ctx->pops) p->n_known = false;
}
template <class F>
void sizes_are(clotho_ctx* ctx, F N) {
    for (size_t i = 0; i < ctx->pops.size(); ++i) {
        ctx->pops[i]->hostN = N(i);
        ctx->pops[i]->n_known = !ctx->captured;
    }
}

void drop_graphs(clotho_ctx* ctx) {
    for (cudaGraphExec_t* g : {&ctx->graph, &ctx->graph_long}) {
        if (*g) cudaGraphExecDestroy(*g);
        *g = nullptr;
    }
    ctx->graph_key.clear();
    ctx->replayed = 0;
}

// Rebuild the device PopDev arrays after the population set changed: entries
// [from, n) are copied (an add changes the last one, a remove shifts the rest).
int sync_pop_arrays(clotho_ctx* ctx, uint32_t from = 0) {
    const uint32_t n = (uint32_t)ctx->pops.size();
    if (n > kMaxPops) return fail(ctx, CLOTHO_E_CAPACITY, "more than 256 populations");
    for (int s = 0; s < 3; ++s) {
        // sized for kMaxPops once, so adding or removing a population allocates nothing here
        if (!ctx->d_pops[s]) CK(cudaMalloc(&ctx->d_pops[s], sizeof(PopDev) * kMaxPops));
        if (!ctx->d_hdr[s]) CK(cudaMalloc(&ctx->d_hdr[s], sizeof(uint32_t) * 2 * kMaxPops));
        if (from >= n) continue;
        std::vector<PopDev> h(n - from);
        for (uint32_t i = from; i < n; ++i) h[i - from] = ctx->pops[i]->dev[s];
        CK(cudaMemcpyAsync(ctx->d_pops[s] + from, h.data(), sizeof(PopDev) * (n - from), cudaMemcpyHostToDevice,
                           ctx->stream));
    }
    ctx->maxW = ctx->maxS = ctx->maxN = ctx->maxNB = ctx->maxA = 0;
    ctx->n_suf = ctx->n_iv = ctx->maxW_suf = ctx->maxW_iv = ctx->maxA_suf = ctx->maxA_iv = 0;
    ctx->n_bm = ctx->n_cm = ctx->maxW_bm = ctx->maxW_cm = ctx->maxA_bm = ctx->maxA_cm = 0;
    for (PopHost* p : ctx->pops) {
        const PopDev& D = p->dev[0];
        ctx->maxW = std::max(ctx->maxW, D.Wcap);
        ctx->maxS = std::max(ctx->maxS, D.Scap);
        ctx->maxN = std::max(ctx->maxN, D.Ncap);
        ctx->maxNB = std::max(ctx->maxNB, D.NB);
        ctx->maxA = std::max(ctx->maxA, D.Acap);
        if (D.suf != nullptr) {
            ctx->n_suf += 1;
            ctx->maxW_suf = std::max(ctx->maxW_suf, D.Wcap);
            ctx->maxA_suf = std::max(ctx->maxA_suf, D.Acap);
            if (D.Acap <= kSufMaxSlots) {
                ctx->n_bm += 1;
                ctx->maxW_bm = std::max(ctx->maxW_bm, D.Wcap);
                ctx->maxA_bm = std::max(ctx->maxA_bm, D.Acap);
            } else {
                ctx->n_cm += 1;
                ctx->maxW_cm = std::max(ctx->maxW_cm, D.Wcap);
                ctx->maxA_cm = std::max(ctx->maxA_cm, D.Acap);
            }
        } else {
            ctx->n_iv += 1;
            ctx->maxW_iv = std::max(ctx->maxW_iv, D.Wcap);
            ctx->maxA_iv = std::max(ctx->maxA_iv, D.Acap);
        }
    }
    drop_graphs(ctx);
    ctx->parts_stale = true;
    CK(cudaStreamSynchronize(ctx->stream));
    return 0;
}

// Lets the thread allocate and wait on streams that are not captured, whatever the mode of its captures.
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// The block tables of a batch, made anew before the first step after its populations (or the tuning) changed: blocks
// in proportion to the populations' rows (plans: rows and breakpoints), a few an SM (by the tuning; two of 1,024
// threads), so that blocks that come later even out what the proportions miss.  A step may be captured in a graph of
// the caller's, so the tables are written on the copy stream (nothing on the context's stream reads stale tables: what
// makes them stale waits for it), and tables that such a graph reads are left as they are.
int block_tables(clotho_ctx* ctx) {
    const size_t n = ctx->pops.size();
    if (n < 2) return 0;
    const bool captured = capturing(ctx);
    if (!ctx->parts_stale) {
        ctx->parts_captured |= captured;
        return 0;
    }
    const RelaxedCapture relaxed;
    if (ctx->d_parts && ctx->parts_captured) {
        ctx->parts_kept.push_back(ctx->d_parts);
        ctx->d_parts = nullptr;
    }
    if (!ctx->d_parts)
        CK(cudaMallocFromPoolAsync(reinterpret_cast<void**>(&ctx->d_parts), sizeof(BlockPart) * 3 * kMaxParts, ctx->pool,
                                   ctx->copy_stream));
    ctx->parts_captured = captured;
    std::vector<BlockPart> h(3 * kMaxParts);
    for (uint32_t k = 0; k < 3; ++k) {
        auto work = [k](const PopHost* p) { return p->dev[0].Scap * (k == kTablePlan ? 1.0 + 0.4 * p->desc.rho : 1.0); };
        double sum = 0.0;
        for (const PopHost* p : ctx->pops) sum += work(p);
        const uint32_t least = k == kTable1024 ? 2u : 1u;   // there a population's first block has a job of its own
        const double all = std::min<double>(
            (double)ctx->num_sms * (k == kTable1024 ? 2u : std::max(1u, ctx->ind_per_sm / 2u)), kMaxParts - (double)n * least);
        uint32_t at = 0;
        for (uint32_t p = 0; p < n; ++p) {
            const uint32_t b = std::max(least, (uint32_t)(all * work(ctx->pops[p]) / sum));
            for (uint32_t i = 0; i < b; ++i) h[k * kMaxParts + at++] = BlockPart{p, i, b, 0u};
        }
        ctx->n_parts[k] = at;
    }
    CK(cudaMemcpyAsync(ctx->d_parts, h.data(), h.size() * sizeof(BlockPart), cudaMemcpyHostToDevice, ctx->copy_stream));
    CK(cudaStreamSynchronize(ctx->copy_stream));
    ctx->parts_stale = false;
    return 0;
}

DevStatus read_status(clotho_ctx* ctx, PopHost* p, int* rc) {
    DevStatus s{};
    cudaError_t e = cudaMemcpyAsync(&s, p->dev[0].st, sizeof(DevStatus), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    *rc = (e == cudaSuccess) ? 0 : fail(ctx, CLOTHO_E_CUDA, std::string("status read: ") + cudaGetErrorString(e));
    return s;
}

// The population's current size: the host's own view, or after a failed call the device's.
uint32_t current_N(clotho_ctx* ctx, PopHost* p, int* rc) {
    *rc = 0;
    if (!p->n_known) {
        const uint32_t N = read_status(ctx, p, rc).N;
        if (*rc == 0) p->hostN = N;
        p->n_known = *rc == 0 && !ctx->captured;
    }
    return p->hostN;
}

// Backs a caller's buffer with memory before the device writes to it.  On a machine whose GPU walks the host's page
// tables, a copy into pages that the host has never touched faults them in one after another from the device: 6.2 ms
// for 6.4 MB, where the kernel call here takes 0.3 and the copy 0.1.  Contents stay; where the call is not known
// the copy faults as before.
void host_pages(void* p, size_t bytes) {
#ifdef MADV_POPULATE_WRITE
    if (bytes < (64u << 10)) return;
    const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE);
    const uintptr_t a = (uintptr_t)p & ~(page - 1), b = ((uintptr_t)p + bytes + page - 1) & ~(page - 1);
    madvise(reinterpret_cast<void*>(a), b - a, MADV_POPULATE_WRITE);
#else
    (void)p;
    (void)bytes;
#endif
}

// ---- profiling around the generation kernel
void prof_begin(clotho_ctx* ctx) {
    if (!ctx->profiling) return;
    if (ctx->prof_used + 2 > ctx->prof_ev.size()) {
        for (int i = 0; i < 64; ++i) {
            cudaEvent_t e;
            if (cudaEventCreate(&e) != cudaSuccess) {  // out of events: stop timing, keep running
                cudaGetLastError();
                ctx->profiling = false;
                return;
            }
            ctx->prof_ev.push_back(e);
        }
    }
    cudaEventRecord(ctx->prof_ev[ctx->prof_used], ctx->stream);
}
void prof_end(clotho_ctx* ctx) {
    if (!ctx->profiling) return;
    cudaEventRecord(ctx->prof_ev[ctx->prof_used + 1], ctx->stream);
    ctx->prof_used += 2;
    ctx->prof_launches += 1;
}
int prof_collect(clotho_ctx* ctx) {
    if (ctx->prof_used == 0) return 0;
    CK(cudaStreamSynchronize(ctx->stream));
    for (size_t i = 0; i + 1 < ctx->prof_used; i += 2) {
        float ms = 0.f;
        CK(cudaEventElapsedTime(&ms, ctx->prof_ev[i], ctx->prof_ev[i + 1]));
        ctx->prof_ms += ms;
    }
    ctx->prof_used = 0;
    return 0;
}

// The fused step's generation kernel counts columns (its counting build) when a population asked and the
// counters fit in shared memory; the step's first kernel zeroes those counts and marks them valid.
bool count_on(clotho_ctx* ctx, uint32_t fuse) {
    return ctx->counting > 0 && ctx->n_bm > 0 && (fuse & kFuseFs) && !(ctx->profiling && ctx->phase_clocks) &&
           generation_counts_fit(ctx->maxW_bm, ctx->maxA_bm);
}

// The generation kernel over every population: one launch when all populations use the same build; in a
// batch that mixes them, one launch per build (bitmap, chunk-mask, interval), each over its own populations,
// so every population runs the build it runs alone.
void launch_gen(clotho_ctx* ctx, const LaunchCfg& L, const PopDev* pops, uint32_t npops, uint32_t fuse) {
    const int prof = ctx->profiling ? (ctx->phase_clocks ? 2 : 1) : 0;
    const uint32_t kinds = (ctx->n_bm > 0) + (ctx->n_cm > 0) + (ctx->n_iv > 0);
    const bool mixed = kinds > 1;
    const bool cnt = count_on(ctx, fuse);
    const uint32_t pn[3] = {ctx->n_bm, ctx->n_cm, ctx->n_iv};
    const uint32_t pW[3] = {ctx->maxW_bm, ctx->maxW_cm, ctx->maxW_iv};
    const uint32_t pA[3] = {ctx->maxA_bm, ctx->maxA_cm, ctx->maxA_iv};
    const GenBuild builds[3] = {kBuildBitmap, kBuildChunk, kBuildInterval};
    for (int pass = 0; pass < 3; ++pass) {
        if (pn[pass] == 0) continue;
        const uint32_t W = mixed ? pW[pass] : ctx->maxW;
        const uint32_t A = mixed ? pA[pass] : ctx->maxA;
        prof_begin(ctx);
        const cudaError_t e =
            launch_generation(L, pops, npops, ctx->d_ctl, W, A, fuse, prof, builds[pass], cnt, mixed);
        if (e != cudaSuccess && ctx->launch_err == cudaSuccess) ctx->launch_err = e;
        prof_end(ctx);
        ctx->launches += 1;
    }
}

template <class T>
int h2d(clotho_ctx* ctx, T* dst, const T* src, size_t n, cudaStream_t s) {
    if (n == 0) return 0;
    if (!src) return fail(ctx, CLOTHO_E_ARG, "null host array");
    CK(cudaMemcpyAsync(dst, src, n * sizeof(T), cudaMemcpyHostToDevice, s));
    return 0;
}

// Host arrays of a tape and where they go in tape set s, in elements.
struct TapeArray {
    void* dst;
    const void* src;
    size_t bytes;
};
int tape_arrays(clotho_ctx* ctx, PopHost* p, uint32_t s, const clotho_gen_tape* t, TapeArray (&out)[7]) {
    const PopDev& D = p->dev[s];
    const uint32_t N = t->N, M = t->M, T = D.T;
    if (N > D.Ncap) return fail(ctx, CLOTHO_E_CAPACITY, "tape N exceeds max_individuals");
    if (M > D.Mcap) return fail(ctx, CLOTHO_E_CAPACITY, "tape M exceeds max_mutations");
    if (!t->ev_off) return fail(ctx, CLOTHO_E_ARG, "tape ev_off is null");
    const size_t S = 2ull * N;
    const uint32_t ev_total = t->ev_off[S];
    if (ev_total > D.EVcap) return fail(ctx, CLOTHO_E_CAPACITY, "tape events exceed max_events");
    uint32_t down = 0;  // no early exit: the loop runs in vectors
    for (size_t g = 0; g < S; ++g) down |= t->ev_off[g] > t->ev_off[g + 1] ? 1u : 0u;
    if (down) return fail(ctx, CLOTHO_E_ARG, "tape ev_off not monotone");
    const TapeArray all[7] = {{D.pairs, t->pairs, S * 4},       {D.swap, t->swap, S},
                              {D.ev_off, t->ev_off, (S + 1) * 4}, {D.ev_pos, t->ev_pos, ev_total * 8ull},
                              {D.mut_seq, t->mut_seq, M * 4ull}, {D.mut_pos, t->mut_pos, M * 8ull},
                              {D.mut_eff, t->mut_eff, (size_t)M * T * 4}};
    for (int i = 0; i < 7; ++i) {
        if (all[i].bytes && !all[i].src) return fail(ctx, CLOTHO_E_ARG, "null host array");
        out[i] = all[i];
    }
    return 0;
}

// Tapes up to this size are packed into a pinned block by the host and read from there by one kernel; above, the host's
// own copying (15 GB/s) takes longer than the copies' calls.
constexpr size_t kTapeStage = 1u << 20;

// Calls that work on the first population, or on all as if there were at least one.
int require_pop(clotho_ctx* ctx) {
    if (!ctx) return CLOTHO_E_ARG;
    return ctx->pops.empty() ? fail(ctx, CLOTHO_E_ARG, "the context has no population") : 0;
}

int require_ready(clotho_ctx* ctx) {
    if (!ctx) return CLOTHO_E_ARG;
    for (PopHost* p : ctx->pops)
        if (!p->ready) return fail(ctx, CLOTHO_E_STATE, "population not initialised (clotho_init / clotho_seed_population)");
    return 0;
}

// None of the first n populations has a fitness metric (every fitness is 1).
bool constant_fitness(const clotho_ctx* ctx, uint32_t n) {
    for (uint32_t i = 0; i < n; ++i)
        if (ctx->pops[i]->desc.fitness >= CLOTHO_FIT_GAUSSIAN && ctx->pops[i]->desc.fitness <= CLOTHO_FIT_GAUSSIAN_VS)
            return false;
    return true;
}

PrepSizes prep_sizes(const clotho_ctx* ctx) {
    return PrepSizes{ctx->maxS, ctx->maxN, ctx->maxNB, ctx->maxA, ctx->n_suf > 0};
}

// Make accF/accV of every population hold the AND/OR of its current rows
// (called before a step when the previous one did not fuse them).
void ensure_parent_acc(clotho_ctx* ctx, const PopDev* pops, uint32_t npops) {
    bool need = false;
    for (PopHost* p : ctx->pops) need |= !p->acc_valid;
    if (need) {
        launch_fs_reduce(cfg(ctx), pops, npops, ctx->maxW, 0u);
        ctx->launches += 1;
    }
}

// The fused step shared by tape and device-drawn modes, for every population.
void enqueue_fused_step(clotho_ctx* ctx, uint32_t set, bool philox, StepEnd::Mode end = StepEnd::kStep) {
    // (block_tables has run: the callers that can hold several populations see to it)
    const uint32_t n = (uint32_t)ctx->pops.size();
    const PopDev* pops = ctx->d_pops[set];
    const LaunchCfg L = cfg(ctx, set);
    ctx->pairs_set = set == 1u ? 1u : 0u;  // the device-drawn set (2) shares set 0's buffers
    ctx->drawn |= philox;
    sizes_open(ctx);
    ensure_parent_acc(ctx, pops, n);
    const PrepSizes z = prep_sizes(ctx);
    const bool cnt = count_on(ctx, kFuseMut | kFusePheno | kFuseFs);
    const uint32_t what = kStepBegin | kStepMut | kStepOrder | (philox ? kStepSelect : kStepTape);
    ctx->launches += launch_prep(L, pops, n, z, ctx->d_hdr[set], ctx->d_ctl, what, cnt);
    ctx->launches += launch_plan(L, pops, n, z, ctx->maxW_suf, what);
    launch_gen(ctx, L, pops, n, kFuseMut | kFusePheno | kFuseFs);
    ctx->launches += launch_fitness(L, pops, n, ctx->maxN, constant_fitness(ctx, n),
                                    StepEnd{end, n, ctx->d_hdr[set], ctx->d_ctl});
    for (PopHost* p : ctx->pops) p->acc_valid = true;
}

// The step header of every population: N(i) individuals.
template <class F>
int put_header(clotho_ctx* ctx, F N) {
    uint32_t slot;
    uint32_t* h = hdr_stage(ctx, &slot);
    if (!h) return fail(ctx, CLOTHO_E_NOMEM, "pinned host memory refused");
    for (size_t i = 0; i < ctx->pops.size(); ++i) {
        h[2 * i] = N(i);
        h[2 * i + 1] = 0;
    }
    return hdr_copy(ctx, slot, ctx->d_hdr[2], (uint32_t)ctx->pops.size(), ctx->stream);
}

// Captures n fused device-drawn generations.  Whatever fails between the start of the capture and the graph's
// instantiation, the capture is ended and the partial graph discarded, so the stream stays usable.
int capture_generations(clotho_ctx* ctx, uint32_t n, StepEnd::Mode end, cudaGraphExec_t* exec) {
    CK(cudaStreamSynchronize(ctx->stream));
    CK(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
    const uint64_t l0 = ctx->launches;
    for (uint32_t k = 0; k < n; ++k) enqueue_fused_step(ctx, 2, true, end);
    ctx->graph_launches = (ctx->launches - l0) / n;
    ctx->launches = l0;
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess && ctx->launch_err != cudaSuccess) e = ctx->launch_err;
    ctx->launch_err = cudaSuccess;
    cudaGraph_t gr = nullptr;
    const cudaError_t e_end = cudaStreamEndCapture(ctx->stream, &gr);  // ends the capture in every case
    if (e == cudaSuccess) e = e_end;
    if (e == cudaSuccess) e = cudaGraphInstantiate(exec, gr, 0);
    if (gr) cudaGraphDestroy(gr);
    if (e != cudaSuccess) {
        *exec = nullptr;
        cudaGetLastError();
        return fail(ctx, CLOTHO_E_CUDA, std::string("graph capture of a generation: ") + cudaGetErrorString(e));
    }
    return 0;
}

// Between two replays of a graph the GPU stands still for about 3 us that the kernels inside a graph do not lose (they
// start as the one before drains): 1,000 individuals 28.4 us a generation in graphs of one, 26.6, 26.1, 25.6 in graphs
// of two, four, eight; 10,000 43.6 and 40.8.  Making a graph of eight takes 0.19 ms, what some 80 generations gain, so
// it is made when nearly as many have been replayed.
constexpr uint32_t kLongGraph = 8, kLongAfter = 64;

// The graphs of the key (the sizes they serve, and the tuning) exist and a step needs nothing before it.
bool graph_ready(const clotho_ctx* ctx, std::vector<uint32_t> key) {
    key.push_back(ctx->tuning_epoch);
    bool ready = ctx->graph && ctx->graph_key == key;
    for (const PopHost* p : ctx->pops) ready = ready && p->acc_valid;
    return ready;
}

// Replays count device-drawn generations, capturing what is missing.
int replay_generations(clotho_ctx* ctx, std::vector<uint32_t> key, uint32_t count, StepEnd::Mode end) {
    if (int rc = block_tables(ctx)) return rc;
    key.push_back(ctx->tuning_epoch);
    if (!ctx->graph || ctx->graph_key != key) {
        drop_graphs(ctx);
        if (int rc = capture_generations(ctx, 1, end, &ctx->graph)) return rc;
        ctx->graph_key = key;
    }
    ctx->replayed += count;
    if (!ctx->graph_long && ctx->replayed >= kLongAfter && count >= kLongGraph)
        if (int rc = capture_generations(ctx, kLongGraph, end, &ctx->graph_long)) return rc;
    ctx->pairs_set = 0u;
    ctx->drawn = true;
    sizes_open(ctx);
    while (count) {
        const bool many = ctx->graph_long && count >= kLongGraph;
        CK(cudaGraphLaunch(many ? ctx->graph_long : ctx->graph, ctx->stream));
        ctx->launches += (many ? kLongGraph : 1u) * ctx->graph_launches;
        count -= many ? kLongGraph : 1u;
    }
    return 0;
}

}  // namespace

// ===========================================================================
extern "C" {

size_t clotho_footprint_for(const clotho_desc* d) {
    if (!d) return 0;
    size_t t = 0;
    for (size_t s : sizes_of(geometry(*d))) t += align256(s);
    return t;
}

int clotho_create(const clotho_desc* desc, clotho_ctx** out) {
    if (!desc || !out) return CLOTHO_E_ARG;
    *out = nullptr;
    clotho_ctx* ctx = new clotho_ctx();
    cudaError_t e = cudaGetDevice(&ctx->device);
    if (e != cudaSuccess) {
        delete ctx;
        return CLOTHO_E_CUDA;
    }
    cudaDeviceGetAttribute(&ctx->num_sms, cudaDevAttrMultiProcessorCount, ctx->device);
    if (init_recip_prep() || init_recip_gen()) {  // constant tables of this device
        cudaGetLastError();
        delete ctx;
        return CLOTHO_E_CUDA;
    }
    if (cudaStreamCreateWithFlags(&ctx->own_stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaStreamCreateWithFlags(&ctx->copy_stream, cudaStreamNonBlocking) != cudaSuccess) {
        cudaGetLastError();
        clotho_destroy(ctx);  // releases whichever stream was made
        return CLOTHO_E_CUDA;
    }
    ctx->stream = ctx->own_stream;
    {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = ctx->device;
        if (cudaMemPoolCreate(&ctx->pool, &props) != cudaSuccess) {
            cudaGetLastError();
            ctx->pool = nullptr;
            clotho_destroy(ctx);
            return CLOTHO_E_CUDA;
        }
        // freed blocks stay in the pool until the context ends; if the attribute is refused, the pool
        // returns memory at each synchronization instead, which is slower, not wrong
        uint64_t keep = ~0ull;
        if (cudaMemPoolSetAttribute(ctx->pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess)
            cudaGetLastError();
    }
    {
        bool ok = true;
        for (int i = 0; i < 2; ++i) {
            ok = ok && cudaEventCreateWithFlags(&ctx->copy_done[i], cudaEventDisableTiming) == cudaSuccess;
            ok = ok && cudaEventCreateWithFlags(&ctx->kern_done[i], cudaEventDisableTiming) == cudaSuccess;
            ok = ok && cudaEventRecord(ctx->kern_done[i], ctx->stream) == cudaSuccess;
        }
        ok = ok && cudaEventCreate(&ctx->t0) == cudaSuccess && cudaEventCreate(&ctx->t1) == cudaSuccess;
        if (!ok) {
            cudaGetLastError();
            clotho_destroy(ctx);
            return CLOTHO_E_CUDA;
        }
    }
    if (cudaMalloc(&ctx->d_ctl, sizeof(WorkCtl)) != cudaSuccess) {
        cudaGetLastError();
        clotho_destroy(ctx);
        return CLOTHO_E_NOMEM;
    }
    {
        const uint32_t rpi = kRowsPerItem;
        if (cudaMemsetAsync(ctx->d_ctl, 0, sizeof(WorkCtl), ctx->stream) != cudaSuccess ||
            cudaMemcpyAsync(&ctx->d_ctl->rows_per_item, &rpi, 4, cudaMemcpyHostToDevice, ctx->stream) != cudaSuccess ||
            cudaStreamSynchronize(ctx->stream) != cudaSuccess) {
            cudaGetLastError();
            clotho_destroy(ctx);
            return CLOTHO_E_CUDA;
        }
    }
    PopHost* p = nullptr;
    int rc = alloc_pop(ctx, *desc, &p);
    if (rc) {
        std::string m = ctx->err;
        clotho_destroy(ctx);
        fprintf(stderr, "clotho_create: %s\n", m.c_str());
        return rc;
    }
    ctx->pops.push_back(p);
    rc = sync_pop_arrays(ctx);
    if (rc) {
        clotho_destroy(ctx);
        return rc;
    }
    *out = ctx;
    return 0;
}

int clotho_destroy(clotho_ctx* ctx) {
    if (!ctx) return CLOTHO_E_ARG;
    if (ctx->stream) cudaStreamSynchronize(ctx->stream);
    if (ctx->copy_stream) cudaStreamSynchronize(ctx->copy_stream);
    for (PopHost* p : ctx->pops) free_pop(ctx, p);
    ctx->pops.clear();
    ctx->parts_kept.push_back(ctx->d_parts);
    for (BlockPart* t : ctx->parts_kept)
        if (t) cudaFreeAsync(t, ctx->own_stream);
    if (ctx->own_stream) cudaStreamSynchronize(ctx->own_stream);
    if (ctx->pool) cudaMemPoolDestroy(ctx->pool);  // its blocks are back: free_pop returned them
    for (int s = 0; s < 3; ++s) {
        if (ctx->d_pops[s]) cudaFree(ctx->d_pops[s]);
        if (ctx->d_hdr[s]) cudaFree(ctx->d_hdr[s]);
    }
    if (ctx->h_ring) cudaFreeHost(ctx->h_ring);
    for (char* h : ctx->h_tape)
        if (h) cudaFreeHost(h);
    if (ctx->h_stat) cudaFreeHost(ctx->h_stat);
    for (uint32_t k = 0; k < kStatRing; ++k)
        if (ctx->stat_ev[k]) cudaEventDestroy(ctx->stat_ev[k]);
    for (uint32_t k = 0; k < kHdrRing; ++k)
        if (ctx->ring_ev[k]) cudaEventDestroy(ctx->ring_ev[k]);
    if (ctx->d_ctl) cudaFree(ctx->d_ctl);
    drop_graphs(ctx);
    for (cudaEvent_t e : ctx->prof_ev) cudaEventDestroy(e);
    for (int i = 0; i < 2; ++i) {
        if (ctx->copy_done[i]) cudaEventDestroy(ctx->copy_done[i]);
        if (ctx->kern_done[i]) cudaEventDestroy(ctx->kern_done[i]);
    }
    if (ctx->t0) cudaEventDestroy(ctx->t0);
    if (ctx->t1) cudaEventDestroy(ctx->t1);
    if (ctx->own_stream) cudaStreamDestroy(ctx->own_stream);
    if (ctx->copy_stream) cudaStreamDestroy(ctx->copy_stream);
    delete ctx;
    return 0;
}

const char* clotho_last_error(const clotho_ctx* ctx) { return ctx ? ctx->err.c_str() : "null context"; }

size_t clotho_footprint(const clotho_ctx* ctx) {
    size_t t = 0;
    if (ctx)
        for (PopHost* p : ctx->pops) t += p->bytes;
    return t;
}

int clotho_sync(clotho_ctx* ctx) {
    if (!ctx) return CLOTHO_E_ARG;
    CK(cudaStreamSynchronize(ctx->copy_stream));
    CK(cudaStreamSynchronize(ctx->stream));
    return 0;
}

int clotho_set_stream(clotho_ctx* ctx, void* stream) {
    if (!ctx) return CLOTHO_E_ARG;
    if (ctx->in_step) return fail(ctx, CLOTHO_E_STATE, "set the stream between generations");
    // work already queued on the old stream finishes before the new one is used
    CK(cudaStreamSynchronize(ctx->copy_stream));
    CK(cudaStreamSynchronize(ctx->stream));
    ctx->stream = stream ? static_cast<cudaStream_t>(stream) : ctx->own_stream;
    return 0;
}

uint64_t clotho_launch_count(const clotho_ctx* ctx) { return ctx ? ctx->launches : 0; }

static int init_pop(clotho_ctx* ctx, uint32_t idx, uint32_t N0) {
    if (!ctx || idx >= ctx->pops.size()) return fail(ctx, CLOTHO_E_ARG, "no such population");
    PopHost* p = ctx->pops[idx];
    const PopDev& D = p->dev[0];
    if (N0 > D.Ncap) return fail(ctx, CLOTHO_E_CAPACITY, "N0 exceeds max_individuals");
    CK(cudaStreamSynchronize(ctx->stream));
    p->n_known = false;
    DevStatus s{};
    s.gen = 1;
    s.cur = 0;
    s.N = N0;
    s.count_cols = p->counting ? 1u : 0u;
    s.fit_const = 1;
    s.fit_total = (double)N0;
    s.all_neutral = 1;
    CK(cudaMemcpyAsync(D.st, &s, sizeof(s), cudaMemcpyHostToDevice, ctx->stream));
    std::vector<double> ones(N0, 1.0);
    if (N0) CK(cudaMemcpyAsync(D.fit, ones.data(), N0 * sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemsetAsync(D.pos, 0, (size_t)D.Acap * 8, ctx->stream));
    CK(cudaMemsetAsync(D.eff, 0, (size_t)D.Acap * 16, ctx->stream));
    CK(cudaMemsetAsync(D.age, 0, (size_t)D.Acap * 4, ctx->stream));
    CK(cudaMemsetAsync(D.accF, 0xff, (size_t)D.Wcap * 8, ctx->stream));
    CK(cudaMemsetAsync(D.accV, 0, (size_t)D.Wcap * 8, ctx->stream));
    CK(cudaMemsetAsync(D.row_cnt, 0, ((size_t)D.Scap + 1) * 4, ctx->stream));
    CK(cudaMemsetAsync(D.row_cur, 0, (size_t)D.Scap * 4, ctx->stream));
    CK(cudaMemsetAsync(D.bcnt, 0, ((size_t)D.NB + 1) * 4, ctx->stream));
    CK(cudaMemsetAsync(D.bcur, 0, (size_t)D.NB * 4, ctx->stream));
    CK(cudaMemsetAsync(D.zg[0], 0, (size_t)D.Scap * 32, ctx->stream));
    CK(cudaMemsetAsync(D.zg[1], 0, (size_t)D.Scap * 32, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    p->acc_valid = true;  // A == 0: the first analysis is skipped (free_space_mt...:46)
    p->ready = true;
    p->hostN = N0;
    p->n_known = !ctx->captured;
    return 0;
}

int clotho_init(clotho_ctx* ctx, uint32_t N0) { return init_pop(ctx, 0, N0); }

// Shared set-up of an explicit or seeded start: status, allele tables, then
// (after the caller fills the rows) reduction, phenotype and fitness.
static int start_population(clotho_ctx* ctx, uint32_t N, uint32_t A, const double* pos, const float* eff) {
    int rc = require_pop(ctx);
    if (rc) return rc;
    PopHost* p = ctx->pops[0];
    const PopDev& D = p->dev[0];
    if (A > D.Acap || ref_width(A) > D.Wcap) return fail(ctx, CLOTHO_E_CAPACITY, "A exceeds max_alleles");
    if ((rc = clotho_init(ctx, N))) return rc;
    const uint32_t T = D.T;
    int32_t nz = 0;
    for (size_t i = 0; i < (size_t)A * T; ++i) nz += (eff[i] != 0.0f);
    DevStatus s{};
    s.gen = 1;
    s.cur = 0;
    s.N = N;
    s.A = A;
    s.count_cols = p->counting ? 1u : 0u;
    s.W = ref_width(A);
    s.nz_eff = nz;
    s.fit_const = 1;
    s.fit_total = (double)N;
    CK(cudaMemcpyAsync(D.st, &s, sizeof(s), cudaMemcpyHostToDevice, ctx->stream));
    if (A) {
        CK(cudaMemcpyAsync(D.pos, pos, (size_t)A * 8, cudaMemcpyHostToDevice, ctx->stream));
        std::vector<float> pad((size_t)A * 4, 0.0f);
        for (size_t i = 0; i < A; ++i)
            for (uint32_t t = 0; t < T; ++t) pad[i * 4 + t] = eff[i * T + t];
        CK(cudaMemcpyAsync(D.eff, pad.data(), (size_t)A * 16, cudaMemcpyHostToDevice, ctx->stream));
        CK(cudaStreamSynchronize(ctx->stream));
    }
    return 0;
}

static int finish_start(clotho_ctx* ctx) {
    PopHost* p = ctx->pops[0];
    LaunchCfg L = cfg(ctx);
    launch_fs_reduce(L, ctx->d_pops[0], 1, ctx->maxW, 0u);
    launch_phenotype(L, ctx->d_pops[0], 1);
    ctx->launches += 2 + launch_fitness(L, ctx->d_pops[0], 1, ctx->maxN, constant_fitness(ctx, 1), StepEnd{});
    int rc = check_launch(ctx, "start");
    if (rc) return rc;
    CK(cudaStreamSynchronize(ctx->stream));
    p->acc_valid = true;
    return 0;
}

int clotho_load_population(clotho_ctx* ctx, uint32_t N, uint32_t A, const uint64_t* rows, const double* pos,
                           const float* eff) {
    if (!ctx || (A && (!pos || !eff || !rows))) return CLOTHO_E_ARG;
    int rc = start_population(ctx, N, A, pos, eff);
    if (rc) return rc;
    const PopDev& D = ctx->pops[0]->dev[0];
    const size_t W = ref_width(A), S = 2ull * N;
    if (S * W) {
        // keep only slots < A (the reference never sets bits past its allele count)
        std::vector<uint64_t> tmp(rows, rows + S * W);
        for (size_t r = 0; r < S; ++r)
            for (size_t w = 0; w < W; ++w) {
                const size_t b = w * 64;
                uint64_t valid = (b + 64 <= A) ? ~0ull : (b >= A ? 0ull : ((1ull << (A - b)) - 1ull));
                tmp[r * W + w] &= valid;
            }
        CK(cudaMemcpy2DAsync(D.rows[0], (size_t)D.Wcap * 8, tmp.data(), W * 8, W * 8, S, cudaMemcpyHostToDevice,
                             ctx->stream));
        CK(cudaStreamSynchronize(ctx->stream));
    }
    return finish_start(ctx);
}

int clotho_seed_population(clotho_ctx* ctx, uint32_t N, uint32_t A, const double* pos, const float* eff,
                           const uint32_t* thr, uint64_t seed) {
    if (!ctx || (A && (!pos || !eff || !thr))) return CLOTHO_E_ARG;
    {
        int rc0 = start_population(ctx, N, A, pos, eff);
        if (rc0) return rc0;
        uint32_t* d_thr = nullptr;
        CK(pool_alloc(ctx, &d_thr, std::max<size_t>(4, (size_t)A * 4)));
        if (A) CK(cudaMemcpyAsync(d_thr, thr, (size_t)A * 4, cudaMemcpyHostToDevice, ctx->stream));
        launch_seed_rows(cfg(ctx), ctx->d_pops[0], 0, d_thr, seed, A);
        ctx->launches += 1;
        CK(cudaFreeAsync(d_thr, ctx->stream));
        CK(cudaStreamSynchronize(ctx->stream));
        return finish_start(ctx);
    }
}

int clotho_generation_tape(clotho_ctx* ctx, const clotho_gen_tape* tape) {
    int rc = require_ready(ctx);
    if (rc) return rc;
    if (!tape || ctx->pops.size() != 1) return fail(ctx, CLOTHO_E_ARG, "bad tape");
    if (ctx->in_step) return fail(ctx, CLOTHO_E_STATE, "a staged generation is in progress");
    // a replay would read what the pinned block holds by then
    if (capturing(ctx)) return fail(ctx, CLOTHO_E_STATE, "a tape cannot be captured in a graph");
    const uint32_t s = ctx->set;
    TapeArray arr[7];
    if ((rc = tape_arrays(ctx, ctx->pops[0], s, tape, arr))) return rc;
    size_t total = 0;
    for (const TapeArray& a : arr) total += (a.bytes + 15) & ~(size_t)15;
    if (total <= kTapeStage && !ctx->h_tape[s] && cudaMallocHost(&ctx->h_tape[s], kTapeStage) != cudaSuccess) {
        cudaGetLastError();
        ctx->h_tape[s] = nullptr;
    }
    const bool staged = total <= kTapeStage && ctx->h_tape[s];
    if (staged) {
        // the block was last read by the step two steps ago; the device arrays are the stream's own
        CK(cudaEventSynchronize(ctx->kern_done[s]));
        TapePieces z{};
        size_t off = 0;
        for (int i = 0; i < 7; ++i) {
            if (arr[i].bytes) std::memcpy(ctx->h_tape[s] + off, arr[i].src, arr[i].bytes);
            z.src[i] = ctx->h_tape[s] + off;
            z.dst[i] = arr[i].dst;
            off += (arr[i].bytes + 15) & ~(size_t)15;
            z.end[i] = (uint32_t)(off / 16);
        }
        z.N = tape->N;
        z.M = tape->M;
        launch_tape_upload(cfg(ctx, s), z, ctx->d_hdr[s]);
        ctx->launches += 1;
    } else {
        // the tape set s was last read by the kernels of two steps ago, set 0 by any device-drawn steps since
        if (s == 0u && (ctx->drawn || ctx->captured)) CK(cudaEventRecord(ctx->kern_done[0], ctx->stream));
        CK(cudaStreamWaitEvent(ctx->copy_stream, ctx->kern_done[s], 0));
        for (const TapeArray& a : arr)
            if (a.bytes) CK(cudaMemcpyAsync(a.dst, a.src, a.bytes, cudaMemcpyHostToDevice, ctx->copy_stream));
        uint32_t slot;
        uint32_t* h = hdr_stage(ctx, &slot);
        if (!h) return fail(ctx, CLOTHO_E_NOMEM, "pinned host memory refused");
        h[0] = tape->N;
        h[1] = tape->M;
        if ((rc = hdr_copy(ctx, slot, ctx->d_hdr[s], 1, ctx->copy_stream))) return rc;
        CK(cudaEventRecord(ctx->copy_done[s], ctx->copy_stream));
        CK(cudaStreamWaitEvent(ctx->stream, ctx->copy_done[s], 0));
    }
    enqueue_fused_step(ctx, s, false);
    // recorded also when a launch was refused: those before it still read the tape
    CK(cudaEventRecord(ctx->kern_done[s], ctx->stream));
    if (s == 0u) ctx->drawn = false;
    // the caller's host arrays are free once the copies are done
    if (!staged) CK(cudaEventSynchronize(ctx->copy_done[s]));
    if ((rc = check_launch(ctx, "generation_tape"))) return rc;
    ctx->set ^= 1u;
    sizes_are(ctx, [tape](size_t) { return tape->N; });
    return 0;
}

int clotho_generation_philox(clotho_ctx* ctx, uint32_t N) {
    int rc = require_ready(ctx);
    if (rc) return rc;
    if ((rc = require_pop(ctx))) return rc;
    if ((rc = block_tables(ctx))) return rc;
    if (ctx->in_step) return fail(ctx, CLOTHO_E_STATE, "a staged generation is in progress");
    for (size_t i = 0; i < ctx->pops.size(); ++i)
        if (N > ctx->pops[i]->dev[2].Ncap) return fail(ctx, CLOTHO_E_CAPACITY, "N exceeds max_individuals");
    if ((rc = put_header(ctx, [N](size_t) { return N; }))) return rc;
    enqueue_fused_step(ctx, 2, true);
    if ((rc = check_launch(ctx, "generation_philox"))) return rc;
    sizes_are(ctx, [N](size_t) { return N; });
    return 0;
}

int clotho_run_philox(clotho_ctx* ctx, uint32_t N, uint32_t G) {
    int rc = require_ready(ctx);
    if (rc) return rc;
    if (ctx->in_step) return fail(ctx, CLOTHO_E_STATE, "a staged generation is in progress");
    if (G == 0) return 0;
    if ((rc = require_pop(ctx))) return rc;
    for (const PopHost* p : ctx->pops)
        if (N > p->dev[2].Ncap) return fail(ctx, CLOTHO_E_CAPACITY, "N exceeds max_individuals");
    const std::vector<uint32_t> key(ctx->pops.size(), N);
    uint32_t left = G;
    if (!ctx->profiling && graph_ready(ctx, key)) {
        if ((rc = put_header(ctx, [N](size_t) { return N; }))) return rc;
    } else {
        // the first generation runs eagerly (it may need the parent reduction)
        if ((rc = clotho_generation_philox(ctx, N))) return rc;
        left -= 1;
    }
    if (ctx->profiling) {  // per-launch events are taken from eager launches
        for (; left; --left)
            if ((rc = clotho_generation_philox(ctx, N))) return rc;
        return 0;
    }
    if (left && (rc = replay_generations(ctx, key, left, StepEnd::kStep))) return rc;
    sizes_are(ctx, [N](size_t) { return N; });
    return 0;
}

// ---- staged entry points -------------------------------------------------
int clotho_begin_generation(clotho_ctx* ctx, uint32_t N, uint32_t M) {
    int rc = require_ready(ctx);
    if (rc) return rc;
    if ((rc = require_pop(ctx))) return rc;
    if (ctx->in_step) return fail(ctx, CLOTHO_E_STATE, "generation already begun");
    PopHost* p = ctx->pops[0];
    if (N > p->dev[0].Ncap) return fail(ctx, CLOTHO_E_CAPACITY, "N exceeds max_individuals");
    if (M > p->dev[0].Mcap) return fail(ctx, CLOTHO_E_CAPACITY, "M exceeds max_mutations");
    CK(cudaStreamSynchronize(ctx->copy_stream));
    uint32_t slot;
    uint32_t* h = hdr_stage(ctx, &slot);
    if (!h) return fail(ctx, CLOTHO_E_NOMEM, "pinned host memory refused");
    h[0] = N;
    h[1] = M;
    if ((rc = hdr_copy(ctx, slot, ctx->d_hdr[0], 1, ctx->stream))) return rc;
    launch_begin(cfg(ctx), ctx->d_pops[0], 1, ctx->d_hdr[0], ctx->d_ctl);
    ctx->launches += 1;
    ctx->in_step = true;
    p->hostN = N;
    rc = check_launch(ctx, "begin");
    p->n_known = rc == 0 && !ctx->captured;
    return rc;
}

int clotho_free_space(clotho_ctx* ctx, uint32_t* counts) {
    if (!ctx || !ctx->in_step) return fail(ctx, CLOTHO_E_STATE, "clotho_begin_generation first");
    PopHost* p = ctx->pops[0];
    if (!p->acc_valid) {
        launch_fs_reduce(cfg(ctx), ctx->d_pops[0], 1, ctx->maxW, 1u);
        ctx->launches += 1;
    }
    launch_fs_finalize(cfg(ctx), ctx->d_pops[0], 1);
    ctx->launches += 1;
    p->acc_valid = false;  // reset for the child; the staged crossover does not refill it
    int rc = check_launch(ctx, "free_space");
    if (rc) return rc;
    if (counts) {
        DevStatus s = read_status(ctx, p, &rc);
        if (rc) return rc;
        counts[0] = s.fixed_cnt;
        counts[1] = s.lost_cnt;
        counts[2] = s.free_cnt;
    }
    return 0;
}

int clotho_set_pairs(clotho_ctx* ctx, const uint32_t* pairs) {
    if (!ctx || !ctx->in_step) return fail(ctx, CLOTHO_E_STATE, "clotho_begin_generation first");
    PopHost* p = ctx->pops[0];
    int rc = h2d(ctx, p->dev[0].pairs, pairs, 2ull * p->hostN, ctx->stream);
    ctx->pairs_set = 0;
    if (rc) return rc;
    CK(cudaStreamSynchronize(ctx->stream));
    return 0;
}

int clotho_select(clotho_ctx* ctx, uint32_t* pairs_out) {
    if (!ctx || !ctx->in_step) return fail(ctx, CLOTHO_E_STATE, "clotho_begin_generation first");
    PopHost* p = ctx->pops[0];
    // device draws write the pairs of the Philox set, which shares buffers with set 0
    launch_select_philox(cfg(ctx), ctx->d_pops[2], 1);
    ctx->launches += 1;
    ctx->pairs_set = 0;
    int rc = check_launch(ctx, "select");
    if (rc) return rc;
    if (pairs_out) {
        CK(cudaMemcpyAsync(pairs_out, p->dev[2].pairs, 2ull * p->hostN * 4, cudaMemcpyDeviceToHost, ctx->stream));
        CK(cudaStreamSynchronize(ctx->stream));
    }
    return 0;
}

int clotho_crossover(clotho_ctx* ctx, const uint8_t* swap, const uint32_t* ev_off, const double* ev_pos) {
    if (!ctx || !ctx->in_step) return fail(ctx, CLOTHO_E_STATE, "clotho_begin_generation first");
    PopHost* p = ctx->pops[0];
    const PopDev& D = p->dev[0];
    const uint32_t N = p->hostN;
    if (!ev_off) return fail(ctx, CLOTHO_E_ARG, "ev_off is null");
    const uint32_t ev_total = ev_off[2ull * N];
    if (ev_total > D.EVcap) return fail(ctx, CLOTHO_E_CAPACITY, "events exceed max_events");
    int rc;
    if ((rc = h2d(ctx, D.swap, swap, 2ull * N, ctx->stream))) return rc;
    if ((rc = h2d(ctx, D.ev_off, ev_off, 2ull * N + 1, ctx->stream))) return rc;
    if ((rc = h2d(ctx, D.ev_pos, ev_pos, (size_t)ev_total, ctx->stream))) return rc;
    // item prefix is already set by begin; the rows' order, ranks over the current positions
    const PrepSizes z = prep_sizes(ctx);
    ctx->launches += launch_prep(cfg(ctx), ctx->d_pops[0], 1, z, nullptr, ctx->d_ctl, kStepOrder, false);
    ctx->launches += launch_plan(cfg(ctx), ctx->d_pops[0], 1, z, ctx->maxW, kStepOrder);
    launch_gen(ctx, cfg(ctx), ctx->d_pops[0], 1, 0u);
    if ((rc = check_launch(ctx, "crossover"))) return rc;
    CK(cudaStreamSynchronize(ctx->stream));
    return 0;
}

int clotho_mutate(clotho_ctx* ctx, const uint32_t* mut_seq, const double* mut_pos, const float* mut_eff) {
    if (!ctx || !ctx->in_step) return fail(ctx, CLOTHO_E_STATE, "clotho_begin_generation first");
    PopHost* p = ctx->pops[0];
    const PopDev& D = p->dev[0];
    int rc;
    DevStatus s = read_status(ctx, p, &rc);
    if (rc) return rc;
    const uint32_t M = s.M;
    if ((rc = h2d(ctx, D.mut_seq, mut_seq, (size_t)M, ctx->stream))) return rc;
    if ((rc = h2d(ctx, D.mut_pos, mut_pos, (size_t)M, ctx->stream))) return rc;
    if ((rc = h2d(ctx, D.mut_eff, mut_eff, (size_t)M * D.T, ctx->stream))) return rc;
    launch_mut_resolve(cfg(ctx), ctx->d_pops[0], 1);
    launch_mut_scatter(cfg(ctx), ctx->d_pops[0], 1);
    ctx->launches += 2;
    if ((rc = check_launch(ctx, "mutate"))) return rc;
    CK(cudaStreamSynchronize(ctx->stream));
    return 0;
}

int clotho_phenotype(clotho_ctx* ctx) {
    if (int rc = require_pop(ctx)) return rc;
    launch_phenotype(cfg(ctx), ctx->d_pops[0], 1);
    ctx->launches += 1;
    return check_launch(ctx, "phenotype");
}

int clotho_fitness(clotho_ctx* ctx) {
    if (int rc = require_pop(ctx)) return rc;
    ctx->launches += launch_fitness(cfg(ctx), ctx->d_pops[0], 1, ctx->maxN, constant_fitness(ctx, 1), StepEnd{});
    return check_launch(ctx, "fitness");
}

int clotho_end_generation(clotho_ctx* ctx) {
    if (!ctx || !ctx->in_step) return fail(ctx, CLOTHO_E_STATE, "no generation in progress");
    launch_end(cfg(ctx), ctx->d_pops[0], 1);
    ctx->launches += 1;
    ctx->in_step = false;
    int rc = check_launch(ctx, "end");
    if (rc) return rc;
    CK(cudaStreamSynchronize(ctx->stream));
    return 0;
}

// ---- read-back -------------------------------------------------------------
static int info_of(clotho_ctx* ctx, uint32_t idx, clotho_info* out) {
    if (!ctx || !out || idx >= ctx->pops.size()) return fail(ctx, CLOTHO_E_ARG, "no such population");
    CK(cudaStreamSynchronize(ctx->copy_stream));
    int rc;
    DevStatus s = read_status(ctx, ctx->pops[idx], &rc);
    if (rc) return rc;
    out->generation = s.gen;
    out->N = s.N;
    out->A = s.A;
    out->W = s.W;
    out->fixed_count = s.fixed_cnt;
    out->lost_count = s.lost_cnt;
    out->free_count = s.free_cnt;
    out->variable_count = (s.pA > s.free_cnt ? s.pA - s.free_cnt : 0);
    out->fixed_total = s.fixed_total;
    out->last_M = s.last_M;
    out->all_neutral = s.all_neutral;
    out->device_error = s.err;
    out->mean_fitness = s.N ? s.fit_total / (double)s.N : 0.0;
    return 0;
}

int clotho_get_info(clotho_ctx* ctx, clotho_info* out) { return info_of(ctx, 0, out); }

static void info_from_status(const DevStatus& s, clotho_info* out) {
    out->generation = s.gen;
    out->N = s.N;
    out->A = s.A;
    out->W = s.W;
    out->fixed_count = s.fixed_cnt;
    out->lost_count = s.lost_cnt;
    out->free_count = s.free_cnt;
    out->variable_count = (s.pA > s.free_cnt ? s.pA - s.free_cnt : 0);
    out->fixed_total = s.fixed_total;
    out->last_M = s.last_M;
    out->all_neutral = s.all_neutral;
    out->device_error = s.err;
    out->mean_fitness = s.N ? s.fit_total / (double)s.N : 0.0;
}


// The status copy is ordered behind everything issued so far on the context's stream; the host
// thread goes on issuing work and collects the copy with clotho_info_wait.
static int info_request(clotho_ctx* ctx, uint32_t idx, uint32_t* ticket) {
    if (!ctx || !ticket || idx >= ctx->pops.size()) return fail(ctx, CLOTHO_E_ARG, "no such population");
    if (!ctx->h_stat) {
        if (cudaMallocHost(&ctx->h_stat, sizeof(DevStatus) * kStatRing) != cudaSuccess) {
            cudaGetLastError();
            ctx->h_stat = nullptr;
            return fail(ctx, CLOTHO_E_NOMEM, "pinned host memory refused");
        }
        for (uint32_t k = 0; k < kStatRing; ++k) CK(cudaEventCreateWithFlags(&ctx->stat_ev[k], cudaEventDisableTiming));
    }
    const uint32_t t = ctx->stat_next;
    const uint32_t k = t % kStatRing;
    if (t >= kStatRing) CK(cudaEventSynchronize(ctx->stat_ev[k]));  // the slot's previous copy has landed
    CK(cudaMemcpyAsync(&ctx->h_stat[k], ctx->pops[idx]->dev[0].st, sizeof(DevStatus), cudaMemcpyDeviceToHost,
                       ctx->stream));
    CK(cudaEventRecord(ctx->stat_ev[k], ctx->stream));
    ctx->stat_next = t + 1;
    *ticket = t;
    return 0;
}

static int info_wait(clotho_ctx* ctx, uint32_t ticket, clotho_info* out) {
    if (!ctx || !out) return CLOTHO_E_ARG;
    if (ticket >= ctx->stat_next || ctx->stat_next - ticket > kStatRing)
        return fail(ctx, CLOTHO_E_ARG, "unknown or overwritten info ticket");
    const uint32_t k = ticket % kStatRing;
    CK(cudaEventSynchronize(ctx->stat_ev[k]));
    info_from_status(ctx->h_stat[k], out);
    return 0;
}

int clotho_info_request(clotho_ctx* ctx, uint32_t* ticket) { return info_request(ctx, 0, ticket); }
int clotho_pop_info_request(clotho_ctx* ctx, uint32_t index, uint32_t* ticket) {
    return info_request(ctx, index, ticket);
}
int clotho_info_wait(clotho_ctx* ctx, uint32_t ticket, clotho_info* out) { return info_wait(ctx, ticket, out); }

static int rows_of(clotho_ctx* ctx, uint32_t idx, uint64_t* dst, size_t dst_words) {
    if (!ctx || idx >= ctx->pops.size()) return fail(ctx, CLOTHO_E_ARG, "no such population");
    int rc;
    PopHost* p = ctx->pops[idx];
    DevStatus s = read_status(ctx, p, &rc);
    if (rc) return rc;
    const size_t S = 2ull * s.N, W = s.W;
    if (S * W == 0) return 0;
    if (!dst || dst_words < S * W) return fail(ctx, CLOTHO_E_ARG, "destination too small");
    host_pages(dst, S * W * 8);
    CK(cudaMemcpy2DAsync(dst, W * 8, p->dev[0].rows[s.cur], (size_t)p->dev[0].Wcap * 8, W * 8, S,
                         cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    return 0;
}

int clotho_get_rows(clotho_ctx* ctx, uint64_t* dst, size_t dst_words) { return rows_of(ctx, 0, dst, dst_words); }

int clotho_get_alleles(clotho_ctx* ctx, double* pos, uint32_t* age, float* eff) {
    int rc = require_pop(ctx);
    if (rc) return rc;
    PopHost* p = ctx->pops[0];
    DevStatus s = read_status(ctx, p, &rc);
    if (rc) return rc;
    const PopDev& D = p->dev[0];
    if (pos && s.A) CK(cudaMemcpyAsync(pos, D.pos, (size_t)s.A * 8, cudaMemcpyDeviceToHost, ctx->stream));
    if (age && s.A) CK(cudaMemcpyAsync(age, D.age, (size_t)s.A * 4, cudaMemcpyDeviceToHost, ctx->stream));
    std::vector<float> pad((size_t)s.A * 4);
    if (eff && s.A) CK(cudaMemcpyAsync(pad.data(), D.eff, (size_t)s.A * 16, cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    if (eff)
        for (size_t i = 0; i < s.A; ++i)
            for (uint32_t t = 0; t < D.T; ++t) eff[i * D.T + t] = pad[i * 4 + t];
    return 0;
}

int clotho_get_fixed(clotho_ctx* ctx, double* pos, uint32_t* age, float* eff) {
    int rc = require_pop(ctx);
    if (rc) return rc;
    PopHost* p = ctx->pops[0];
    DevStatus s = read_status(ctx, p, &rc);
    if (rc) return rc;
    const PopDev& D = p->dev[0];
    const size_t F = s.fixed_total;
    if (pos && F) CK(cudaMemcpyAsync(pos, D.fx_pos, F * 8, cudaMemcpyDeviceToHost, ctx->stream));
    if (age && F) CK(cudaMemcpyAsync(age, D.fx_age, F * 4, cudaMemcpyDeviceToHost, ctx->stream));
    if (eff && F) CK(cudaMemcpyAsync(eff, D.fx_eff, F * D.T * 4, cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    return 0;
}

int clotho_get_free(clotho_ctx* ctx, uint32_t* dst) {
    int rc = require_pop(ctx);
    if (rc) return rc;
    PopHost* p = ctx->pops[0];
    DevStatus s = read_status(ctx, p, &rc);
    if (rc) return rc;
    if (s.free_cnt && !dst) return fail(ctx, CLOTHO_E_ARG, "null destination");
    if (s.free_cnt)
        CK(cudaMemcpyAsync(dst, p->dev[0].free_list, (size_t)s.free_cnt * 4, cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    return 0;
}

// n rows of T of four doubles: four are the caller's layout, fewer are packed on the device first.
static int get_double4(clotho_ctx* ctx, const double* src, size_t n, double* dst) {
    const uint32_t T = ctx->pops[0]->dev[0].T;
    if (n == 0) return 0;
    host_pages(dst, n * T * 8);
    if (T == 4) {
        CK(cudaMemcpyAsync(dst, src, n * 32, cudaMemcpyDeviceToHost, ctx->stream));
        CK(cudaStreamSynchronize(ctx->stream));
        return 0;
    }
    double* d = nullptr;
    CK(pool_alloc(ctx, &d, n * T * 8));
    launch_pack_traits(cfg(ctx), src, d, (uint32_t)n, T);
    ctx->launches += 1;
    int rc = check_launch(ctx, "pack");
    const cudaError_t e_copy = cudaMemcpyAsync(dst, d, n * T * 8, cudaMemcpyDeviceToHost, ctx->stream);
    const cudaError_t e_free = cudaFreeAsync(d, ctx->stream);
    const cudaError_t e_sync = cudaStreamSynchronize(ctx->stream);
    if (rc) return rc;
    CK(e_copy);
    CK(e_free);
    CK(e_sync);
    return 0;
}

int clotho_get_genome_traits(clotho_ctx* ctx, double* dst) {
    int rc = require_pop(ctx);
    if (rc) return rc;
    DevStatus s = read_status(ctx, ctx->pops[0], &rc);
    if (rc) return rc;
    return get_double4(ctx, ctx->pops[0]->dev[0].zg[s.cur], 2ull * s.N, dst);
}

int clotho_get_phenotypes(clotho_ctx* ctx, double* dst) {
    if (int rc = require_pop(ctx)) return rc;
    int rc;
    const uint32_t N = current_N(ctx, ctx->pops[0], &rc);
    return rc ? rc : get_double4(ctx, ctx->pops[0]->dev[0].zi, N, dst);
}

int clotho_get_fitness(clotho_ctx* ctx, double* dst) {
    if (int rc = require_pop(ctx)) return rc;
    int rc;
    const size_t N = current_N(ctx, ctx->pops[0], &rc);
    if (rc) return rc;
    host_pages(dst, N * 8);
    if (N) CK(cudaMemcpyAsync(dst, ctx->pops[0]->dev[0].fit, N * 8, cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    return 0;
}

int clotho_get_pairs(clotho_ctx* ctx, uint32_t* dst) {
    int rc = require_pop(ctx);
    if (rc) return rc;
    DevStatus s = read_status(ctx, ctx->pops[0], &rc);
    if (rc) return rc;
    // tape steps alternate between sets 0 and 1; device draws and the staged calls use set 0's buffer
    const PopDev& D = ctx->pops[0]->dev[ctx->pairs_set];
    host_pages(dst, 2ull * s.N * 4);
    if (s.N) CK(cudaMemcpyAsync(dst, D.pairs, 2ull * s.N * 4, cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    return 0;
}

static int stats_of(clotho_ctx* ctx, uint32_t idx, clotho_stats* out, uint32_t* sfs, uint32_t sfs_len) {
    if (!ctx || !out || idx >= ctx->pops.size()) return fail(ctx, CLOTHO_E_ARG, "no such population");
    int rc;
    PopHost* p = ctx->pops[idx];
    DevStatus s = read_status(ctx, p, &rc);
    if (rc) return rc;
    const PopDev& D = p->dev[0];
    const uint32_t S = 2 * s.N;
    // one scratch block from the context's pool (stream-ordered, no device-wide synchronisation): the results,
    // the spectrum, and the column counts unless the last fused step counted the columns of these rows
    const size_t head = align256(sizeof(StatsOut)), len = sfs ? sfs_len : 0;
    const size_t spectrum = align256(len * 4), cols = s.cols_valid ? 0 : (size_t)s.W * 256;
    char* d = nullptr;
    CK(pool_alloc(ctx, &d, head + spectrum + cols));
    StatsOut* d_out = reinterpret_cast<StatsOut*>(d);
    uint32_t* d_sfs = reinterpret_cast<uint32_t*>(d + head);
    uint32_t* d_counts = s.cols_valid ? D.colcnt : reinterpret_cast<uint32_t*>(d + head + spectrum);
    std::vector<char> h(head + len * 4);
    auto body = [&]() -> int {
        CK(cudaMemsetAsync(d, 0, head + spectrum + cols, ctx->stream));
        if (cols) {
            launch_margins(cfg(ctx), ctx->d_pops[0], idx, S, s.W, d_counts, nullptr);
            ctx->launches += 1;
        }
        launch_stats(cfg(ctx), ctx->d_pops[0], idx, d_counts, (uint32_t)len, d_out, d_sfs);
        ctx->launches += 1;
        if (int r = check_launch(ctx, "stats")) return r;
        CK(cudaMemcpyAsync(h.data(), d, h.size(), cudaMemcpyDeviceToHost, ctx->stream));
        return 0;
    };
    rc = body();
    const cudaError_t e_free = cudaFreeAsync(d, ctx->stream);
    const cudaError_t e_sync = cudaStreamSynchronize(ctx->stream);
    if (rc) return rc;
    CK(e_free);
    CK(e_sync);
    const StatsOut& o = *reinterpret_cast<const StatsOut*>(h.data());
    double sum[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    for (uint32_t i = 0; i < kStatBlocks; ++i)
        for (uint32_t t = 0; t < 5; ++t) sum[t] += o.part[i][t];
    *out = clotho_stats{};
    out->segregating = o.segregating;
    out->fixed_now = o.fixed_now;
    out->heterozygosity = sum[4];
    out->mean_fitness = s.N ? s.fit_total / (double)s.N : 0.0;
    for (uint32_t t = 0; t < 4; ++t) out->mean_phenotype[t] = s.N ? sum[t] / s.N : 0.0;
    if (len) std::memcpy(sfs, h.data() + head, len * 4);
    return 0;
}

int clotho_stats_compute(clotho_ctx* ctx, clotho_stats* out, uint32_t* sfs, uint32_t sfs_len) {
    return stats_of(ctx, 0, out, sfs, sfs_len);
}

// Up to this many counts both margins come in one copy to the host, which hands them on: a copy to pageable memory has a
// fixed cost (a call on 150 individuals of 400 slots 68 us, so 59; on 7,900, just below the line, 71 and 65).
constexpr size_t kMarginsInOne = 16384;
static int margins_of(clotho_ctx* ctx, uint32_t idx, uint32_t* col, uint32_t* row) {
    if (!ctx || idx >= ctx->pops.size()) return fail(ctx, CLOTHO_E_ARG, "no such population");
    int rc;
    PopHost* p = ctx->pops[idx];
    const DevStatus s = read_status(ctx, p, &rc);
    if (rc) return rc;
    const uint32_t S = 2 * s.N;
    const size_t ncol = std::max<size_t>(1, (size_t)s.W * 64), nrow = std::max<uint32_t>(1, S);
    uint32_t* d = nullptr;
    CK(pool_alloc(ctx, &d, (ncol + nrow) * 4));
    CK(cudaMemsetAsync(d, 0, (ncol + nrow) * 4, ctx->stream));
    launch_margins(cfg(ctx), ctx->d_pops[0], idx, S, s.W, col ? d : nullptr, row ? d + ncol : nullptr);
    std::vector<uint32_t> h(col && row && ncol + nrow <= kMarginsInOne ? ncol + nrow : 0);
    if (!h.empty()) {
        CK(cudaMemcpyAsync(h.data(), d, h.size() * 4, cudaMemcpyDeviceToHost, ctx->stream));
    } else {
        if (col) host_pages(col, (size_t)s.A * 4);
        if (row) host_pages(row, (size_t)S * 4);
        if (col && s.A) CK(cudaMemcpyAsync(col, d, (size_t)s.A * 4, cudaMemcpyDeviceToHost, ctx->stream));
        if (row && S) CK(cudaMemcpyAsync(row, d + ncol, (size_t)S * 4, cudaMemcpyDeviceToHost, ctx->stream));
    }
    CK(cudaFreeAsync(d, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    if (!h.empty()) {
        std::memcpy(col, h.data(), (size_t)s.A * 4);
        std::memcpy(row, h.data() + ncol, (size_t)S * 4);
    }
    ctx->launches += (col || row) ? 1 : 0;
    return check_launch(ctx, "margins");
}

int clotho_margins(clotho_ctx* ctx, uint32_t* col, uint32_t* row) { return margins_of(ctx, 0, col, row); }
int clotho_pop_margins(clotho_ctx* ctx, uint32_t index, uint32_t* col, uint32_t* row) {
    return margins_of(ctx, index, col, row);
}

static int pairwise_of(clotho_ctx* ctx, uint32_t idx, const uint32_t* sample, uint32_t n, uint32_t* dist,
                       clotho_pairwise* out) {
    if (!ctx || !out || idx >= ctx->pops.size()) return fail(ctx, CLOTHO_E_ARG, "no such population");
    if (n > 65536u) return fail(ctx, CLOTHO_E_CAPACITY, "pairwise difference: sample of more than 65,536 rows");
    if (dist && n > 16384u) return fail(ctx, CLOTHO_E_CAPACITY, "pairwise distances: sample of more than 16,384 rows");
    int rc;
    PopHost* p = ctx->pops[idx];
    const DevStatus s = read_status(ctx, p, &rc);
    if (rc) return rc;
    const uint32_t S = 2 * s.N;
    std::vector<uint32_t> smp(n);
    for (uint32_t i = 0; i < n; ++i) {
        smp[i] = sample ? sample[i] : i;
        if (smp[i] >= S) return fail(ctx, CLOTHO_E_ARG, "pairwise difference: sample row out of range");
    }
    *out = clotho_pairwise{};
    const uint64_t pairs = n > 1 ? (uint64_t)n * (n - 1) / 2 : 0;
    if (!pairs) return 0;
    // one scratch block: accumulators, sample and, when the slots are split over CTAs, tile counts
    const PairwisePlan z = pairwise_plan(cfg(ctx), n, s.W);
    const size_t at_smp = align256(sizeof(PairwiseOut)), at_sums = at_smp + align256((size_t)n * 4);
    const size_t at_dist = align256(at_sums + z.sum_bytes);
    std::vector<char> head(at_smp + (size_t)n * 4);
    PairwiseOut h{};
    h.min = 0xffffffffu;
    std::memcpy(head.data(), &h, sizeof(h));
    std::memcpy(head.data() + at_smp, smp.data(), (size_t)n * 4);
    char* d = nullptr;
    CK(pool_alloc(ctx, &d, at_dist + (dist ? pairs * 4 : 0)));
    auto body = [&]() -> int {
        CK(cudaMemcpyAsync(d, head.data(), head.size(), cudaMemcpyHostToDevice, ctx->stream));
        CK(launch_pairwise(cfg(ctx), ctx->d_pops[0], idx, reinterpret_cast<uint32_t*>(d + at_smp), n, z, d + at_sums,
                           dist ? reinterpret_cast<uint32_t*>(d + at_dist) : nullptr, reinterpret_cast<PairwiseOut*>(d)));
        ctx->launches += (z.tiles + z.group - 1u) / z.group;
        if (int r = check_launch(ctx, "pairwise difference")) return r;
        CK(cudaMemcpyAsync(&h, d, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream));
        if (dist) host_pages(dist, pairs * 4);
        if (dist) CK(cudaMemcpyAsync(dist, d + at_dist, pairs * 4, cudaMemcpyDeviceToHost, ctx->stream));
        return 0;
    };
    rc = body();
    const cudaError_t e_free = cudaFreeAsync(d, ctx->stream);
    const cudaError_t e_sync = cudaStreamSynchronize(ctx->stream);
    if (rc) return rc;
    CK(e_free);
    CK(e_sync);
    if (h.err) return fail(ctx, CLOTHO_E_DEVICE, "pairwise difference: a tile's multiplications did not end");
    out->count = h.count;
    out->total = h.total;
    out->min = h.count ? h.min : 0;
    out->max = h.max;
    out->mean = h.count ? (double)h.total / (double)h.count : 0.0;
    out->variance = h.count ? (double)h.sumsq / (double)h.count - out->mean * out->mean : 0.0;
    if (out->variance < 0.0) out->variance = 0.0;
    return 0;
}

int clotho_pairwise_difference(clotho_ctx* ctx, const uint32_t* sample, uint32_t n, uint32_t* dist,
                               clotho_pairwise* out) {
    return pairwise_of(ctx, 0, sample, n, dist, out);
}
int clotho_pop_pairwise_difference(clotho_ctx* ctx, uint32_t index, const uint32_t* sample, uint32_t n,
                                   uint32_t* dist, clotho_pairwise* out) {
    return pairwise_of(ctx, index, sample, n, dist, out);
}

// ---- checkpoint / resume ---------------------------------------------------
namespace {
constexpr char kSnapMagic[8] = {'C', 'L', 'O', 'T', 'H', 'O', 'S', '1'};

struct SnapHeader {
    char magic[8];
    uint32_t version, header_bytes;
    clotho_desc desc;
    DevStatus st;
    uint64_t total_bytes;
};

struct SnapLayout {
    size_t rows, pos, age, eff, fx_pos, fx_age, fx_eff, free_list, zg, zi, fit, cdf, total;
};

// Byte offsets of the sections after the header, each 8-byte aligned.
SnapLayout snap_layout(const DevStatus& st, uint32_t T) {
    SnapLayout L{};
    const size_t S = 2ull * st.N, N = st.N, A = st.A, F = st.fixed_total;
    size_t o = sizeof(SnapHeader);
    auto take = [&](size_t bytes) {
        const size_t at = o;
        o += (bytes + 7) & ~(size_t)7;
        return at;
    };
    L.rows = take(S * st.W * 8);
    L.pos = take(A * 8);
    L.age = take(A * 4);
    L.eff = take(A * 16);
    L.fx_pos = take(F * 8);
    L.fx_age = take(F * 4);
    L.fx_eff = take(F * T * 4);
    L.free_list = take((size_t)st.free_cnt * 4);
    L.zg = take(S * 32);
    L.zi = take(N * 32);
    L.fit = take(N * 8);
    L.cdf = take(N * 8);
    L.total = o;
    return L;
}

bool same_parameters(const clotho_desc& a, const clotho_desc& b) {
    return a.traits == b.traits && a.fitness == b.fitness && a.flags == b.flags && a.fit_param == b.fit_param &&
           a.mu == b.mu && a.rho == b.rho && a.bias == b.bias && a.p_neutral == b.p_neutral &&
           a.eff_mean == b.eff_mean && a.eff_sigma == b.eff_sigma && a.seed == b.seed;
}
}  // namespace

size_t clotho_snapshot_size(clotho_ctx* ctx) {
    if (!ctx || ctx->pops.size() != 1 || ctx->in_step || !ctx->pops[0]->ready) return 0;
    int rc;
    const DevStatus st = read_status(ctx, ctx->pops[0], &rc);
    return rc ? 0 : snap_layout(st, ctx->pops[0]->dev[0].T).total;
}

int clotho_snapshot(clotho_ctx* ctx, void* dst, size_t len) {
    if (!ctx || !dst) return CLOTHO_E_ARG;
    if (ctx->pops.size() != 1) return fail(ctx, CLOTHO_E_ARG, "snapshot takes a single-population context");
    if (ctx->in_step) return fail(ctx, CLOTHO_E_STATE, "snapshot between generations only");
    PopHost* p = ctx->pops[0];
    if (!p->ready) return fail(ctx, CLOTHO_E_STATE, "population not initialised");
    int rc;
    const DevStatus st = read_status(ctx, p, &rc);
    if (rc) return rc;
    const PopDev& D = p->dev[0];
    const SnapLayout L = snap_layout(st, D.T);
    if (len < L.total) return fail(ctx, CLOTHO_E_CAPACITY, "snapshot buffer too small");
    host_pages(dst, L.total);
    char* b = static_cast<char*>(dst);
    SnapHeader h{};
    std::memcpy(h.magic, kSnapMagic, 8);
    h.version = 2;
    h.header_bytes = sizeof(SnapHeader);
    h.desc = p->desc;
    h.st = st;
    h.total_bytes = L.total;
    std::memcpy(b, &h, sizeof(h));
    const size_t S = 2ull * st.N, F = st.fixed_total;
    cudaStream_t s = ctx->stream;
    if (S * st.W)
        CK(cudaMemcpy2DAsync(b + L.rows, (size_t)st.W * 8, D.rows[st.cur], (size_t)D.Wcap * 8, (size_t)st.W * 8, S,
                             cudaMemcpyDeviceToHost, s));
    if (st.A) {
        CK(cudaMemcpyAsync(b + L.pos, D.pos, (size_t)st.A * 8, cudaMemcpyDeviceToHost, s));
        CK(cudaMemcpyAsync(b + L.age, D.age, (size_t)st.A * 4, cudaMemcpyDeviceToHost, s));
        CK(cudaMemcpyAsync(b + L.eff, D.eff, (size_t)st.A * 16, cudaMemcpyDeviceToHost, s));
    }
    if (F) {
        CK(cudaMemcpyAsync(b + L.fx_pos, D.fx_pos, F * 8, cudaMemcpyDeviceToHost, s));
        CK(cudaMemcpyAsync(b + L.fx_age, D.fx_age, F * 4, cudaMemcpyDeviceToHost, s));
        CK(cudaMemcpyAsync(b + L.fx_eff, D.fx_eff, F * D.T * 4, cudaMemcpyDeviceToHost, s));
    }
    if (st.free_cnt)
        CK(cudaMemcpyAsync(b + L.free_list, D.free_list, (size_t)st.free_cnt * 4, cudaMemcpyDeviceToHost, s));
    if (S) CK(cudaMemcpyAsync(b + L.zg, D.zg[st.cur], S * 32, cudaMemcpyDeviceToHost, s));
    if (st.N) {
        CK(cudaMemcpyAsync(b + L.zi, D.zi, (size_t)st.N * 32, cudaMemcpyDeviceToHost, s));
        CK(cudaMemcpyAsync(b + L.fit, D.fit, (size_t)st.N * 8, cudaMemcpyDeviceToHost, s));
        CK(cudaMemcpyAsync(b + L.cdf, D.cdf, (size_t)st.N * 8, cudaMemcpyDeviceToHost, s));
    }
    CK(cudaStreamSynchronize(s));
    return 0;
}

int clotho_restore(clotho_ctx* ctx, const void* src, size_t len) {
    if (!ctx || !src) return CLOTHO_E_ARG;
    if (ctx->pops.size() != 1) return fail(ctx, CLOTHO_E_ARG, "restore takes a single-population context");
    if (ctx->in_step) return fail(ctx, CLOTHO_E_STATE, "restore between generations only");
    if (len < sizeof(SnapHeader)) return fail(ctx, CLOTHO_E_ARG, "not a snapshot (too short)");
    SnapHeader h;
    std::memcpy(&h, src, sizeof(h));
    if (std::memcmp(h.magic, kSnapMagic, 8) != 0 || h.version != 2 || h.header_bytes != sizeof(SnapHeader))
        return fail(ctx, CLOTHO_E_ARG, "not a snapshot of this library version");
    PopHost* p = ctx->pops[0];
    const PopDev& D = p->dev[0];
    DevStatus st = h.st;
    if (st.cur > 1u || st.W != ref_width(st.A)) return fail(ctx, CLOTHO_E_ARG, "snapshot status is inconsistent");
    const SnapLayout L = snap_layout(st, D.T);
    if (h.total_bytes != L.total || len < L.total) return fail(ctx, CLOTHO_E_ARG, "snapshot truncated");
    if (!same_parameters(h.desc, p->desc))
        return fail(ctx, CLOTHO_E_ARG, "snapshot parameters differ from the context's");
    if (st.N > D.Ncap || st.A > D.Acap || st.W > D.Wcap || st.fixed_total > D.FXcap || st.free_cnt > D.Acap)
        return fail(ctx, CLOTHO_E_CAPACITY, "snapshot does not fit the context's capacities");
    const char* b = static_cast<const char*>(src);
    const size_t S = 2ull * st.N, F = st.fixed_total;
    // Everything below reaches device kernels as an index or a count: check it here, on the host, so a
    // damaged or hand-edited snapshot is refused instead of sending a kernel out of bounds.
    {
        if ((uint64_t)st.fixed_cnt + st.lost_cnt != st.free_cnt)
            return fail(ctx, CLOTHO_E_ARG, "snapshot free-list counts are inconsistent");
        std::vector<uint32_t> fl(st.free_cnt);
        if (st.free_cnt) std::memcpy(fl.data(), b + L.free_list, fl.size() * 4);
        for (uint32_t v : fl)
            if (v >= st.W * 64u) return fail(ctx, CLOTHO_E_ARG, "snapshot free list holds a slot beyond the rows");
        std::vector<double> pos(st.A);
        if (st.A) std::memcpy(pos.data(), b + L.pos, pos.size() * 8);
        for (double x : pos)
            if (!(x >= 0.0) || !std::isfinite(x)) return fail(ctx, CLOTHO_E_ARG, "snapshot allele position invalid");
        std::vector<float> eff((size_t)st.A * 4);
        if (st.A) std::memcpy(eff.data(), b + L.eff, eff.size() * 4);
        int64_t nz = 0;
        for (size_t a = 0; a < st.A; ++a)
            for (uint32_t t = 0; t < 4; ++t) {
                if (t >= D.T && eff[a * 4 + t] != 0.0f)
                    return fail(ctx, CLOTHO_E_ARG, "snapshot effects of unused traits are not zero");
                nz += eff[a * 4 + t] != 0.0f;
            }
        if (nz != st.nz_eff) return fail(ctx, CLOTHO_E_ARG, "snapshot effect count is inconsistent");
        // no row carries a slot at or beyond A (the reference never sets one; the classifiers index by slot)
        const uint32_t tail = st.A % 64u, last = st.A / 64u;
        if (st.W && (tail || last < st.W))
            for (size_t r = 0; r < S; ++r) {
                const uint64_t* row = reinterpret_cast<const uint64_t*>(b + L.rows) + r * st.W;
                uint64_t beyond = 0;
                std::memcpy(&beyond, row + last, last < st.W ? 8 : 0);
                if (tail) beyond &= ~((1ull << tail) - 1ull);
                for (uint32_t w = last + 1; w < st.W; ++w) {
                    uint64_t x;
                    std::memcpy(&x, row + w, 8);
                    beyond |= x;
                }
                if (beyond) return fail(ctx, CLOTHO_E_ARG, "snapshot rows carry slots beyond the allele count");
            }
    }
    int rc = init_pop(ctx, 0, st.N);  // zeroed tables and counters
    if (rc) return rc;
    st.count_cols = ctx->pops[0]->counting ? 1u : 0u;  // the context's own choice, not the snapshot's
    st.cols_valid = 0u;
    cudaStream_t s = ctx->stream;
    CK(cudaMemcpyAsync(D.st, &st, sizeof(DevStatus), cudaMemcpyHostToDevice, s));
    if (S * st.W)
        CK(cudaMemcpy2DAsync(D.rows[st.cur], (size_t)D.Wcap * 8, b + L.rows, (size_t)st.W * 8, (size_t)st.W * 8, S,
                             cudaMemcpyHostToDevice, s));
    if (st.A) {
        CK(cudaMemcpyAsync(D.pos, b + L.pos, (size_t)st.A * 8, cudaMemcpyHostToDevice, s));
        CK(cudaMemcpyAsync(D.age, b + L.age, (size_t)st.A * 4, cudaMemcpyHostToDevice, s));
        CK(cudaMemcpyAsync(D.eff, b + L.eff, (size_t)st.A * 16, cudaMemcpyHostToDevice, s));
    }
    if (F) {
        CK(cudaMemcpyAsync(D.fx_pos, b + L.fx_pos, F * 8, cudaMemcpyHostToDevice, s));
        CK(cudaMemcpyAsync(D.fx_age, b + L.fx_age, F * 4, cudaMemcpyHostToDevice, s));
        CK(cudaMemcpyAsync(D.fx_eff, b + L.fx_eff, F * D.T * 4, cudaMemcpyHostToDevice, s));
    }
    if (st.free_cnt)
        CK(cudaMemcpyAsync(D.free_list, b + L.free_list, (size_t)st.free_cnt * 4, cudaMemcpyHostToDevice, s));
    if (S) CK(cudaMemcpyAsync(D.zg[st.cur], b + L.zg, S * 32, cudaMemcpyHostToDevice, s));
    if (st.N) {
        CK(cudaMemcpyAsync(D.zi, b + L.zi, (size_t)st.N * 32, cudaMemcpyHostToDevice, s));
        CK(cudaMemcpyAsync(D.fit, b + L.fit, (size_t)st.N * 8, cudaMemcpyHostToDevice, s));
        CK(cudaMemcpyAsync(D.cdf, b + L.cdf, (size_t)st.N * 8, cudaMemcpyHostToDevice, s));
    }
    CK(cudaStreamSynchronize(s));
    p->acc_valid = false;  // the next step reduces the restored rows again
    drop_graphs(ctx);
    return 0;
}

// ---- timing --------------------------------------------------------------
int clotho_profile(clotho_ctx* ctx, int enable) {
    if (!ctx) return CLOTHO_E_ARG;
    int rc = prof_collect(ctx);
    if (rc) return rc;
    ctx->profiling = enable != 0;
    ctx->phase_clocks = enable == 2;
    ctx->prof_ms = 0.0;
    ctx->prof_launches = 0;
    drop_graphs(ctx);
    CK(cudaMemsetAsync(&ctx->d_ctl->rows_done, 0, 16 + sizeof(ctx->d_ctl->phase), ctx->stream));
    return 0;
}

int clotho_phase_clocks(clotho_ctx* ctx, uint64_t* out, uint32_t n) {
    static_assert(kPhCount == CLOTHO_PHASE_COUNT, "phase list of the header and the kernel differ");
    if (!ctx || (!out && n) || n > CLOTHO_PHASE_COUNT) return CLOTHO_E_ARG;
    uint64_t ph[kPhCount];
    CK(cudaMemcpyAsync(ph, ctx->d_ctl->phase, sizeof(ph), cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    for (uint32_t i = 0; i < n; ++i) out[i] = ph[i];
    return 0;
}

int clotho_kernel_time(clotho_ctx* ctx, double* total_ms, uint32_t* launches, uint64_t* rows, uint64_t* words) {
    if (!ctx) return CLOTHO_E_ARG;
    int rc = prof_collect(ctx);
    if (rc) return rc;
    uint64_t rw[2] = {0, 0};
    CK(cudaMemcpyAsync(rw, &ctx->d_ctl->rows_done, 16, cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    if (total_ms) *total_ms = ctx->prof_ms;
    if (launches) *launches = ctx->prof_launches;
    if (rows) *rows = rw[0];
    if (words) *words = rw[1];
    return 0;
}

int clotho_host_alloc(size_t bytes, void** out) {
    if (!out) return CLOTHO_E_ARG;
    *out = nullptr;
    if (cudaMallocHost(out, bytes ? bytes : 1) != cudaSuccess) {
        cudaGetLastError();
        return CLOTHO_E_NOMEM;
    }
    return 0;
}

int clotho_host_free(void* p) {
    if (p && cudaFreeHost(p) != cudaSuccess) return CLOTHO_E_CUDA;
    return 0;
}

int clotho_timer_begin(clotho_ctx* ctx) {
    if (!ctx) return CLOTHO_E_ARG;
    CK(cudaEventRecord(ctx->t0, ctx->stream));
    return 0;
}

int clotho_timer_end(clotho_ctx* ctx, double* ms) {
    if (!ctx) return CLOTHO_E_ARG;
    CK(cudaEventRecord(ctx->t1, ctx->stream));
    CK(cudaEventSynchronize(ctx->t1));
    float f = 0.f;
    CK(cudaEventElapsedTime(&f, ctx->t0, ctx->t1));
    if (ms) *ms = f;
    return 0;
}

// ---- batched and served populations --------------------------------------
int clotho_batch_create(const clotho_desc* descs, uint32_t n, clotho_ctx** out) {
    if (!out || (n && !descs) || n > kMaxPops) return CLOTHO_E_ARG;
    *out = nullptr;
    clotho_ctx* ctx = nullptr;
    if (n == 0) {
        // an empty context for a serving loop: create with a tiny population, then drop it
        clotho_desc d{};
        d.max_individuals = 1;
        d.max_alleles = 64;
        d.traits = 1;
        int rc = clotho_create(&d, &ctx);
        if (rc) return rc;
        free_pop(ctx, ctx->pops[0]);
        ctx->pops.clear();
        rc = sync_pop_arrays(ctx);
        if (rc) { clotho_destroy(ctx); return rc; }
        *out = ctx;
        return 0;
    }
    int rc = clotho_create(&descs[0], &ctx);
    if (rc) return rc;
    for (uint32_t i = 1; i < n; ++i) {
        PopHost* p = nullptr;
        rc = alloc_pop(ctx, descs[i], &p);
        if (rc) { clotho_destroy(ctx); return rc; }
        ctx->pops.push_back(p);
    }
    rc = sync_pop_arrays(ctx);
    if (rc) { clotho_destroy(ctx); return rc; }
    *out = ctx;
    return 0;
}

uint32_t clotho_pop_count(const clotho_ctx* ctx) { return ctx ? (uint32_t)ctx->pops.size() : 0u; }

int clotho_pop_add(clotho_ctx* ctx, const clotho_desc* desc, uint32_t* index) {
    if (!ctx || !desc) return CLOTHO_E_ARG;
    if (ctx->in_step) return fail(ctx, CLOTHO_E_STATE, "a staged generation is in progress");
    if (ctx->pops.size() >= kMaxPops) return fail(ctx, CLOTHO_E_CAPACITY, "256 populations resident");
    CK(cudaStreamSynchronize(ctx->stream));
    PopHost* p = nullptr;
    int rc = alloc_pop(ctx, *desc, &p);
    if (rc) return rc;
    ctx->pops.push_back(p);
    rc = sync_pop_arrays(ctx, (uint32_t)ctx->pops.size() - 1);
    if (rc) return rc;
    if (index) *index = (uint32_t)ctx->pops.size() - 1;
    return 0;
}

int clotho_pop_remove(clotho_ctx* ctx, uint32_t index) {
    if (!ctx || index >= ctx->pops.size()) return fail(ctx, CLOTHO_E_ARG, "no such population");
    CK(cudaStreamSynchronize(ctx->copy_stream));
    CK(cudaStreamSynchronize(ctx->stream));
    if (ctx->pops[index]->counting) {
        ctx->counting -= 1;
        ctx->tuning_epoch += 1;  // the step's kernels change when the last counting population leaves
    }
    free_pop(ctx, ctx->pops[index]);
    ctx->pops.erase(ctx->pops.begin() + index);
    return sync_pop_arrays(ctx, index);
}

int clotho_pop_count_columns(clotho_ctx* ctx, uint32_t index, int enable) {
    if (!ctx || index >= ctx->pops.size()) return fail(ctx, CLOTHO_E_ARG, "no such population");
    PopHost* p = ctx->pops[index];
    const bool on = enable != 0;
    if (p->counting == on) return 0;
    const uint32_t v = on ? 1u : 0u;
    CK(cudaMemcpyAsync(&p->dev[0].st->count_cols, &v, 4, cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    p->counting = on;
    ctx->counting += on ? 1u : (uint32_t)-1;
    ctx->tuning_epoch += 1;  // a captured step re-captures with (or without) the counting build
    return 0;
}

int clotho_pop_init(clotho_ctx* ctx, uint32_t index, uint32_t N0) { return init_pop(ctx, index, N0); }

int clotho_pop_info(clotho_ctx* ctx, uint32_t index, clotho_info* out) { return info_of(ctx, index, out); }

int clotho_pop_rows(clotho_ctx* ctx, uint32_t index, uint64_t* dst, size_t dst_words) {
    return rows_of(ctx, index, dst, dst_words);
}

int clotho_pop_stats(clotho_ctx* ctx, uint32_t index, clotho_stats* out, uint32_t* sfs, uint32_t sfs_len) {
    return stats_of(ctx, index, out, sfs, sfs_len);
}

int clotho_batch_generation_philox(clotho_ctx* ctx, const uint32_t* N) {
    int rc = require_ready(ctx);
    if (rc) return rc;
    if ((rc = block_tables(ctx))) return rc;
    if (!N) return fail(ctx, CLOTHO_E_ARG, "null N");
    if (ctx->pops.empty()) return 0;
    if (ctx->in_step) return fail(ctx, CLOTHO_E_STATE, "a staged generation is in progress");
    for (size_t i = 0; i < ctx->pops.size(); ++i)
        if (N[i] > ctx->pops[i]->dev[2].Ncap) return fail(ctx, CLOTHO_E_CAPACITY, "N exceeds max_individuals");
    if ((rc = put_header(ctx, [N](size_t i) { return N[i]; }))) return rc;
    enqueue_fused_step(ctx, 2, true);
    if ((rc = check_launch(ctx, "batch_generation_philox"))) return rc;
    sizes_are(ctx, [N](size_t i) { return N[i]; });
    return 0;
}

int clotho_batch_run_philox(clotho_ctx* ctx, const uint32_t* N, uint32_t G) {
    int rc = require_ready(ctx);
    if (rc) return rc;
    if (G == 0 || ctx->pops.empty()) return 0;
    if (!N) return fail(ctx, CLOTHO_E_ARG, "null N");
    if (ctx->in_step) return fail(ctx, CLOTHO_E_STATE, "a staged generation is in progress");
    for (size_t i = 0; i < ctx->pops.size(); ++i)
        if (N[i] > ctx->pops[i]->dev[2].Ncap) return fail(ctx, CLOTHO_E_CAPACITY, "N exceeds max_individuals");
    const std::vector<uint32_t> key(N, N + ctx->pops.size());
    uint32_t left = G;
    if (!ctx->profiling && graph_ready(ctx, key)) {
        if ((rc = put_header(ctx, [N](size_t i) { return N[i]; }))) return rc;
    } else {
        if ((rc = clotho_batch_generation_philox(ctx, N))) return rc;
        left -= 1;
    }
    if (ctx->profiling) {
        for (; left; --left)
            if ((rc = clotho_batch_generation_philox(ctx, N))) return rc;
        return 0;
    }
    if (left && (rc = replay_generations(ctx, key, left, StepEnd::kStep))) return rc;
    sizes_are(ctx, [N](size_t i) { return N[i]; });
    return 0;
}

int clotho_run_philox_schedule(clotho_ctx* ctx, const uint32_t* N, uint32_t G) {
    int rc = require_ready(ctx);
    if (rc) return rc;
    if ((rc = block_tables(ctx))) return rc;
    if (!N) return fail(ctx, CLOTHO_E_ARG, "null schedule");
    if (ctx->in_step) return fail(ctx, CLOTHO_E_STATE, "a staged generation is in progress");
    const uint32_t n = (uint32_t)ctx->pops.size();
    if (G == 0 || n == 0) return 0;
    // one step more than the schedule: the last one copies a header that nobody reads
    std::vector<uint32_t> hdr(2ull * n * (G + 1ull) + 4u, 0u);
    for (uint32_t g = 0; g < G; ++g)
        for (uint32_t i = 0; i < n; ++i) {
            const uint32_t v = N[(size_t)g * n + i];
            if (v > ctx->pops[i]->dev[2].Ncap)
                return fail(ctx, CLOTHO_E_CAPACITY, "schedule N exceeds max_individuals");
            hdr[2ull * ((size_t)g * n + i)] = v;
        }
    if (ctx->profiling) {  // per-launch events are taken from eager launches
        for (uint32_t g = 0; g < G; ++g)
            if ((rc = clotho_batch_generation_philox(ctx, N + (size_t)g * n))) return rc;
        return 0;
    }
    uint32_t* d_sched = nullptr;
    CK(pool_alloc(ctx, &d_sched, hdr.size() * 4));
    // every exit after the allocation goes through the one free below
    auto body = [&]() -> int {
        struct {
            const uint32_t* sched;
            uint32_t at;
        } const ctl{d_sched, 0u};   // as in WorkCtl
        const size_t ctl_bytes = sizeof(ctl.sched) + sizeof(ctl.at), ctl_word = hdr.size() - 4u;
        std::memcpy(hdr.data() + ctl_word, &ctl, ctl_bytes);
        CK(cudaMemcpyAsync(d_sched, hdr.data(), hdr.size() * 4, cudaMemcpyHostToDevice, ctx->stream));
        CK(cudaMemcpyAsync(&ctx->d_ctl->sched, d_sched + ctl_word, ctl_bytes, cudaMemcpyDeviceToDevice, ctx->stream));
        CK(cudaMemcpyAsync(ctx->d_hdr[2], d_sched, 8ull * n, cudaMemcpyDeviceToDevice, ctx->stream));
        // every size of a step is read from the device status word and a step leaves the next one's header, so one
        // graph serves all generations (with a copy of the header between replays, and graphs of one step, 32
        // generations of 301 to 5,003 individuals took 2.15 ms; 1.95)
        const std::vector<uint32_t> key{0xffffffffu, n};
        uint32_t left = G;
        if (!graph_ready(ctx, key)) {   // the first generation runs eagerly (it may need the parent reduction)
            enqueue_fused_step(ctx, 2, true, StepEnd::kSchedule);
            if (int r = check_launch(ctx, "run_philox_schedule")) return r;
            left -= 1;
        }
        if (left)
            if (int r = replay_generations(ctx, key, left, StepEnd::kSchedule)) return r;
        return 0;
    };
    rc = body();
    const cudaError_t e_free = cudaFreeAsync(d_sched, ctx->stream);
    const cudaError_t e_sync = cudaStreamSynchronize(ctx->stream);
    if (rc) return rc;
    CK(e_free);
    CK(e_sync);
    sizes_are(ctx, [=](size_t i) { return N[(size_t)(G - 1) * n + i]; });
    return 0;
}

int clotho_set_copy_wait_limit(clotho_ctx* ctx, uint32_t rounds) {
    if (!ctx) return CLOTHO_E_ARG;
    if (rounds > (1u << 30)) return fail(ctx, CLOTHO_E_ARG, "wait limit above 2^30 rounds");
    CK(cudaMemcpyAsync(&ctx->d_ctl->wait_limit, &rounds, sizeof(rounds), cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    return 0;
}

int clotho_set_tuning(clotho_ctx* ctx, const clotho_tuning* t) {
    if (!ctx || !t) return CLOTHO_E_ARG;
    if (t->rows_per_item > 65536 || t->row_blocks_per_sm > 64 || t->narrow_build > 1)
        return fail(ctx, CLOTHO_E_ARG, "tuning value out of range");
    if (t->rows_per_item) {
        int rc = clotho_set_rows_per_item(ctx, t->rows_per_item);
        if (rc) return rc;
    }
    if (ctx->pops.size() > 1) {   // steps under way read the block tables
        if (capturing(ctx)) ctx->parts_captured = true;
        else CK(cudaStreamSynchronize(ctx->stream));
    }
    ctx->ind_per_sm = t->row_blocks_per_sm ? t->row_blocks_per_sm : 16u;
    ctx->narrow_ok = t->narrow_build != 0u;
    ctx->parts_stale = true;
    ctx->tuning_epoch += 1;  // graphs captured under the old launch shapes are not replayed
    return 0;
}

int clotho_get_tuning(clotho_ctx* ctx, clotho_tuning* t) {
    if (!ctx || !t) return CLOTHO_E_ARG;
    uint32_t rpi = 0;
    CK(cudaMemcpyAsync(&rpi, &ctx->d_ctl->rows_per_item, 4, cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    t->rows_per_item = rpi;
    t->narrow_build = ctx->narrow_ok ? 1u : 0u;
    t->row_blocks_per_sm = ctx->ind_per_sm;
    return 0;
}

int clotho_set_rows_per_item(clotho_ctx* ctx, uint32_t rows) {
    if (!ctx || rows == 0 || rows > 65536) return CLOTHO_E_ARG;
    CK(cudaMemcpyAsync(&ctx->d_ctl->rows_per_item, &rows, 4, cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    drop_graphs(ctx);
    return 0;
}

int clotho_mem_info(size_t* free_bytes, size_t* total_bytes) {
    size_t f = 0, t = 0;
    if (cudaMemGetInfo(&f, &t) != cudaSuccess) {
        cudaGetLastError();
        return CLOTHO_E_CUDA;
    }
    if (free_bytes) *free_bytes = f;
    if (total_bytes) *total_bytes = t;
    return 0;
}

}  // extern "C"
