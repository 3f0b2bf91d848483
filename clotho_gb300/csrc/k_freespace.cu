// k_freespace.cu -- free-space analysis of a population_space_row.
//
// Restates FreeSpaceAnalyzerMT<population_space_row>
// (data_spaces/free_space/free_space_mt_population_space_row_interlaced.hpp:41-121)
// and free_space_details::analyze_free_indices (free_space_details.hpp:299-357)
// for the GPU:
//  * k_fs_reduce  -- AND (fixed) / OR (variable) of every column over all rows,
//                    coalesced 128-bit row loads, folded into per-population
//                    accF/accV with global atomics.  In the fused path this
//                    reduction is done in the epilogue of the generation kernel
//                    and this kernel is only used for a freshly loaded population.
//  * fs_finalize_block (step.cuh) -- tail padding, ordered compaction (fixed
//                    indices ascending, then lost indices ascending) and
//                    fixed-table append (engine_batched_task.hpp:303-345): a
//                    block of the fused step's first kernel, or k_fs_finalize
//                    of the staged API, which sets the child allele count as
//                    well (child_max_alleles, :287-301).
#include "step.cuh"

namespace clotho {

// which == 0: the current child rows; which == 1: the parent of the step in progress.
__global__ void __launch_bounds__(256) k_fs_reduce(const PopDev* __restrict__ pops, uint32_t npops,
                                                   uint32_t which) {
    for (uint32_t p = blockIdx.z; p < npops; p += gridDim.z) {
        const PopDev& P = pops[p];
        const DevStatus st = *P.st;
        const uint32_t S = 2u * (which ? st.pN : st.N);
        const uint32_t W = which ? st.pW : st.W;
        const uint64_t* rows = P.rows[which ? (st.cur ^ 1u) : st.cur];
        const uint32_t nchunks = (W + 511u) / 512u;  // 256 threads x 2 words
        if (S == 0 || W == 0) continue;
        const uint32_t groups = gridDim.y;
        const uint32_t rows_per = (S + groups - 1) / groups;
        const uint32_t r0 = blockIdx.y * rows_per, r1 = min(S, r0 + rows_per);
        if (r0 >= r1) continue;
        for (uint32_t c = blockIdx.x; c < nchunks; c += gridDim.x) {
            const uint32_t w = c * 512u + 2u * threadIdx.x;
            if (w >= W) continue;
            uint64_t f0 = ~0ull, f1 = ~0ull, v0 = 0, v1 = 0;
            for (uint32_t r = r0; r < r1; ++r) {
                const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(rows + (size_t)r * P.Wcap + w);
                f0 &= x.x; f1 &= x.y; v0 |= x.x; v1 |= x.y;
            }
            atomicAnd((unsigned long long*)&P.accF[w], (unsigned long long)f0);
            atomicAnd((unsigned long long*)&P.accF[w + 1], (unsigned long long)f1);
            atomicOr((unsigned long long*)&P.accV[w], (unsigned long long)v0);
            atomicOr((unsigned long long*)&P.accV[w + 1], (unsigned long long)v1);
        }
    }
}

void launch_fs_reduce(const LaunchCfg& L, const PopDev* pops, uint32_t npops, uint32_t maxW, uint32_t which) {
    const dim3 pg = pop_grid(npops, 0x7fffffffu, L.num_sms, 4);  // blocks per population in pg.x
    const uint32_t gx = max(1u, min(16u, (maxW + 511u) / 512u));
    const dim3 grid(gx, max(1u, pg.x / gx), pg.z);
    k_fs_reduce<<<grid, 256, 0, L.stream>>>(pops, npops, which);
}

// Staged API: the analysis and the child's allele count (child_max_alleles, :287-301).
__global__ void __launch_bounds__(1024) k_fs_finalize(const PopDev* __restrict__ pops) {
    const PopDev& P = pops[blockIdx.x];
    DevStatus* st = P.st;
    fs_finalize_block(P, st->pN, st->pA, st->pW, false);
    if (threadIdx.x == 0) {
        const uint32_t M = st->M, fr = st->free_cnt;
        const uint32_t Ac = st->pA + (M > fr ? M - fr : 0u);
        if (Ac > P.Acap) st->err |= kErrAlleles;
        st->A = min(Ac, P.Acap);
        st->W = ref_width(st->A);
    }
}

void launch_fs_finalize(const LaunchCfg& L, const PopDev* pops, uint32_t npops) {
    k_fs_finalize<<<npops, 1024, 0, L.stream>>>(pops);
}

}  // namespace clotho
