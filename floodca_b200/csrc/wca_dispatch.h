// Kernel variant table shared by the session code and the per-precision
// instantiation units (wca_inst_*.cu), so the variants compile in parallel.
#pragma once

#include <cuda_runtime.h>

#include "wca_kernels.cuh"

namespace fcab {

// Selects one compiled step-kernel variant.
struct VariantKey {
    int prec;   // FCAB_PREC_*
    int K;      // 4 or 8
    int cpl;    // 1, 2 or 4
    int math;   // MATH_*
    int rainf;  // per-cell rain field
    int landonly; // every cell LAND (mask not read, padding at PAD_Z)
    int blk = 0;  // FP32: the block sweep (needs the session's row maps and coded mask)
    int solo = 0; // block sweep: a missed seed's velocity pass by the last CTA
};

// Type-erased launchers; `g`, `rk` point at GridD<T>/RunK<T> of the variant's T.
struct Launchers {
    // split: ranges of a strip, 0 for an even split (sweeps by warp); rows of a
    // unit (block sweep)
    cudaError_t (*step)(const void *g, const void *rk, const TimeCfg &tc, Ctl *ctl, int split,
                        int grid, cudaStream_t s, int smem);
    // full velocity pass + step control: the first step's dt, or
    // (only_if_needed) a dt deferred by a step whose pruned maximum fell
    // below its seed
    cudaError_t (*init)(const void *g, const void *rk, const TimeCfg &tc, Ctl *ctl, int grid,
                        cudaStream_t s, int only_if_needed);
    const void *step_fn;   // __global__ symbol, for occupancy queries
    int threads;           // threads per CTA of the step kernel
    int smem;              // dynamic shared memory of the step kernel
    int blk;               // the block sweep: `grid` CTAs share the rows
    int nested;            // the step kernel holds a device-side launch
};

// Batched-ensemble launchers (FP32 state, FP64 accumulation).
struct BatchLaunchers {
    cudaError_t (*step)(const void *members, const int *unit_member, int total_units, BatchQ *q,
                        int *need_list, int grid, cudaStream_t s);
    // full velocity pass of the members whose step deferred its dt
    cudaError_t (*vfull)(const void *members, const int *need_list, BatchQ *q, int grid,
                         cudaStream_t s);
    cudaError_t (*window)(const void *members, int n, double window, cudaStream_t s);
    const void *step_fn;
    int threads, smem;     // per CTA of the step
};
bool lookup_batch_f32(const VariantKey &k, BatchLaunchers *out);

template <typename T, typename AccT, int K, int CPL, int MATH, bool RAINF, bool LAND>
cudaError_t launch_batch(const void *members, const int *unit_member, int total_units, BatchQ *q,
                         int *need_list, int grid, cudaStream_t s)
{
    k_step_batch<T, AccT, K, CPL, MATH, RAINF, LAND><<<grid, 128, 0, s>>>(
        static_cast<const MemberD<T> *>(members), unit_member, total_units, q, need_list);
    return cudaGetLastError();
}

template <typename AccT, int K, int MATH, bool RAINF, bool GEN>
cudaError_t launch_batch_blk(const void *members, const int *unit_member, int total_units,
                             BatchQ *q, int *need_list, int grid, cudaStream_t s)
{
    k_batch_blk<AccT, K, MATH, RAINF, GEN><<<grid, BLK_THREADS, blk_smem_bytes<K>(), s>>>(
        static_cast<const MemberD<float> *>(members), unit_member, total_units, q, need_list);
    return cudaGetLastError();
}

template <typename T, int K, int MATH>
cudaError_t launch_batch_vfull(const void *members, const int *need_list, BatchQ *q, int grid,
                               cudaStream_t s)
{
    k_batch_vfull<T, K, MATH><<<grid, 256, 0, s>>>(static_cast<const MemberD<T> *>(members),
                                                  need_list, q);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_window(const void *members, int n, double window, cudaStream_t s)
{
    k_batch_window<T><<<(n + 127) / 128, 128, 0, s>>>(static_cast<const MemberD<T> *>(members),
                                                       n, window);
    return cudaGetLastError();
}

// Returns false when the variant is not compiled.
bool lookup_f32(const VariantKey &k, Launchers *out);
bool lookup_f32all(const VariantKey &k, Launchers *out);
bool lookup_f64(const VariantKey &k, Launchers *out);

template <typename T, typename AccT, int K, int CPL, int MATH, bool RAINF, bool LAND>
cudaError_t launch_step(const void *g, const void *rk, const TimeCfg &tc, Ctl *ctl,
                        int segs, int grid, cudaStream_t s, int smem)
{
    k_step<T, AccT, K, CPL, MATH, RAINF, LAND><<<grid, step_threads<CPL, MATH>(), smem, s>>>(
        *static_cast<const GridD<T> *>(g), *static_cast<const RunK<T> *>(rk), tc, ctl,
        segs);
    return cudaGetLastError();
}

template <typename T, int K, int MATH>
cudaError_t launch_init(const void *g, const void *rk, const TimeCfg &tc, Ctl *ctl, int grid,
                        cudaStream_t s, int only_if_needed)
{
    k_init_dt<T, K, MATH><<<grid, 256, 0, s>>>(*static_cast<const GridD<T> *>(g),
                                              *static_cast<const RunK<T> *>(rk), tc, ctl,
                                              only_if_needed);
    return cudaGetLastError();
}

template <typename T, typename AccT, int K, int CPL, int MATH, bool RAINF, bool LAND>
Launchers make_launchers()
{
    Launchers L;
    L.step = &launch_step<T, AccT, K, CPL, MATH, RAINF, LAND>;
    L.init = &launch_init<T, K, MATH>;
    L.step_fn = (const void *)&k_step<T, AccT, K, CPL, MATH, RAINF, LAND>;
    L.threads = step_threads<CPL, MATH>();
    L.smem = 0;
    L.blk = 0;
    L.nested = 1;
    return L;
}

template <typename AccT, int K, int MATH, bool RAINF, bool GEN, bool TAILV>
cudaError_t launch_step_blk(const void *g, const void *rk, const TimeCfg &tc, Ctl *ctl, int seg,
                            int grid, cudaStream_t s, int smem)
{
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3((unsigned)grid);
    c.blockDim = dim3(BLK_THREADS);
    c.dynamicSmemBytes = (size_t)smem;
    c.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    c.attrs = at;
    // only where both launches fit on the GPU (two CTAs of each per SM of the
    // B200's 148): measured 3 to 9 % faster up to 512^2, 3 % slower at 733 x
    // 1101. Kernels that hold a launch (above BLK_SOLO cells) have none.
    c.numAttrs = !TAILV && grid <= 2 * 148 ? 1 : 0;
    return cudaLaunchKernelEx(&c, &k_step_blk<AccT, K, MATH, RAINF, GEN, TAILV>,
                              *static_cast<const GridD<float> *>(g),
                              *static_cast<const RunK<float> *>(rk), tc, ctl, seg);
}

template <typename AccT, int K, int MATH, bool RAINF, bool GEN, bool TAILV>
Launchers make_launchers_blk()
{
    Launchers L;
    L.step = &launch_step_blk<AccT, K, MATH, RAINF, GEN, TAILV>;
    L.init = &launch_init<float, K, MATH>;
    L.step_fn = (const void *)&k_step_blk<AccT, K, MATH, RAINF, GEN, TAILV>;
    L.threads = BLK_THREADS;
    L.smem = blk_smem_bytes<K>();
    L.blk = 1;
    L.nested = TAILV;
    return L;
}

template <typename AccT, int K, int MATH, bool TAILV>
Launchers pick_launchers_blk(const VariantKey &k)
{
    if (!k.landonly)
        return make_launchers_blk<AccT, K, MATH, true, true, TAILV>();
    return k.rainf ? make_launchers_blk<AccT, K, MATH, true, false, TAILV>()
                   : make_launchers_blk<AccT, K, MATH, false, false, TAILV>();
}

// Expands the (K, CPL, RAINF) combinations for one (T, AccT, MATH). FP32
// all-LAND grids run the block sweep, or one column per lane.
template <typename T, typename AccT, int MATH>
bool lookup_kcr(const VariantKey &k, Launchers *out)
{
    if constexpr (sizeof(T) == 4) {
        if (k.blk) {
            if (k.K == 4)
                *out = k.solo ? pick_launchers_blk<AccT, 4, MATH, false>(k)
                              : pick_launchers_blk<AccT, 4, MATH, true>(k);
            else
                *out = k.solo ? pick_launchers_blk<AccT, 8, MATH, false>(k)
                              : pick_launchers_blk<AccT, 8, MATH, true>(k);
            return true;
        }
    }
#define FCAB_CASE(KK, CC, RR)                                                    \
    if (k.K == KK && k.cpl == CC && (k.rainf != 0) == RR) {                      \
        if (k.landonly) {                                                        \
            if constexpr (sizeof(T) == 4 && CC != 1)                             \
                return false;                                                    \
            else                                                                 \
                *out = make_launchers<T, AccT, KK, CC, MATH, RR, true>();        \
        } else {                                                                 \
            *out = make_launchers<T, AccT, KK, CC, MATH, RR, false>();           \
        }                                                                        \
        return true;                                                             \
    }
    FCAB_CASE(4, 1, false) FCAB_CASE(4, 1, true)
    FCAB_CASE(4, 2, false) FCAB_CASE(4, 2, true)
    FCAB_CASE(4, 4, false) FCAB_CASE(4, 4, true)
    FCAB_CASE(8, 1, false) FCAB_CASE(8, 1, true)
    FCAB_CASE(8, 2, false) FCAB_CASE(8, 2, true)
    FCAB_CASE(8, 4, false) FCAB_CASE(8, 4, true)
#undef FCAB_CASE
    return false;
}

}  // namespace fcab
