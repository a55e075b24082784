// Batched-ensemble step-kernel variants (FP32 state, FP64 accumulation).
#include "wca_dispatch.h"

namespace fcab {

template <int K, int MATH, bool RAINF, bool GEN>
static void blk_batch(BatchLaunchers *out)
{
    out->step = &launch_batch_blk<double, K, MATH, RAINF, GEN>;
    out->step_fn = (const void *)&k_batch_blk<double, K, MATH, RAINF, GEN>;
    out->threads = BLK_THREADS;
    out->smem = blk_smem_bytes<K>();
    out->window = &launch_window<float>;
    out->vfull = &launch_batch_vfull<float, K, MATH>;
}

template <int MATH>
static bool lookup_batch_math(const VariantKey &k, BatchLaunchers *out)
{
    if (k.blk) {
        if (k.K == 4)
            !k.landonly ? blk_batch<4, MATH, true, true>(out)
                        : k.rainf ? blk_batch<4, MATH, true, false>(out)
                                  : blk_batch<4, MATH, false, false>(out);
        else
            !k.landonly ? blk_batch<8, MATH, true, true>(out)
                        : k.rainf ? blk_batch<8, MATH, true, false>(out)
                                  : blk_batch<8, MATH, false, false>(out);
        return true;
    }
#define FCAB_BCASE(KK, RR)                                                               \
    if (k.K == KK && k.cpl == 1 && (k.rainf != 0) == RR) {                               \
        if (k.landonly) {                                                                \
            out->step = &launch_batch<float, double, KK, 1, MATH, RR, true>;             \
            out->step_fn = (const void *)&k_step_batch<float, double, KK, 1, MATH, RR, true>; \
        } else {                                                                         \
            out->step = &launch_batch<float, double, KK, 1, MATH, RR, false>;            \
            out->step_fn = (const void *)&k_step_batch<float, double, KK, 1, MATH, RR, false>; \
        }                                                                                \
        out->threads = 128;                                                              \
        out->smem = 0;                                                                   \
        out->window = &launch_window<float>;                                             \
        out->vfull = &launch_batch_vfull<float, KK, MATH>;                               \
        return true;                                                                     \
    }
    FCAB_BCASE(4, false) FCAB_BCASE(4, true)
    FCAB_BCASE(8, false) FCAB_BCASE(8, true)
#undef FCAB_BCASE
    return false;
}

bool lookup_batch_f32(const VariantKey &k, BatchLaunchers *out)
{
    if (k.prec != 0)
        return false;
    return k.math == MATH_FAST ? lookup_batch_math<MATH_FAST>(k, out)
                               : lookup_batch_math<MATH_EXACT>(k, out);
}

}  // namespace fcab
