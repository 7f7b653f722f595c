// Launch interface of the fused tree passes and segment sums (hm_fused.cu).
#pragma once
#include <type_traits>

#include "hm_kernels.cuh"

namespace hm {

constexpr int kFusedThreads = 256;
constexpr int kFusedCtas = 16;       // one cluster (16 against 8 CTAs: 21.7 / 24.9 us at 4,096 points, FP32)
constexpr int kFusedBands = 24;      // bands of one direction at most (24 x 4 tree levels)

// Everything tree_fused reads: the tables of the stage kernels and the warps per
// CTA of the stages whose warps need their own shared memory.
template <typename S, typename A>
struct TreeArgs {
    MulArgs<S> ma;
    const hm_vpanel *vp;
    const void *V, *T, *F;             // T: read only where there are bands (null in assembled matrices)
    LeafParts<A> lp;
    const hm_task *up_tasks, *down_tasks;
    const hm_step *up_steps, *down_steps;
    const hm_xfer *up_ents, *down_ents;
    const hm_m2l_row *rows;
    const hm_m2l_ent *ents;
    A *t, *s;
    int n_vp, cap, wcap, leaf_warps, m2l_warps, n_rows, fstride, r, n_up, n_down;
    int up_band[kFusedBands + 1], down_band[kFusedBands + 1];
};

// One cluster of kFusedThreads threads per CTA; shared memory: the two
// transfer matrices (2 HM_RMAX^2) and the largest stage's area.
template <typename S, typename A, int QC, bool DF>
__global__ void tree_fused(const __grid_constant__ TreeArgs<S, A> a);

// One warp per segment, 4 per CTA, shared memory maxw KB values per warp; pf:
// the panel values per chunk whose summation order the near field follows for
// 3 to 8 FP32 right-hand sides.
template <typename S, typename A, int KB>
__global__ void expand_both(MulArgs<S> ma, const hm_seg *segs, int nsegs, const hm_piece *pieces, const S *P,
                            const A *s, const A *t, int r, int maxw, int pf, bool far_rows);
template <int KB>
__global__ void expand_both_df(MulArgs<double> ma, const hm_seg *segs, int nsegs, const hm_piece *pieces,
                               const float2 *P, const double *s, const double *t, int r, int maxw, bool far_rows);

}  // namespace hm
