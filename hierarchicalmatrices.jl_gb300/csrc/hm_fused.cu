// A product in two launches, for small matrices whose tree passes are a chain
// of short dependent kernels.  Written for sm_103a.
//
// tree_fused runs every stage of the tree passes (leaf bases, upward bands,
// far field, downward bands) in one thread-block cluster of 16 CTAs, with a
// cluster barrier where the stage kernels have a launch boundary; expand_both, a
// programmatic dependent of it, sums the near-field columns of every row
// segment on the other SMs while the tree passes run, waits for them, sums the
// far-field columns and writes y once.  The bodies are those of the stage
// kernels (hm_tree.cuh, hm_df.cuh) and every sum has the same order, so results
// equal the stage kernels' bit for bit.
//
// What bounds it: latency.  At 4,096 points in FP32 the stages take 0.9 to 2.5 us
// each and are separated by a launch boundary of about 2 us, beside 11 launches
// and six event calls on the host (30.8 us per product); here a barrier costs
// well under 1 us (21.7 us; 27.6 -> 15.1 us at 1,000 points).  A grid-wide
// barrier in a cooperative launch, which would use every SM, measured 2.1 to 2.9
// us per stage, no better than the launch boundary.
#include "hm_async.cuh"
#include "hm_df.cuh"
#include "hm_fused.cuh"
#include "hm_kernels.cuh"
#include "hm_tree.cuh"

namespace hm {
namespace {

// Barrier over the CTAs of the cluster (all threads): what they wrote to global
// memory before it is visible after it.  `meanwhile` runs between this CTA's
// arrival and its wait: work that does not depend on the other CTAs.
template <typename F>
__device__ __forceinline__ void cluster_barrier(F meanwhile)
{
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    meanwhile();
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

}  // namespace

// Work of a stage goes over the grid item by item, warps of different CTAs
// first (a chain's latency, not its throughput, is what these sizes pay for).
// DF: HM_DF64 storage (S = A = double in memory, QC = 1; the transfer tasks
// take one right-hand side each, leaf bases and far field all of them).
template <typename S, typename A, int QC, bool DF>
__global__ void __launch_bounds__(kFusedThreads) tree_fused(const __grid_constant__ TreeArgs<S, A> a)
{
    extern __shared__ __align__(16) unsigned char fused_smem[];
    using TS = typename std::conditional<DF, float2, A>::type;     // stored transfer matrices and local vectors
    TS *Ts = reinterpret_cast<TS *>(fused_smem);
    unsigned char *work = fused_smem + 2 * HM_RMAX * HM_RMAX * sizeof(TS);
    const int wib = threadIdx.x >> 5, ctas = gridDim.x, cta = blockIdx.x;
    const int r = a.r, k = a.ma.k, nq = DF ? k : (k + QC - 1) / QC;
    pdl_trigger();                                             // expand_both may start its near field
    if (a.n_up || a.n_down) {                                  // without bands there is no T (assembled matrices)
        const TS *T = static_cast<const TS *>(a.T);
        for (int i = threadIdx.x; i < 2 * r * r; i += kFusedThreads) Ts[i] = T[i];
    }
    __shared__ TaskRecs recs;
    if (wib < a.leaf_warps) {
        for (int64_t i = (int64_t)wib * ctas + cta; i < a.n_vp; i += (int64_t)a.leaf_warps * ctas) {
            if constexpr (DF) {
                leaf_panel_df(a.ma, a.vp[i], static_cast<const float2 *>(a.V), a.t, r, a.cap,
                              reinterpret_cast<float2 *>(work) + (size_t)wib * a.cap);
            } else {
                hm_vpart part{};
                if (a.lp.rec) part = a.lp.rec[i];
                leaf_panel<S, A, QC>(a.ma, k, a.vp[i], part, static_cast<const S *>(a.V), a.t, r, a.cap, a.wcap,
                                     work + (size_t)wib * leaf_up_warp_bytes<S, A, QC>(a.cap, a.wcap), a.lp);
            }
            __syncwarp();
        }
    }
    for (int b = 0; b < a.n_up; ++b) {
        const int n = a.up_band[b + 1] - a.up_band[b];
        auto load = [&](int64_t i) {
            if (i < (int64_t)n * nq) load_task(a.up_tasks + a.up_band[b] + i % n, a.up_steps, a.up_ents, recs);
        };
        cluster_barrier([&] { load(cta); });
        __syncthreads();                                       // recs
        for (int64_t i = cta; i < (int64_t)n * nq; i += ctas) {
            TS *L = reinterpret_cast<TS *>(work);
            if constexpr (DF) {
                const int q = (int)(i / n);
                xfer_df_fetch<true>(recs, a.t, L, r, k, q);
                __syncthreads();
                if (r == 20) xfer_df_levels<true, 20>(recs, Ts, a.t, L, r, k, q);
                else xfer_df_levels<true, 0>(recs, Ts, a.t, L, r, k, q);
            } else {
                const int q0 = (int)(i / n) * QC;
                xfer_up_fetch<A, QC>(recs, a.t, L, r, k, q0);
                async_wait_all();
                __syncthreads();
                if (r == 20) xfer_up_levels<A, QC, 20>(recs, Ts, a.t, L, r, k, q0);
                else xfer_up_levels<A, QC, 0>(recs, Ts, a.t, L, r, k, q0);
            }
            if (i + ctas < (int64_t)n * nq) {
                load(i + ctas);                                // the walk ended with a CTA barrier
                __syncthreads();
            }
        }
    }
    if (a.n_rows) {
        // m2l_first writes between this warp's arrival and its wait, into shared memory
        // that other warps may still read leaf panels from; a band's last level ended
        // with a CTA barrier, without bands there was none since
        if (a.n_up == 0) __syncthreads();
        const int nm = DF ? 1 : nq;
        const int64_t items = (int64_t)a.n_rows * nm, i0 = (int64_t)wib * ctas + cta;
        const bool mine = wib < a.m2l_warps && i0 < items;
        hm_m2l_row R{};
        unsigned char *sm = work;
        if constexpr (!DF) sm += (size_t)wib * m2l_warp_bytes<S, A, QC>(a.fstride);
        cluster_barrier([&] {
            if (!mine) return;
            R = a.rows[i0 / nm];
            if constexpr (!DF) m2l_first(R, a.ents, static_cast<const S *>(a.F), a.fstride, sm);
        });
        if (mine) {
            for (int64_t i = i0; i < items; i += (int64_t)a.m2l_warps * ctas) {
                if (i != i0) R = a.rows[i / nm];
                if constexpr (DF) {
                    constexpr int NS = kM2lDfStages;
                    float2 *ring = reinterpret_cast<float2 *>(work) + (size_t)wib * (NS * 400 + 32);
                    m2l_row_df<NS>(R, a.ents, static_cast<const float2 *>(a.F), a.t, a.s, k, ring, ring + NS * 400);
                } else {
                    const int q0 = (int)(i % nm) * QC;
                    const S *F = static_cast<const S *>(a.F);
                    if (i != i0) m2l_first(R, a.ents, F, a.fstride, sm);
                    if (r == 20) m2l_row<S, A, QC, 20>(R, q0, a.ents, F, a.fstride, a.t, a.s, r, k, sm);
                    else m2l_row<S, A, QC, 0>(R, q0, a.ents, F, a.fstride, a.t, a.s, r, k, sm);
                }
                __syncwarp();
            }
        }
    }
    for (int b = 0; b < a.n_down; ++b) {
        const int n = a.down_band[b + 1] - a.down_band[b];
        auto load = [&](int64_t i) {
            if (i < (int64_t)n * nq) load_task(a.down_tasks + a.down_band[b] + i % n, a.down_steps, a.down_ents, recs);
        };
        cluster_barrier([&] { load(cta); });
        __syncthreads();                                       // recs
        for (int64_t i = cta; i < (int64_t)n * nq; i += ctas) {
            TS *L = reinterpret_cast<TS *>(work);
            if constexpr (DF) {
                const int q = (int)(i / n);
                xfer_df_fetch<false>(recs, a.s, L, r, k, q);
                __syncthreads();
                if (r == 20) xfer_df_levels<false, 20>(recs, Ts, a.s, L, r, k, q);
                else xfer_df_levels<false, 0>(recs, Ts, a.s, L, r, k, q);
            } else {
                const int q0 = (int)(i / n) * QC;
                xfer_down_fetch<A, QC>(recs, a.s, L, r, k, q0);
                async_wait_all();
                __syncthreads();
                if (r == 20) xfer_down_levels<A, QC, 20>(recs, Ts, a.s, L, r, k, q0);
                else xfer_down_levels<A, QC, 0>(recs, Ts, a.s, L, r, k, q0);
            }
            if (i + ctas < (int64_t)n * nq) {
                load(i + ctas);                                // the walk ended with a CTA barrier
                __syncthreads();
            }
        }
    }
}

namespace {

// The near-field sums of 3 to 8 FP32 right-hand sides in ring_part's order:
// chunks of at most 32 columns and pf panel values, the partial sums folded
// before a chunk that would take them past 64 columns, a chunk's columns dealt out to
// the lane groups of a low segment.
template <int KB>
__device__ __forceinline__ void seg_columns_ring(const float *Pg, int ld, const float *g, int c0, int c1, int pf,
                                                 float (&val)[KB][2])
{
    const int lane = threadIdx.x & 31;
    SegAcc<float, KB> a0, a1;
    a0.zero(); a1.zero();
    const int64_t ld2 = ld / 2;
    const int cc = min(kRingCols, pf / max(ld, 4)), cg = ring_groups(ld);
    if (cg > 1) {
        const int lr = lane & (32 / cg - 1);
        const float2 *base = reinterpret_cast<const float2 *>(Pg + 2 * lr);
        int nfold = 0;
        for (int c = c0; c < c1; c += cc) {
            const int n = min(cc, c1 - c);
            if (nfold + n > 64) {
                a0.fold(); a1.fold();
                nfold = 0;
            }
            nfold += n;
            if (2 * lr >= ld) continue;
            for (int u = lane / (32 / cg); u < n; u += 4 * cg) {
                float2 p[4];
#pragma unroll
                for (int v = 0; v < 4; ++v)
                    if (u + v * cg < n) p[v] = __ldcs(base + ld2 * (c + u + v * cg));
#pragma unroll
                for (int v = 0; v < 4; ++v)
                    if (u + v * cg < n) {
                        float gv[KB];
                        ld_vec<KB>(g + (c + u + v * cg) * KB, gv);
                        a0.add(p[v].x, gv); a1.add(p[v].y, gv);
                    }
            }
        }
        a0.fold(); a1.fold();
        ring_combine<KB>(32 / cg, [&](int i, int q) -> float & { return i ? a1.h[q] : a0.h[q]; },
                         [&](int i, int q) -> float & { return i ? a1.l[q] : a0.l[q]; });
    } else if (2 * lane < ld) {
        const float2 *base = reinterpret_cast<const float2 *>(Pg + 2 * lane);
        int left = 0, nfold = 0;
        auto use = [&](const float2 &p, int c) {
            if (left == 0) {
                left = min(cc, c1 - c);
                if (nfold + left > 64) {
                    a0.fold(); a1.fold();
                    nfold = 0;
                }
                nfold += left;
            }
            --left;
            float gv[KB];
            ld_vec<KB>(g + c * KB, gv);
            a0.add(p.x, gv); a1.add(p.y, gv);
        };
        int c = c0;
        for (; c + 16 <= c1; c += 16) {                        // 16 loads in flight per lane
            float2 p[16];
#pragma unroll
            for (int u = 0; u < 16; ++u) p[u] = __ldcs(base + ld2 * (c + u));
#pragma unroll
            for (int u = 0; u < 16; ++u) use(p[u], c + u);
        }
        for (; c + 4 <= c1; c += 4) {
            float2 p[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) p[u] = __ldcs(base + ld2 * (c + u));
#pragma unroll
            for (int u = 0; u < 4; ++u) use(p[u], c + u);
        }
        for (; c < c1; ++c) use(__ldcs(base + ld2 * c), c);
        a0.fold(); a1.fold();
    }
#pragma unroll
    for (int q = 0; q < KB; ++q) { val[q][0] = a0.merged(q, 0, 0); val[q][1] = a1.merged(q, 0, 0); }
}

// The far-field sums in far_rows' order: one FMA chain per row and right-hand side.
template <typename S, typename A, int KB>
__device__ __forceinline__ void seg_columns_plain(const S *Pg, int ld, const A *g, int c0, int c1, A (&val)[KB][2])
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < KB; ++q) val[q][0] = val[q][1] = A(0);
    if (2 * lane >= ld) return;
    using V2 = typename std::conditional<sizeof(S) == 4, float2, double2>::type;
    const V2 *base = reinterpret_cast<const V2 *>(Pg + 2 * lane);
    const int64_t ld2 = ld / 2;
    auto use = [&](const V2 &p, int c) {
#pragma unroll
        for (int q = 0; q < KB; ++q) {
            val[q][0] = fma((A)p.x, g[c * KB + q], val[q][0]);
            val[q][1] = fma((A)p.y, g[c * KB + q], val[q][1]);
        }
    };
    int c = c0;
    for (; c + 8 <= c1; c += 8) {
        V2 p[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) p[u] = __ldcs(base + ld2 * (c + u));
#pragma unroll
        for (int u = 0; u < 8; ++u) use(p[u], c + u);
    }
    for (; c < c1; ++c) use(__ldcs(base + ld2 * c), c);
}

}  // namespace

// Both parts of one row segment per warp: the near field before, the far field
// after the tree passes; y (+)= near, then + far, as the stage kernels do (far_rows: their
// far field is a thread per row, whose sums run column by column).
template <typename S, typename A, int KB>
__global__ void __launch_bounds__(128)
    expand_both(MulArgs<S> ma, const hm_seg *segs, int nsegs, const hm_piece *pieces, const S *P, const A *s,
                const A *t, int r, int maxw, int pf, bool far_rows)
{
    extern __shared__ __align__(16) unsigned char both_smem[];
    const int wib = threadIdx.x >> 5;
    const int seg = blockIdx.x * (blockDim.x >> 5) + wib;
    constexpr int NR = SegRows<S, KB>::per_lane;
    const bool live = seg < nsegs;
    A *g = reinterpret_cast<A *>(both_smem) + (int64_t)wib * maxw * KB;
    const hm_seg G = live ? segs[seg] : hm_seg{};
    A near[KB][NR], far[KB][NR];
    int c0, c1;
    if (live) {
        seg_gather<S, A, false, KB>(ma, G, pieces, s, t, r, g, c0, c1);
        __syncwarp();
        if constexpr (sizeof(S) == 4 && KB >= 4) seg_columns_ring<KB>(P + G.poff, G.ld, g, c0, c1, pf, near);
        else seg_columns<S, A, KB>(P + G.poff, G.ld, g, c0, c1, near);
    }
    pdl_wait();                                                // the tree passes' coefficients are ready
    if (!live) return;
    seg_gather<S, A, true, KB>(ma, G, pieces, s, t, r, g, c0, c1);
    __syncwarp();
    bool plain = KB >= 4;
    if constexpr (sizeof(S) == 8 && KB < 4) plain = far_rows;
    if constexpr (NR == 2) {
        if (plain) seg_columns_plain<S, A, KB>(P + G.poff, G.ld, g, c0, c1, far);
        else seg_columns<S, A, KB>(P + G.poff, G.ld, g, c0, c1, far);
    } else {
        seg_columns<S, A, KB>(P + G.poff, G.ld, g, c0, c1, far);
    }
#pragma unroll
    for (int q = 0; q < KB; ++q) {
        if (q >= ma.k) break;
#pragma unroll
        for (int j = 0; j < NR; ++j) {
            const int row = SegRows<S, KB>::row(j);
            if (row >= G.nrows) continue;
            S *yp = ma.y + (G.row0 + row) * ma.incy + (int64_t)q * ma.ldy;
            A v = near[q][j];
            if (ma.accumulate) v += (A)(*yp);
            *yp = (S)((S)v + (S)far[q][j]);
        }
    }
}

// The same with HM_DF64 panels: double-float sums, two rows per lane.
template <int KB>
__global__ void __launch_bounds__(128)
    expand_both_df(MulArgs<double> ma, const hm_seg *segs, int nsegs, const hm_piece *pieces, const float2 *P,
                   const double *s, const double *t, int r, int maxw, bool far_rows)
{
    extern __shared__ __align__(16) unsigned char both_smem[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int seg = blockIdx.x * (blockDim.x >> 5) + wib;
    const bool live = seg < nsegs;
    float2 *g = reinterpret_cast<float2 *>(both_smem) + (int64_t)wib * maxw * KB;
    const hm_seg G = live ? segs[seg] : hm_seg{};
    const int k = ma.k;
    auto gather = [&](bool far, int &c0, int &c1) {
        int col = 0;
        c0 = -1;
        c1 = 0;
        for (int pc = 0; pc < G.npieces; ++pc) {
            const hm_piece Q = pieces[G.piece0 + pc];
            if (far == (Q.kind != HM_PIECE_X)) {
                if (c0 < 0) c0 = col;
                for (int i = lane; i < Q.width * KB; i += 32) {
                    const int c = i / KB, q = i % KB;
                    double v = 0.0;
                    if (q < k)
                        v = far ? (Q.kind == HM_PIECE_TCOEF ? t : s)[((int64_t)Q.src * k + q) * r + c]
                                : ma.x[(Q.src + c) * ma.incx + (int64_t)q * ma.ldx];
                    g[(col + c) * KB + q] = df_split(v);
                }
                c1 = col + Q.width;
            }
            col += Q.width;
        }
        if (c0 < 0) c0 = c1 = 0;
        __syncwarp();
    };
    auto sums = [&](int c0, int c1, bool groups, double (&val)[KB][2]) {
        float sh[2][KB], sl[2][KB];
        df_columns<KB>(P + G.poff, G.ld, g, c0, c1, groups, sh, sl);
#pragma unroll
        for (int q = 0; q < KB; ++q)
#pragma unroll
            for (int j = 0; j < 2; ++j) val[q][j] = __dadd_rn((double)sh[j][q], (double)sl[j][q]);
    };
    double near[KB][2], far[KB][2];
    int c0, c1;
    if (live) {
        gather(false, c0, c1);
        sums(c0, c1, true, near);
    }
    pdl_wait();                                                // the tree passes' coefficients are ready
    if (!live) return;
    gather(true, c0, c1);
    sums(c0, c1, !far_rows, far);                          // far_rows_df sums column by column
#pragma unroll
    for (int q = 0; q < KB; ++q) {
        if (q >= k) break;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int row = 2 * lane + j;
            if (row >= G.nrows) continue;
            double *yp = ma.y + (G.row0 + row) * ma.incy + (int64_t)q * ma.ldy;
            double v = near[q][j];
            if (ma.accumulate) v = *yp + v;
            *yp = v + far[q][j];
        }
    }
}

#define HM_INST_FUSED(S, QC) template __global__ void tree_fused<S, S, QC, false>(const __grid_constant__ TreeArgs<S, S>);
HM_INST_FUSED(float, 1) HM_INST_FUSED(float, 2) HM_INST_FUSED(float, 4) HM_INST_FUSED(float, 8)
HM_INST_FUSED(double, 1) HM_INST_FUSED(double, 2) HM_INST_FUSED(double, 4) HM_INST_FUSED(double, 8)
template __global__ void tree_fused<double, double, 1, true>(const __grid_constant__ TreeArgs<double, double>);
#define HM_INST_BOTH(S, KB)                                                                                   \
    template __global__ void expand_both<S, S, KB>(MulArgs<S>, const hm_seg *, int, const hm_piece *, const S *, \
                                                   const S *, const S *, int, int, int, bool);
HM_INST_BOTH(float, 2) HM_INST_BOTH(float, 4) HM_INST_BOTH(float, 8)
HM_INST_BOTH(double, 1) HM_INST_BOTH(double, 2) HM_INST_BOTH(double, 4) HM_INST_BOTH(double, 8)
#define HM_INST_BOTH_DF(KB)                                                                                     \
    template __global__ void expand_both_df<KB>(MulArgs<double>, const hm_seg *, int, const hm_piece *,        \
                                                const float2 *, const double *, const double *, int, int, bool);
HM_INST_BOTH_DF(1) HM_INST_BOTH_DF(2) HM_INST_BOTH_DF(4) HM_INST_BOTH_DF(8)

}  // namespace hm
