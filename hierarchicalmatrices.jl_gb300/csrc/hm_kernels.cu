// CUDA kernels: batched compression (fill) and the hierarchical matvec.
#include "hm_kernels.cuh"
#include "hm_async.cuh"
#include "hm_tree.cuh"

#include <type_traits>

namespace hm {

// ============================================================== fill kernels

// Explicit column bases: V[j, m] = (lam_m / (y_j - yh_m)) / sum_m' (...),
// the second barycentric form of src/BarycentricMatrix.jl:276-287, computed in
// FP64 and stored row-major (r values per point).  One CTA per panel.
template <typename S>
__global__ void fill_vpanels(FillArgs fa, const hm_vpanel *vp, const hm_fill_vpanel *vf,
                             int npanels, S *V)
{
    __shared__ double nodes[HM_RMAX], lam[HM_RMAX];
    const int p = blockIdx.x;
    if (p >= npanels) return;
    const hm_vpanel P = vp[p];
    const int r = fa.r;
    if (threadIdx.x < r) {
        nodes[threadIdx.x] = box_node(vf[p].a, vf[p].b, fa.cheb[threadIdx.x]);
        lam[threadIdx.x] = fa.lam[threadIdx.x];
    }
    __syncthreads();
    for (int j = threadIdx.x; j < P.nrows; j += blockDim.x) {
        const double yj = fa.y[P.row0 + j];
        double w[HM_RMAX];
        double sum = 0.0;
#pragma unroll
        for (int m = 0; m < HM_RMAX; ++m) {
            if (m < r) {
                w[m] = __dmul_rn(lam[m], 1.0 / __dsub_rn(yj, nodes[m]));
                sum = __dadd_rn(sum, w[m]);
            }
        }
        S *row = V + P.off + (int64_t)j * P.ld;
#pragma unroll
        for (int m = 0; m < HM_RMAX; ++m)
            if (m < r) row[m] = (S)(w[m] / sum);
    }
}

// F[m + r n] = f(xh_m, yh_n)  (src/BarycentricMatrix.jl:147-178).  One CTA per block.
template <typename S>
__global__ void fill_f(FillArgs fa, const hm_fill_f *ff, const hm_m2l_ent *ents, int nblocks, S *F)
{
    __shared__ double xh[HM_RMAX], yh[HM_RMAX];
    const int e = blockIdx.x;
    if (e >= nblocks) return;
    const int r = fa.r;
    if (threadIdx.x < r) {
        xh[threadIdx.x] = box_node(ff[e].xa, ff[e].xb, fa.cheb[threadIdx.x]);
        yh[threadIdx.x] = box_node(ff[e].ya, ff[e].yb, fa.cheb[threadIdx.x]);
    }
    __syncthreads();
    S *Fe = F + ents[e].foff;
    for (int idx = threadIdx.x; idx < r * r; idx += blockDim.x) {
        const int m = idx % r, n = idx / r;
        Fe[idx] = (S)fill_kernel(fa, xh[m], yh[n]);
    }
}

// Segment panels: the first basis_w columns hold the row basis U[i, m] of the
// segment's deepest row box (src/BarycentricMatrix.jl:256-267), the rest the
// near-field dense blocks f(x_i, y_j) (src/KernelMatrix.jl:57-60).  Column-major
// with leading dimension ld.  One CTA per segment.  DROW = true fills the
// derivative of every entry with respect to its row point instead: the basis
// derivative U_m'(x) = U_m(x) (sum_k U_k(x)/(x - xh_k) - 1/(x - xh_m)) and
// d f / d(row point) for the dense blocks.
template <typename S, bool DROW>
__global__ void fill_segments(FillArgs fa, const hm_seg *segs, const hm_piece *pieces,
                              const hm_fill_seg *sf, int nsegs, S *P)
{
    __shared__ double nodes[HM_RMAX], lam[HM_RMAX];
    const int sidx = blockIdx.x;
    if (sidx >= nsegs) return;
    const hm_seg G = segs[sidx];
    const hm_fill_seg Fi = sf[sidx];
    const int r = fa.r;
    S *Pg = P + G.poff;
    int col = 0;
    if (Fi.has_basis) {
        if (threadIdx.x < r) {
            nodes[threadIdx.x] = box_node(Fi.a, Fi.b, fa.cheb[threadIdx.x]);
            lam[threadIdx.x] = fa.lam[threadIdx.x];
        }
        __syncthreads();
        for (int i = threadIdx.x; i < G.nrows; i += blockDim.x) {
            const double xi = fa.x[G.row0 + i];
            double w[HM_RMAX];
            double sum = 0.0;
#pragma unroll
            for (int m = 0; m < HM_RMAX; ++m) {
                if (m < r) {
                    w[m] = __dmul_rn(lam[m], 1.0 / __dsub_rn(xi, nodes[m]));
                    sum = __dadd_rn(sum, w[m]);
                }
            }
            if (DROW) {
                double sd = 0.0;
#pragma unroll
                for (int m = 0; m < HM_RMAX; ++m)
                    if (m < r) sd += (w[m] / sum) / __dsub_rn(xi, nodes[m]);
#pragma unroll
                for (int m = 0; m < HM_RMAX; ++m)
                    if (m < r) Pg[i + (int64_t)G.ld * m] = (S)((w[m] / sum) * (sd - 1.0 / __dsub_rn(xi, nodes[m])));
            } else {
#pragma unroll
                for (int m = 0; m < HM_RMAX; ++m)
                    if (m < r) Pg[i + (int64_t)G.ld * m] = (S)(w[m] / sum);
            }
        }
        col = Fi.basis_w;
    }
    for (int pc = (Fi.has_basis ? 1 : 0); pc < G.npieces; ++pc) {
        const hm_piece Q = pieces[G.piece0 + pc];
        const int64_t tot = (int64_t)Q.width * G.nrows;
        for (int64_t idx = threadIdx.x; idx < tot; idx += blockDim.x) {
            const int i = (int)(idx % G.nrows), j = (int)(idx / G.nrows);
            Pg[i + (int64_t)G.ld * (col + j)] =
                (S)(DROW ? fill_kernel_drow(fa, fa.x[G.row0 + i], fa.y[Q.src + j])
                         : fill_kernel(fa, fa.x[G.row0 + i], fa.y[Q.src + j]));
        }
        col += Q.width;
    }
}

template __global__ void fill_vpanels<double>(FillArgs, const hm_vpanel *, const hm_fill_vpanel *, int, double *);
template __global__ void fill_vpanels<float>(FillArgs, const hm_vpanel *, const hm_fill_vpanel *, int, float *);
template __global__ void fill_f<double>(FillArgs, const hm_fill_f *, const hm_m2l_ent *, int, double *);
template __global__ void fill_f<float>(FillArgs, const hm_fill_f *, const hm_m2l_ent *, int, float *);
template __global__ void fill_segments<double, false>(FillArgs, const hm_seg *, const hm_piece *, const hm_fill_seg *, int, double *);
template __global__ void fill_segments<float, false>(FillArgs, const hm_seg *, const hm_piece *, const hm_fill_seg *, int, float *);
template __global__ void fill_segments<double, true>(FillArgs, const hm_seg *, const hm_piece *, const hm_fill_seg *, int, double *);
template __global__ void fill_segments<float, true>(FillArgs, const hm_seg *, const hm_piece *, const hm_fill_seg *, int, float *);

// ============================================================== matvec kernels
//
// Coefficients of slot `sl` for right-hand side q live at coef[(sl*k + q)*r + m].
// A product runs the tree passes (leaf_up, xfer_up per level, m2l, xfer_down
// per level) on a side stream while expand_part<.., false> streams the
// near-field dense panels on the caller's stream; after the join
// expand_part<.., true> adds the far field U s.


// One warp per explicit basis panel (leaf_panel, hm_tree.cuh).
template <typename S, typename A, int QC>
__global__ void leaf_up(MulArgs<S> ma, const hm_vpanel *vp, int npanels, const S *V, A *t, int r, int cap, int wcap,
                        LeafParts<A> lp)
{
    extern __shared__ unsigned char smem_raw[];
    pdl_trigger();
    const int wib = threadIdx.x >> 5;
    const int64_t w = (int64_t)blockIdx.x * (blockDim.x >> 5) + wib;
    if (w >= (int64_t)npanels) return;
    hm_vpart part{};
    const int kt = ma.k;
    if (lp.rec) {
        part = lp.rec[w];
        ma.x += (int64_t)lp.q0 * ma.ldx;
        if (ma.xin) ma.xin += (int64_t)lp.q0 * ma.ldx;
        ma.k = lp.nq;
        t += (int64_t)lp.q0 * r;
    }
    leaf_panel<S, A, QC>(ma, kt, vp[w], part, V, t, r, cap, wcap,
                         smem_raw + (size_t)wib * leaf_up_warp_bytes<S, A, QC>(cap, wcap), lp);
}

// FP64 leaf bases of rank 20, eight panels per CTA of five warps, thread (panel, m), for
// the reason m2l_flat has: 160 threads hold the 160 coefficients of eight panels.  A
// panel's rows stream from HBM (20 consecutive values a row, eight rows in flight),
// the right-hand sides' rows are staged in shared memory.  The sums are those of
// leaf_panel, in its order.  Upward half of the tree at n = 2^20: one right-hand side 145
// -> 119 us, two 238 -> 197.
template <int QC>
__global__ void __launch_bounds__(kFlatThreads)
    leaf_flat(MulArgs<double> ma, const hm_vpanel *vp, int npanels, const double *V, double *t, int cap)
{
    extern __shared__ __align__(16) double flat_smem[];
    constexpr int R = 20;
    const int i = threadIdx.x / R, m = threadIdx.x % R;
    const int64_t p = (int64_t)blockIdx.x * kFlatRows + i;
    const int k = ma.k, q0 = blockIdx.y * QC, qc = min(QC, k - q0);
    pdl_trigger();
    hm_vpanel P{};
    if (p < npanels) P = vp[p];
    double *xs = flat_smem + (size_t)i * cap * QC;             // [row][q]
    for (int j = m; j < P.nrows; j += R) {
#pragma unroll
        for (int q = 0; q < QC; ++q) {
            double *d = xs + j * QC + q;
            if (q < qc) async_copy<8>(d, ma.x + (P.row0 + j) * ma.incx + (int64_t)(q0 + q) * ma.ldx);
            else *d = 0.0;
        }
    }
    async_commit();
    const double *v = V + P.off + m;
    double acc[QC];
#pragma unroll
    for (int q = 0; q < QC; ++q) acc[q] = 0.0;
    constexpr int U = 8;
    double next[U];
#pragma unroll
    for (int u = 0; u < U; ++u) next[u] = u < P.nrows ? v[R * u] : 0.0;
    async_wait_all();
    __syncthreads();                                           // x is staged
    for (int j = 0; j < P.nrows; j += U) {
        double vv[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            vv[u] = next[u];
            if (j + U + u < P.nrows) next[u] = v[(int64_t)R * (j + U + u)];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (j + u >= P.nrows) break;
            double xv[QC];
            ld_vec<QC>(xs + (j + u) * QC, xv);
#pragma unroll
            for (int q = 0; q < QC; ++q) acc[q] = fma(vv[u], xv[q], acc[q]);
        }
    }
    if (p < npanels) {
#pragma unroll
        for (int q = 0; q < QC; ++q)
            if (q < qc) t[((int64_t)P.slot * k + q0 + q) * R + P.col0 + m] = acc[q];
    }
}

// Upward transfers of one band: t[parent][m] = sum_c sum_m' T_c[m', m] t[child_c][m'].
// One CTA per task (a subtree cut to the band's levels); the task's steps
// (levels, deepest first) run in order with a CTA barrier between them, warps
// taking (record, chunk of QC right-hand sides) pairs.  T (T_0 then T_1, each
// r x r with T_c[m' * r + m]) and the children's coefficients are staged in
// shared memory.
template <typename A, int QC>
__global__ void xfer_up_band(const hm_task *tasks, const hm_step *steps, const hm_xfer *ents, const A *T, A *t,
                             int r, int k)
{
    extern __shared__ unsigned char smem_raw[];
    A *Ts = reinterpret_cast<A *>(smem_raw);
    A *cs = Ts + 2 * HM_RMAX * HM_RMAX + (threadIdx.x >> 5) * 2 * QC * HM_RMAX;   // [c][qq][m']
    for (int i = threadIdx.x; i < 2 * r * r; i += blockDim.x) Ts[i] = T[i];
    __syncthreads();
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const int nq = (k + QC - 1) / QC;
    const hm_task tk = tasks[blockIdx.x];
    for (int st = tk.step0; st < tk.step1; ++st) {
        const hm_step S = steps[st];
        for (int64_t w = threadIdx.x >> 5; w < (int64_t)(S.e1 - S.e0) * nq; w += nw) {
            const hm_xfer X = ents[S.e0 + w / nq];
            const int q0 = (int)(w % nq) * QC, qc = min(QC, k - q0);
            for (int i = lane; i < QC * r; i += 32) {
                const int qq = i / r, m = i % r;
                cs[qq * HM_RMAX + m] = qq < qc ? t[((int64_t)X.c0 * k + q0 + qq) * r + m] : (A)0;
                cs[(QC + qq) * HM_RMAX + m] = qq < qc ? t[((int64_t)X.c1 * k + q0 + qq) * r + m] : (A)0;
            }
            __syncwarp();
            if (lane < r) {
                A acc[QC];
#pragma unroll
                for (int qq = 0; qq < QC; ++qq) acc[qq] = 0;
                for (int mp = 0; mp < r; ++mp) {
                    const A a0 = Ts[mp * r + lane], a1 = Ts[r * r + mp * r + lane];
#pragma unroll
                    for (int qq = 0; qq < QC; ++qq)
                        acc[qq] += a0 * cs[qq * HM_RMAX + mp] + a1 * cs[(QC + qq) * HM_RMAX + mp];
                }
#pragma unroll
                for (int qq = 0; qq < QC; ++qq)
                    if (qq < qc) t[((int64_t)X.slot * k + q0 + qq) * r + lane] = acc[qq];
            }
            __syncwarp();
        }
        __syncthreads();
    }
}

// Band tasks, one CTA per (task, chunk of QC right-hand sides: blockIdx.y)
// (xfer_up_fetch / xfer_up_levels and the downward pair, hm_tree.cuh).
template <typename A, int QC>
__global__ void xfer_up_task(const hm_task *tasks, const hm_step *steps, const hm_xfer *ents, const A *T, A *t,
                             int r, int k, int early)
{
    extern __shared__ unsigned char smem_raw[];
    __shared__ TaskRecs recs;
    A *Ts = reinterpret_cast<A *>(smem_raw);
    A *L = Ts + 2 * HM_RMAX * HM_RMAX;
    const int q0 = blockIdx.y * QC;                            // this CTA's right-hand sides
    if (early) pdl_trigger();     // the next band may be scheduled now (a small grid; not before a large one)
    for (int i = threadIdx.x; i < 2 * r * r; i += blockDim.x) async_copy<sizeof(A)>(Ts + i, T + i);
    load_task(tasks + blockIdx.x, steps, ents, recs);
    __syncthreads();
    pdl_wait();                                                // the children's coefficients are ready
    xfer_up_fetch<A, QC>(recs, t, L, r, k, q0);
    async_wait_all();
    __syncthreads();
    if (r == 20) xfer_up_levels<A, QC, 20>(recs, Ts, t, L, r, k, q0);
    else xfer_up_levels<A, QC, 0>(recs, Ts, t, L, r, k, q0);
}

template <typename A, int QC>
__global__ void xfer_down_task(const hm_task *tasks, const hm_step *steps, const hm_xfer *ents, const A *T, A *s,
                             int r, int k, int early)
{
    extern __shared__ unsigned char smem_raw[];
    __shared__ TaskRecs recs;
    A *Ts = reinterpret_cast<A *>(smem_raw);
    A *L = Ts + 2 * HM_RMAX * HM_RMAX;
    const int q0 = blockIdx.y * QC;                            // this CTA's right-hand sides
    if (early) pdl_trigger();
    for (int i = threadIdx.x; i < 2 * r * r; i += blockDim.x) async_copy<sizeof(A)>(Ts + i, T + i);
    load_task(tasks + blockIdx.x, steps, ents, recs);
    __syncthreads();
    pdl_wait();                                                // far-field and parent coefficients are ready
    xfer_down_fetch<A, QC>(recs, s, L, r, k, q0);
    async_wait_all();
    __syncthreads();
    if (r == 20) xfer_down_levels<A, QC, 20>(recs, Ts, s, L, r, k, q0);
    else xfer_down_levels<A, QC, 0>(recs, Ts, s, L, r, k, q0);
}

// One warp per (row slot, chunk of up to QC right-hand sides) (m2l_row, hm_tree.cuh).
template <typename S, typename A, int QC>
__global__ void m2l(const hm_m2l_row *rows, int nrows, const hm_m2l_ent *ents, const S *F, int fstride,
                    const A *t, A *s, int r, int k)
{
    extern __shared__ unsigned char smem_raw[];
    const int wib = threadIdx.x >> 5;
    const int nq = (k + QC - 1) / QC;
    const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    unsigned char *smem = smem_raw + wib * m2l_warp_bytes<S, A, QC>(fstride);
    const bool live = w < (int64_t)nrows * nq;
    pdl_trigger();
    hm_m2l_row R{};
    if (live) {
        R = rows[w / nq];
        m2l_first(R, ents, F, fstride, smem);
    }
    pdl_wait();                                                // the upward pass's coefficients are ready
    if (!live) return;
    const int q0 = (int)(w % nq) * QC;
    if (r == 20) m2l_row<S, A, QC, 20>(R, q0, ents, F, fstride, t, s, r, k, smem);
    else m2l_row<S, A, QC, 0>(R, q0, ents, F, fstride, t, s, r, k, smem);
}

// FP64 far field, rank 20: eight row slots per CTA of five warps, thread (row, m).  An
// FP64 warp instruction takes its 64 cycles with 20 lanes live as with 32, so one row
// slot per warp (m2l) left three eighths of the pipe unused; here 160 threads hold 160
// outputs.  Blocks (all eight rows' e-th at a time) and column coefficients are
// double-buffered in shared memory, a row's by its own 20 threads.  The sums are those
// of m2l_row, in its order.  Downward half of the tree at n = 2^20: one
// right-hand side 181 -> 164 us, two 331 -> 286.
template <int QC>
__global__ void __launch_bounds__(kFlatThreads)
    m2l_flat(const hm_m2l_row *rows, int nrows, const hm_m2l_ent *ents, const double *F, int fstride, const double *t,
             double *s, int k)
{
    extern __shared__ __align__(16) double flat_smem[];
    constexpr int R = 20, LD = R * R + kFlatPad;               // values between the rows' blocks
    const int i = threadIdx.x / R, m = threadIdx.x % R;
    const int row = blockIdx.x * kFlatRows + i, q0 = blockIdx.y * QC, qc = min(QC, k - q0);
    double *Fb = flat_smem;                                    // [stage][row][LD]
    double *Tb = Fb + 2 * kFlatRows * LD;                      // [stage][row][q][R]
    pdl_trigger();
    hm_m2l_row Rw{};
    if (row < nrows) Rw = rows[row];
    const int nb = Rw.end - Rw.begin;
    __shared__ int s_most;
    if (threadIdx.x == 0) s_most = 0;
    __syncthreads();
    if (m == 0) atomicMax(&s_most, nb);
    auto block = [&](int e) {
        if (e >= nb) return;
        const char *src = reinterpret_cast<const char *>(F + ents[Rw.begin + e].foff);
        char *dst = reinterpret_cast<char *>(Fb + ((e & 1) * kFlatRows + i) * LD);
#pragma unroll
        for (int c = 0; c < R * R / 2; c += R) async_copy16(dst + 16 * (c + m), src + 16 * (c + m));
    };
    auto coefs = [&](int e) {
        if (e >= nb) return;
        const double *src = t + ((int64_t)ents[Rw.begin + e].yslot * k + q0) * R + m;
        double *dst = Tb + ((e & 1) * kFlatRows + i) * QC * R + m;
#pragma unroll
        for (int q = 0; q < QC; ++q) {
            if (q < qc) async_copy<8>(dst + q * R, src + q * R);
            else dst[q * R] = 0.0;
        }
    };
    block(0);                                                  // F does not depend on the upward pass
    pdl_wait();
    coefs(0);
    async_commit();
    double acc[QC];
#pragma unroll
    for (int q = 0; q < QC; ++q) acc[q] = 0.0;
    __syncthreads();
    const int most = s_most;
    for (int e = 0; e < most; ++e) {
        block(e + 1);
        coefs(e + 1);
        async_commit();
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();                                       // the rows' copies are visible
        if (e < nb) {
            const double *f = Fb + ((e & 1) * kFlatRows + i) * LD + m;
            const double *tv = Tb + ((e & 1) * kFlatRows + i) * QC * R;
#pragma unroll
            for (int n = 0; n < R; ++n) {
                const double fv = f[R * n];
#pragma unroll
                for (int q = 0; q < QC; ++q) acc[q] = fma(fv, tv[q * R + n], acc[q]);
            }
        }
        __syncthreads();                                       // the stage is refilled by the next step
    }
    async_wait_all();
    if (row < nrows) {
#pragma unroll
        for (int q = 0; q < QC; ++q)
            if (q < qc) s[((int64_t)Rw.slot * k + q0 + q) * R + m] = acc[q];
    }
}

// Far field for many right-hand sides (k > QC): one CTA (4 warps) per row
// slot.  The row's r x r blocks are staged once in shared memory (up to
// kM2lBlocks at a time, cp.async); the warps then take chunks of QC
// right-hand sides in turn, double-buffering each block's column
// coefficients, lane m accumulating row m of the chunk.
constexpr int kM2lBlocks = 8;
template <typename S, typename A, int QC>
__global__ void m2l_k(const hm_m2l_row *rows, int nrows, const hm_m2l_ent *ents, const S *F, int fstride,
                      const A *t, A *s, int r, int k)
{
    extern __shared__ unsigned char smem_raw[];
    S *Fb = reinterpret_cast<S *>(smem_raw);                                      // kM2lBlocks x fstride
    A *Tb = reinterpret_cast<A *>(Fb + kM2lBlocks * fstride) + (threadIdx.x >> 5) * 2 * QC * HM_RMAX;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    pdl_trigger();
    pdl_wait();
    if (blockIdx.x >= nrows) return;
    const hm_m2l_row R = rows[blockIdx.x];
    for (int e0 = R.begin; e0 < R.end || e0 == R.begin; e0 += kM2lBlocks) {
        const int nb = min(kM2lBlocks, R.end - e0);
        __syncthreads();                                                           // previous batch used
        for (int b = 0; b < nb; ++b) {
            const char *src = reinterpret_cast<const char *>(F + ents[e0 + b].foff);
            char *dst = reinterpret_cast<char *>(Fb + b * fstride);
            for (int i = threadIdx.x; i < (int)(fstride * sizeof(S) / 16); i += blockDim.x)
                async_copy16(dst + 16 * i, src + 16 * i);
        }
        async_commit();
        async_wait_all();
        __syncthreads();
        for (int q0 = warp * QC; q0 < k; q0 += nw * QC) {
            const int qc = min(QC, k - q0);
            auto fetch = [&](int b, int buf) {
                A *tb = Tb + buf * QC * HM_RMAX;
                if (lane < r) {
                    const A *src = t + ((int64_t)ents[e0 + b].yslot * k + q0) * r + lane;
#pragma unroll
                    for (int qq = 0; qq < QC; ++qq) {
                        if (qq < qc) async_copy<sizeof(A)>(tb + qq * HM_RMAX + lane, src + (int64_t)qq * r);
                        else tb[qq * HM_RMAX + lane] = A(0);
                    }
                }
                async_commit();
            };
            A acc[QC];
#pragma unroll
            for (int qq = 0; qq < QC; ++qq) acc[qq] = 0;
            if (nb > 0) fetch(0, 0);
            for (int b = 0; b < nb; ++b) {
                if (b + 1 < nb) {
                    fetch(b + 1, (b + 1) & 1);
                    asm volatile("cp.async.wait_group 1;" ::: "memory");
                } else {
                    async_wait_all();
                }
                __syncwarp();
                const S *fb = Fb + b * fstride;
                const A *tb = Tb + (b & 1) * QC * HM_RMAX;
                if (lane < r) {
                    for (int n = 0; n < r; ++n) {
                        const A f = (A)fb[lane + r * n];
#pragma unroll
                        for (int qq = 0; qq < QC; ++qq) acc[qq] += f * tb[qq * HM_RMAX + n];
                    }
                }
                __syncwarp();
            }
            if (lane < r) {
                A *sp = s + ((int64_t)R.slot * k + q0) * r + lane;
#pragma unroll
                for (int qq = 0; qq < QC; ++qq) {
                    if (qq >= qc) break;
                    if (e0 == R.begin) sp[(int64_t)qq * r] = acc[qq];
                    else sp[(int64_t)qq * r] += acc[qq];
                }
            }
        }
        if (R.end <= R.begin) break;                                               // empty row: zeros written once
    }
}

// Downward transfers of one band: s[child_c][m'] += sum_m T_c[m', m] s[parent][m].
// Same task/step structure as xfer_up_band, topmost level first.
template <typename A, int QC>
__global__ void xfer_down_band(const hm_task *tasks, const hm_step *steps, const hm_xfer *ents, const A *T, A *s,
                               int r, int k)
{
    extern __shared__ unsigned char smem_raw[];
    A *Ts = reinterpret_cast<A *>(smem_raw);
    A *ps = Ts + 2 * HM_RMAX * HM_RMAX + (threadIdx.x >> 5) * QC * HM_RMAX;   // [qq][m]
    for (int i = threadIdx.x; i < 2 * r * r; i += blockDim.x) Ts[i] = T[i];
    __syncthreads();
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const int nq = (k + QC - 1) / QC;
    const hm_task tk = tasks[blockIdx.x];
    for (int st = tk.step0; st < tk.step1; ++st) {
        const hm_step S = steps[st];
        for (int64_t w = threadIdx.x >> 5; w < (int64_t)(S.e1 - S.e0) * nq; w += nw) {
            const hm_xfer X = ents[S.e0 + w / nq];
            const int q0 = (int)(w % nq) * QC, qc = min(QC, k - q0);
            for (int i = lane; i < QC * r; i += 32) {
                const int qq = i / r, m = i % r;
                ps[qq * HM_RMAX + m] = qq < qc ? s[((int64_t)X.slot * k + q0 + qq) * r + m] : (A)0;
            }
            __syncwarp();
            if (lane < r) {
                A a0[QC], a1[QC];
#pragma unroll
                for (int qq = 0; qq < QC; ++qq) { a0[qq] = 0; a1[qq] = 0; }
                for (int m = 0; m < r; ++m) {
                    const A t0 = Ts[lane * r + m], t1 = Ts[r * r + lane * r + m];
#pragma unroll
                    for (int qq = 0; qq < QC; ++qq) {
                        const A v = ps[qq * HM_RMAX + m];
                        a0[qq] += t0 * v;
                        a1[qq] += t1 * v;
                    }
                }
#pragma unroll
                for (int qq = 0; qq < QC; ++qq) {
                    if (qq < qc) {
                        s[((int64_t)X.c0 * k + q0 + qq) * r + lane] += a0[qq];
                        s[((int64_t)X.c1 * k + q0 + qq) * r + lane] += a1[qq];
                    }
                }
            }
            __syncwarp();
        }
        __syncthreads();
    }
}

// Row segments, up to KB right-hand sides: one warp per segment (<= 64 rows).
// FAR = false: the near-field dense columns, y (+)= D x (written with the
// caller's accumulate flag); FAR = true: the row-basis columns, y += U s.
// FP32: lanes 0-15 and 16-31 take alternate panel columns, each lane four
// consecutive rows through one 16-byte load per column; FP64: each lane two
// rows per 16-byte load.  The panel streams once from HBM whatever the
// number of right-hand sides; the gathered right-hand sides [s ; x pieces]
// are staged per warp in shared memory (g[c * KB + q]).  KB = 1 accumulates
// with compensated (TwoProd/TwoSum) sums, KB > 1 with FMA per piece folded
// in with TwoSum.
// Near field (FAR = false: y (+)= D x) or far field (FAR = true: U s) of one
// row segment per warp.  The far field goes to yfar (leading dimension ldf)
// when given, else it is added into y.
template <typename S, typename A, bool FAR, int KB>
__global__ void expand_part(MulArgs<S> ma, const hm_seg *segs, int nsegs, const hm_piece *pieces, const S *P,
                            const A *s, const A *t, int r, int maxw, S *yfar, int64_t ldf)
{
    extern __shared__ unsigned char smem_raw[];
    const int wib = threadIdx.x >> 5;
    const int seg = blockIdx.x * (blockDim.x >> 5) + wib;
    if constexpr (FAR) pdl_wait();                             // the downward pass's coefficients are ready
    if (seg >= nsegs) return;
    A *g = reinterpret_cast<A *>(smem_raw) + (int64_t)wib * maxw * KB;
    const hm_seg G = segs[seg];
    int c0, c1;
    if (!seg_gather<S, A, FAR, KB>(ma, G, pieces, s, t, r, g, c0, c1) && FAR && !yfar) return;   // no far field
    __syncwarp();
    constexpr int NR = SegRows<S, KB>::per_lane;
    A val[KB][NR];
    seg_columns<S, A, KB>(P + G.poff, G.ld, g, c0, c1, val);
    // FAR with yfar: write the far-field rows to yfar (added to y later);
    // FAR without: add into y; near field: y (+)= per the caller's flag
    const bool acc_y = FAR ? (yfar == nullptr) : (ma.accumulate != 0);
#pragma unroll
    for (int q = 0; q < KB; ++q) {
        if (q >= ma.k) break;
#pragma unroll
        for (int j = 0; j < NR; ++j) {
            const int row = SegRows<S, KB>::row(j);
            if (row >= G.nrows) continue;
            if (FAR && yfar) {
                yfar[(G.row0 + row) + (int64_t)q * ldf] = (S)val[q][j];
            } else {
                S *yp = ma.y + (G.row0 + row) * ma.incy + (int64_t)q * ma.ldy;
                A v = val[q][j];
                if (acc_y) v += (A)(*yp);
                *yp = (S)v;
            }
        }
    }
}

// Far-field rows U s with one thread per row: four segments per CTA of 256
// threads, 64 threads per segment.  The segment's far-field coefficients (its
// non-X pieces, at most 64 columns, KB right-hand sides) are gathered once into
// shared memory; thread `row` then reads its row of the column-major basis
// columns (consecutive threads, consecutive rows: coalesced) and accumulates
// KB sums with FMA (at most 64 terms, as the warp kernels' folds do); ks: right-hand
// sides of the coefficients (ma.k of them from s, t on).  The
// rows go to yfar (leading dimension ldf) or, without it, are added into y.
template <typename S, typename A, int KB>
__global__ void __launch_bounds__(256)
    far_rows(MulArgs<S> ma, const hm_seg *segs, int nsegs, const hm_piece *pieces, const S *P, const A *s,
             const A *t, int r, int ks, S *yfar, int64_t ldf)
{
    __shared__ A cs[4][64 * KB];                               // [segment][column][q]
    pdl_wait();                                                // the downward pass's coefficients are ready
    const int ls = threadIdx.x >> 6, row = threadIdx.x & 63;
    const int j = blockIdx.x * 4 + ls;
    const int k = ma.k;
    hm_seg G{};
    int nfar = 0;
    if (j < nsegs) {
        G = segs[j];
        nfar = G.nfar;
        // coefficients of the far columns: element e = (column c, q) with c = e / KB
        for (int e = row; e < nfar * KB; e += 64) {
            const int c = e / KB, q = e % KB;
            int pc = 0, pi = 0;
            hm_piece Q = pieces[G.piece0];
            while (c >= pc + Q.width) {
                pc += Q.width;
                Q = pieces[G.piece0 + ++pi];
            }
            A v = A(0);
            if (q < k) v = (Q.kind == HM_PIECE_TCOEF ? t : s)[((int64_t)Q.src * ks + q) * r + (c - pc)];
            cs[ls][e] = v;
        }
    }
    __syncthreads();
    if (j >= nsegs || row >= G.nrows) return;
    if (nfar == 0 && !yfar) return;                            // y += 0
    A acc[KB];
#pragma unroll
    for (int q = 0; q < KB; ++q) acc[q] = A(0);
    const S *pr = P + G.poff + row;
    // eight columns' loads issued before their FMAs (eight loads in flight per
    // thread), the sums in column order as one column at a time
    constexpr int CU = 8;
    int c = 0;
    for (; c + CU <= nfar; c += CU) {
        A u[CU];
#pragma unroll
        for (int i = 0; i < CU; ++i) u[i] = (A)__ldcs(pr + (int64_t)(c + i) * G.ld);
#pragma unroll
        for (int i = 0; i < CU; ++i)
#pragma unroll
            for (int q = 0; q < KB; ++q) acc[q] = fma(u[i], cs[ls][(c + i) * KB + q], acc[q]);
    }
    for (; c < nfar; ++c) {
        const A u = (A)__ldcs(pr + (int64_t)c * G.ld);
#pragma unroll
        for (int q = 0; q < KB; ++q) acc[q] = fma(u, cs[ls][c * KB + q], acc[q]);
    }
#pragma unroll
    for (int q = 0; q < KB; ++q) {
        if (q >= k) break;
        if (yfar) {
            yfar[(G.row0 + row) + (int64_t)q * ldf] = (S)acc[q];
        } else {
            S *yp = ma.y + (G.row0 + row) * ma.incy + (int64_t)q * ma.ldy;
            *yp = (S)((A)(*yp) + acc[q]);
        }
    }
}

// y[i*incy + q*ldy] += yfar[i + q*ldf]: adds the far-field rows computed on the
// side stream (after the join).
template <typename S>
__global__ void add_far(MulArgs<S> ma, int64_t n, const S *yfar, int64_t ldf)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n * ma.k) return;
    const int64_t row = i % n, q = i / n;
    S *yp = ma.y + row * ma.incy + q * ma.ldy;
    S *dst = ma.yout ? ma.yout + row + q * n : yp;
    *dst = *yp + yfar[row + q * ldf];
}

// ------------------------------------------------------- streamed panels
//
// One persistent CTA of 256 threads per slot (two per SM).  CTA b owns the
// segments [cta_seg[b], cta_seg[b+1]), balanced by panel bytes on the host.
// Thread 0 streams the part's columns of those panels chunk by chunk (ld rows
// x cc columns, one contiguous run of the column-major panel) into a ring of
// nst shared-memory stages with cp.async.bulk; each stage's mbarrier
// completes when its bytes have landed.  All threads consume: thread
// (row = tid % 64, group = tid / 64) multiplies its row by a quarter of the
// chunk's columns with plain FMA and folds the chunk's partial into a
// compensated (TwoSum) pair.  The gathered right-hand sides of the next
// segment are fetched with cp.async while the current one streams.  Every
// wait is bounded: after wait_ns (the handle's HM_OPT_WAIT_LIMIT_NS) the CTA
// records HM_DEV_WAIT_TIMEOUT in *status, waits (bounded by kDrainLimitNs) for
// its copies in flight and returns.  stall != 0 (a test hook) makes the first
// wait of every CTA run out.


template <typename S, typename A, bool FAR, int KB>
__global__ void __launch_bounds__(kStreamThreads, KB >= 4 ? (sizeof(S) == 4 ? 2 : 1) : 3)   // registers of 4+ right-hand sides
    stream_part(MulArgs<S> ma, const hm_seg *segs, const int *cta_seg, const hm_piece *pieces, const S *P,
                const A *s, const A *t, int r, int nst, int gcap, int ngb, int dsegs, S *yfar, int *status,
                unsigned long long wait_ns, int stall)
{
    static_assert(sizeof(S) == sizeof(A), "right-hand sides are copied into shared memory as they are");
    // rows per thread: one 16-byte load; FP32 with 4+ right-hand sides takes 2
    // (8-byte loads) to keep its accumulators in registers
    constexpr bool kNarrow = sizeof(S) == 4 && KB >= 4;
    using V = typename std::conditional<sizeof(S) == 4, typename std::conditional<kNarrow, float2, float4>::type,
                                        double2>::type;
    constexpr int VEC = kNarrow ? 2 : 16 / (int)sizeof(S);
    constexpr int RQ = 64 / VEC;                               // row vectors of a 64-row segment
    constexpr int NG = kStreamThreads / RQ;                    // column groups
    constexpr int CC = kChunkBytes / (64 * (int)sizeof(S));   // columns per chunk
    constexpr int CPG = CC / NG;                               // columns per group per chunk
    constexpr int FOLDC = 4;                                   // chunks between compensated folds
    constexpr bool kFold = sizeof(A) == 4;                     // FP64 sums plainly
    static_assert(CPG * NG == CC && NG * RQ == kStreamThreads, "chunk geometry");
    extern __shared__ unsigned char stream_smem[];
    const int seg_lo = cta_seg[blockIdx.x], seg_hi = cta_seg[blockIdx.x + 1];
    if (seg_lo >= seg_hi) return;
    const int tid = threadIdx.x, rv = tid % RQ, grp = tid / RQ;
    const int lane = tid & 31, warp = tid >> 5;
    const int k = ma.k;
    unsigned char *ring = stream_smem;
    uint64_t *full = reinterpret_cast<uint64_t *>(stream_smem + (size_t)nst * kChunkBytes);
    uint64_t *never = full + nst;                              // nothing arrives on it (stall hook)
    A *gbuf = reinterpret_cast<A *>(full + nst + 1);
    A *red = gbuf + ngb * gcap * KB;                           // [warp][row][q][hi, lo]
    // the CTA's segment and piece records, staged once (records of one CTA
    // are consecutive in both arrays)
    hm_seg *sseg = reinterpret_cast<hm_seg *>(red + 8 * 64 * KB * 2);
    hm_piece *spc = reinterpret_cast<hm_piece *>(sseg + dsegs);
    {
        const int ns = seg_hi - seg_lo;
        const int p_lo = segs[seg_lo].piece0;
        const int np = segs[seg_hi - 1].piece0 + segs[seg_hi - 1].npieces - p_lo;
        const int64_t *gs = reinterpret_cast<const int64_t *>(segs + seg_lo);
        int64_t *ds = reinterpret_cast<int64_t *>(sseg);
        for (int i = tid; i < ns * (int)(sizeof(hm_seg) / 8); i += kStreamThreads) ds[i] = gs[i];
        const int64_t *gp = reinterpret_cast<const int64_t *>(pieces + p_lo);
        int64_t *dp = reinterpret_cast<int64_t *>(spc);
        for (int i = tid; i < np * (int)(sizeof(hm_piece) / 8); i += kStreamThreads) dp[i] = gp[i];
        __syncthreads();
        for (int i = tid; i < ns; i += kStreamThreads) sseg[i].piece0 -= p_lo;
        __syncthreads();
    }

    auto part_range = [&](const hm_seg &G, int &cb, int &ce) {
        cb = FAR ? 0 : G.nfar;
        ce = FAR ? G.nfar : G.width;
    };
    // right-hand side entries of segment j's part columns into dst (cp.async)
    auto gather = [&](int j, A *dst) {
        const hm_seg G = sseg[j - seg_lo];
        int col = 0;
        for (int pc = 0; pc < G.npieces; ++pc) {
            const hm_piece Q = spc[G.piece0 + pc];
            const bool take = FAR ? (Q.kind != HM_PIECE_X) : (Q.kind == HM_PIECE_X);
            if (!take) continue;
            for (int i = tid; i < Q.width * KB; i += kStreamThreads) {
                const int c = i / KB, q = i % KB;
                A *d = dst + (col + c) * KB + q;
                if (q < k) {
                    const void *src;
                    if (FAR)
                        src = (Q.kind == HM_PIECE_TCOEF ? t : s) + ((int64_t)Q.src * k + q) * r + c;
                    else
                        src = ma.x + (Q.src + c) * ma.incx + (int64_t)q * ma.ldx;
                    async_copy<sizeof(A)>(d, src);
                } else {
                    *d = A(0);
                }
            }
            col += Q.width;
        }
    };

    // producer state (thread 0): next chunk to issue
    int pj = seg_lo, pc = 0, pce = 0, pld = 0, issued = 0;
    int64_t pbase = 0;
    auto seek = [&](int j) {
        for (; j < seg_hi; ++j) {
            const hm_seg G = sseg[j - seg_lo];
            int cb, ce;
            part_range(G, cb, ce);
            if (ce > cb) {
                pc = cb; pce = ce; pld = G.ld; pbase = G.poff;
                break;
            }
        }
        pj = j;
    };
    auto issue = [&](int stage) {
        const int cols = min(CC, pce - pc);
        const uint32_t bytes = (uint32_t)(cols * pld) * (uint32_t)sizeof(S);
        bulk_load(ring + (size_t)stage * kChunkBytes, P + pbase + (int64_t)pc * pld, bytes, &full[stage]);
        ++issued;
        pc += CC;
        if (pc >= pce) seek(pj + 1);
    };

    if (tid == 0) {
        for (int i = 0; i <= nst; ++i) mbar_init(&full[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // right-hand sides run ngb - 1 segments ahead (one cp.async group per segment)
    for (int j = seg_lo; j < seg_lo + ngb - 1; ++j) {
        if (j < seg_hi) gather(j, gbuf + ((j - seg_lo) % ngb) * gcap * KB);
        async_commit();
    }
    __syncthreads();
    if (tid == 0) {
        seek(seg_lo);
        for (int i = 0; i < nst && pj < seg_hi; ++i) issue(i);
    }

    int stage = 0, consumed = 0;
    uint32_t phase = 0;
    bool abort = false;
    bool stall_first = stall != 0;
    for (int j = seg_lo; j < seg_hi && !abort; ++j) {
        async_wait_pending(ngb - 2);
        __syncthreads();                      // g of segment j visible; g and partials of j - 1 read
        {
            const int ja = j + ngb - 1;       // into the buffer segment j - 1 used
            if (ja < seg_hi) gather(ja, gbuf + ((ja - seg_lo) % ngb) * gcap * KB);
            async_commit();
        }
        const hm_seg G = sseg[j - seg_lo];
        int cb, ce;
        part_range(G, cb, ce);
        const A *g = gbuf + ((j - seg_lo) % ngb) * gcap * KB;
        const int row0 = VEC * rv;
        const bool live = row0 < G.nrows;
        const bool acc_y = FAR ? (yfar == nullptr && ce > cb) : (ma.accumulate != 0);
        A part[VEC][KB], hi[VEC][KB], lo[VEC][KB];
#pragma unroll
        for (int v = 0; v < VEC; ++v)
#pragma unroll
            for (int q = 0; q < KB; ++q) part[v][q] = hi[v][q] = lo[v][q] = A(0);
        // the final merge: thread t combines the partials of row t / 4 (the
        // four threads of a row sit in one warp); t % 4 == 0 writes the row
        const int mrow = tid >> 2, mpart = tid & 3;
        const bool writer = mpart == 0 && mrow < G.nrows;
        // y values the segment adds to, loaded now and used at its end
        S yold[KB];
#pragma unroll
        for (int q = 0; q < KB; ++q) {
            yold[q] = S(0);
            if (acc_y && writer && q < k) yold[q] = ma.y[(G.row0 + mrow) * ma.incy + (int64_t)q * ma.ldy];
        }
        int nchunk = 0;
        for (int c0 = cb; c0 < ce; c0 += CC) {
            const int cols = min(CC, ce - c0);
            const bool ok = mbar_wait_first(&full[stage], phase, wait_ns, stall_first, never);
            if (ok && live) {
                const S *st = reinterpret_cast<const S *>(ring + (size_t)stage * kChunkBytes);
#pragma unroll
                for (int u = 0; u < CPG; ++u) {
                    const int c = grp * CPG + u;
                    if (c < cols) {
                        const V pv = *reinterpret_cast<const V *>(st + c * G.ld + row0);
                        const A *gc = g + (c0 - cb + c) * KB;
                        A pr[VEC];
                        if constexpr (VEC == 4) {
                            pr[0] = pv.x; pr[1] = pv.y; pr[2] = pv.z; pr[3] = pv.w;
                        } else {
                            pr[0] = pv.x; pr[1] = pv.y;
                        }
#pragma unroll
                        for (int q = 0; q < KB; ++q) {
                            const A gq = gc[q];
#pragma unroll
                            for (int v = 0; v < VEC; ++v) part[v][q] = fma(pr[v], gq, part[v][q]);
                        }
                    }
                }
                if (kFold && ++nchunk == FOLDC) {
                    nchunk = 0;
#pragma unroll
                    for (int v = 0; v < VEC; ++v)
#pragma unroll
                        for (int q = 0; q < KB; ++q) { fold(hi[v][q], lo[v][q], part[v][q]); part[v][q] = A(0); }
                }
            }
            if (__syncthreads_or(!ok)) {      // every thread leaves together
                abort = true;
                break;
            }
            ++consumed;
            if (tid == 0 && pj < seg_hi) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                issue(stage);
            }
            if (++stage == nst) { stage = 0; phase ^= 1; }
        }
        if (abort) break;
#pragma unroll
        for (int v = 0; v < VEC; ++v)
#pragma unroll
            for (int q = 0; q < KB; ++q) fold(hi[v][q], lo[v][q], part[v][q]);
        // the column groups of a warp first (float: lanes l and l + 16 hold the same rows)
        if constexpr (RQ == 16) {
#pragma unroll
            for (int v = 0; v < VEC; ++v)
#pragma unroll
                for (int q = 0; q < KB; ++q) {
                    const A oh = __shfl_xor_sync(0xffffffffu, hi[v][q], 16);
                    const A ol = __shfl_xor_sync(0xffffffffu, lo[v][q], 16);
                    fold(hi[v][q], lo[v][q], oh);
                    lo[v][q] += ol;
                }
        }
        // every warp's partial to shared memory: red[warp][row][q][hi, lo]
        const bool holder = RQ == 16 ? lane < 16 : true;
        if (holder && live) {
#pragma unroll
            for (int v = 0; v < VEC; ++v) {
                A *rd = red + (warp * 64 + row0 + v) * KB * 2;
#pragma unroll
                for (int q = 0; q < KB; ++q) { rd[2 * q] = hi[v][q]; rd[2 * q + 1] = lo[v][q]; }
            }
        }
        __syncthreads();
        // fixed-order tree: warps (2p, 2p + 1) per thread, then lanes ^1, ^2
        if (mrow < 64) {
#pragma unroll
            for (int q = 0; q < KB; ++q) {
                A h0 = A(0), l0 = A(0);
                if (mrow < G.nrows) {
                    const A *ra = red + ((2 * mpart) * 64 + mrow) * KB * 2;
                    const A *rb = red + ((2 * mpart + 1) * 64 + mrow) * KB * 2;
                    h0 = ra[2 * q];
                    l0 = ra[2 * q + 1];
                    fold(h0, l0, rb[2 * q]);
                    l0 += rb[2 * q + 1];
                }
#pragma unroll
                for (int o = 1; o <= 2; o <<= 1) {
                    const A oh = __shfl_xor_sync(0xffffffffu, h0, o);
                    const A ol = __shfl_xor_sync(0xffffffffu, l0, o);
                    fold(h0, l0, oh);
                    l0 += ol;
                }
                if (writer && q < k && !(FAR && !yfar && ce == cb)) {
                    const A val = h0 + l0;
                    if (FAR && yfar)
                        yfar[(G.row0 + mrow) + (int64_t)q * ma.ldy] = (S)val;
                    else {
                        S *yp = ma.y + (G.row0 + mrow) * ma.incy + (int64_t)q * ma.ldy;
                        *yp = acc_y ? (S)((A)yold[q] + val) : (S)val;
                    }
                }
            }
        }
    }
    if (abort) {
        async_wait_all();
        if (tid == 0) {
            atomicExch(status, HM_DEV_WAIT_TIMEOUT);
            for (int m = consumed; m < issued; ++m) mbar_wait(&full[m % nst], (m / nst) & 1, kDrainLimitNs);
        }
    }
}

// Row segments, several right-hand sides.  One CTA (128 threads) per
// segment: the whole column-major panel is staged once in shared memory
// (16-byte streaming loads), then right-hand sides are processed in chunks
// of QC: the gathered [s ; x pieces] chunk goes to shared memory and each
// thread accumulates an RB-row x QB-column register tile.  Each piece is
// summed in plain FMA and folded into the output with a compensated
// (TwoSum) addition.
template <typename A>
struct KTile;
template <> struct KTile<float> { static constexpr int RB = 4, QB = 4, RG = 16, QG = 8; };   // 64 rows x 32 rhs
template <> struct KTile<double> { static constexpr int RB = 2, QB = 4, RG = 32, QG = 4; };  // 64 rows x 16 rhs

// n consecutive shared-memory values (16-byte aligned) converted to A.
template <typename S, typename A, int n>
__device__ __forceinline__ void load_vec(const S *p, A *out)
{
    if (sizeof(S) * n == 16) {
        if (sizeof(S) == 4) {
            const float4 v = *reinterpret_cast<const float4 *>(p);
            out[0] = (A)v.x; out[1] = (A)v.y; out[2] = (A)v.z; out[3] = (A)v.w;
        } else {
            const double2 v = *reinterpret_cast<const double2 *>(p);
            out[0] = (A)v.x; out[1] = (A)v.y;
        }
    } else if (sizeof(S) * n == 32 && sizeof(S) == 8) {
        const double2 v0 = *reinterpret_cast<const double2 *>(p), v1 = *reinterpret_cast<const double2 *>(p + 2);
        out[0] = (A)v0.x; out[1] = (A)v0.y; out[2] = (A)v1.x; out[3] = (A)v1.y;
    } else {
#pragma unroll
        for (int i = 0; i < n; ++i) out[i] = (A)p[i];
    }
}

template <typename A>
__device__ __forceinline__ void comp_add(A &hi, A &lo, A v)
{
    const A t = hi + v;
    const A bp = t - hi;
    lo += (hi - (t - bp)) + (v - bp);
    hi = t;
}

template <typename S, typename A>
__global__ void expand_k(MulArgs<S> ma, const hm_seg *segs, const hm_piece *pieces, const S *P, const A *s,
                         const A *t, int r, int maxw)
{
    constexpr int RB = KTile<A>::RB, QB = KTile<A>::QB, RG = KTile<A>::RG, QG = KTile<A>::QG;
    constexpr int QC = QB * QG;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const hm_seg G = segs[blockIdx.x];
    S *Ps = reinterpret_cast<S *>(smem_raw);                              // ld x width
    A *Gs = reinterpret_cast<A *>(smem_raw + (((size_t)64 * maxw * sizeof(S) + 31) / 32) * 32);  // QC x width
    {
        // the whole panel in flight at once
        const int n16 = (int)((int64_t)G.ld * G.width * sizeof(S) / 16);
        const char *src = reinterpret_cast<const char *>(P + G.poff);
        char *dst = reinterpret_cast<char *>(Ps);
        for (int i = threadIdx.x; i < n16; i += blockDim.x) async_copy16(dst + 16 * i, src + 16 * i);
    }
    const int W = G.width;
    const int rg = threadIdx.x % RG, qg = threadIdx.x / RG;
    for (int q0 = 0; q0 < ma.k; q0 += QC) {
        const int qc = min(QC, ma.k - q0);
        __syncthreads();                      // the previous chunk's Gs is consumed
        // gathered [s ; x pieces] chunk, right-hand side major: Gs[qq * W + c];
        // consecutive threads take consecutive entries of one right-hand side
        int col = 0;
        for (int pc = 0; pc < G.npieces; ++pc) {
            const hm_piece Q = pieces[G.piece0 + pc];
            for (int idx = threadIdx.x; idx < Q.width * QC; idx += blockDim.x) {
                const int qq = idx / Q.width, c = idx - qq * Q.width;
                A *d = Gs + qq * W + col + c;
                if (qq < qc) {
                    if (Q.kind == HM_PIECE_X)
                        async_copy<sizeof(A)>(d, ma.x + (Q.src + c) * ma.incx + (int64_t)(q0 + qq) * ma.ldx);
                    else
                        async_copy<sizeof(A)>(d, (Q.kind == HM_PIECE_TCOEF ? t : s) +
                                                     ((int64_t)Q.src * ma.k + q0 + qq) * r + c);
                } else {
                    *d = A(0);
                }
            }
            col += Q.width;
        }
        async_wait_all();
        __syncthreads();
        A hi[RB][QB], lo[RB][QB];
#pragma unroll
        for (int i = 0; i < RB; ++i)
#pragma unroll
            for (int j = 0; j < QB; ++j) { hi[i][j] = 0; lo[i][j] = 0; }
        if (rg * RB < G.ld) {
            int c = 0;
            for (int pc = 0; pc < G.npieces; ++pc) {
                const int cend = c + pieces[G.piece0 + pc].width;
                A part[RB][QB];
#pragma unroll
                for (int i = 0; i < RB; ++i)
#pragma unroll
                    for (int j = 0; j < QB; ++j) part[i][j] = 0;
                for (; c < cend; ++c) {
                    A pv[RB], gv[QB];
                    load_vec<S, A, RB>(Ps + (int64_t)c * G.ld + rg * RB, pv);
#pragma unroll
                    for (int j = 0; j < QB; ++j) gv[j] = Gs[(qg * QB + j) * W + c];
#pragma unroll
                    for (int i = 0; i < RB; ++i)
#pragma unroll
                        for (int j = 0; j < QB; ++j) part[i][j] = fma(pv[i], gv[j], part[i][j]);
                }
#pragma unroll
                for (int i = 0; i < RB; ++i)
#pragma unroll
                    for (int j = 0; j < QB; ++j) comp_add(hi[i][j], lo[i][j], part[i][j]);
            }
        }
#pragma unroll
        for (int i = 0; i < RB; ++i) {
            const int row = rg * RB + i;
            if (row >= G.nrows) continue;
#pragma unroll
            for (int j = 0; j < QB; ++j) {
                const int q = qg * QB + j;
                if (q >= qc) continue;
                S *yp = ma.y + (G.row0 + row) * ma.incy + (int64_t)(q0 + q) * ma.ldy;
                A v = hi[i][j] + lo[i][j];
                if (ma.accumulate) v += (A)(*yp);
                *yp = (S)v;
            }
        }
    }
}

#define HM_INST_PART(S, A, KB)                                                                       \
    template __global__ void expand_part<S, A, false, KB>(MulArgs<S>, const hm_seg *, int, const hm_piece *, \
                                                          const S *, const A *, const A *, int, int, S *, \
                                                          int64_t);                                     \
    template __global__ void expand_part<S, A, true, KB>(MulArgs<S>, const hm_seg *, int, const hm_piece *,  \
                                                         const S *, const A *, const A *, int, int, S *,  \
                                                         int64_t);
#define HM_INST_STREAM(S, A, KB)                                                                      \
    template __global__ void stream_part<S, A, false, KB>(MulArgs<S>, const hm_seg *, const int *,       \
                                                          const hm_piece *, const S *, const A *, const A *, \
                                                          int, int, int, int, int, S *, int *,          \
                                                          unsigned long long, int);                     \
    template __global__ void stream_part<S, A, true, KB>(MulArgs<S>, const hm_seg *, const int *,        \
                                                         const hm_piece *, const S *, const A *, const A *,  \
                                                         int, int, int, int, int, S *, int *,           \
                                                         unsigned long long, int);
#define HM_INST_FLAT(QC)                                                                                  \
    template __global__ void m2l_flat<QC>(const hm_m2l_row *, int, const hm_m2l_ent *, const double *, int, \
                                          const double *, double *, int);                                  \
    template __global__ void leaf_flat<QC>(MulArgs<double>, const hm_vpanel *, int, const double *, double *, int);
HM_INST_FLAT(1) HM_INST_FLAT(2) HM_INST_FLAT(4) HM_INST_FLAT(8)
#define HM_INST_FAR(S, A, KB)                                                                        \
    template __global__ void far_rows<S, A, KB>(MulArgs<S>, const hm_seg *, int, const hm_piece *, const S *, \
                                                const A *, const A *, int, int, S *, int64_t);
HM_INST_FAR(float, float, 4) HM_INST_FAR(float, float, 8) HM_INST_FAR(double, double, 4)
HM_INST_FAR(double, double, 8) HM_INST_FAR(double, double, 1) HM_INST_FAR(double, double, 2)
HM_INST_FAR(float, float, 2)
#define HM_INST_MV(S, A)                                                                             \
    template __global__ void leaf_up<S, A, 1>(MulArgs<S>, const hm_vpanel *, int, const S *, A *, int, int, int, LeafParts<A>); \
    template __global__ void leaf_up<S, A, 2>(MulArgs<S>, const hm_vpanel *, int, const S *, A *, int, int, int, LeafParts<A>); \
    template __global__ void leaf_up<S, A, 4>(MulArgs<S>, const hm_vpanel *, int, const S *, A *, int, int, int, LeafParts<A>); \
    template __global__ void leaf_up<S, A, 8>(MulArgs<S>, const hm_vpanel *, int, const S *, A *, int, int, int, LeafParts<A>); \
    template __global__ void m2l<S, A, 1>(const hm_m2l_row *, int, const hm_m2l_ent *, const S *, int,    \
                                          const A *, A *, int, int);                                    \
    template __global__ void m2l<S, A, 2>(const hm_m2l_row *, int, const hm_m2l_ent *, const S *, int,    \
                                          const A *, A *, int, int);                                    \
    template __global__ void m2l<S, A, 4>(const hm_m2l_row *, int, const hm_m2l_ent *, const S *, int,    \
                                          const A *, A *, int, int);                                    \
    template __global__ void m2l<S, A, 8>(const hm_m2l_row *, int, const hm_m2l_ent *, const S *, int,    \
                                          const A *, A *, int, int);                                    \
    template __global__ void m2l_k<S, A, 8>(const hm_m2l_row *, int, const hm_m2l_ent *, const S *, int,  \
                                            const A *, A *, int, int);                                  \
    HM_INST_PART(S, A, 1) HM_INST_PART(S, A, 2) HM_INST_PART(S, A, 4) HM_INST_PART(S, A, 8)               \
    HM_INST_STREAM(S, A, 1) HM_INST_STREAM(S, A, 2) HM_INST_STREAM(S, A, 4) HM_INST_STREAM(S, A, 8)       \
    template __global__ void expand_k<S, A>(MulArgs<S>, const hm_seg *, const hm_piece *, const S *,  \
                                            const A *, const A *, int, int);                            \
    template __global__ void xfer_up_band<A, 1>(const hm_task *, const hm_step *, const hm_xfer *, const A *, \
                                                A *, int, int);                                         \
    template __global__ void xfer_up_band<A, 2>(const hm_task *, const hm_step *, const hm_xfer *, const A *, \
                                                A *, int, int);                                         \
    template __global__ void xfer_up_band<A, 4>(const hm_task *, const hm_step *, const hm_xfer *, const A *, \
                                                A *, int, int);                                         \
    template __global__ void xfer_up_band<A, 8>(const hm_task *, const hm_step *, const hm_xfer *, const A *, \
                                                A *, int, int);                                         \
    template __global__ void xfer_down_band<A, 1>(const hm_task *, const hm_step *, const hm_xfer *,        \
                                                  const A *, A *, int, int);                            \
    template __global__ void xfer_down_band<A, 2>(const hm_task *, const hm_step *, const hm_xfer *,        \
                                                  const A *, A *, int, int);                            \
    template __global__ void xfer_down_band<A, 4>(const hm_task *, const hm_step *, const hm_xfer *,        \
                                                  const A *, A *, int, int);                            \
    template __global__ void xfer_down_band<A, 8>(const hm_task *, const hm_step *, const hm_xfer *,        \
                                                  const A *, A *, int, int);                            \
    template __global__ void xfer_up_task<A, 1>(const hm_task *, const hm_step *, const hm_xfer *, const A *, \
                                                A *, int, int, int);                                    \
    template __global__ void xfer_up_task<A, 2>(const hm_task *, const hm_step *, const hm_xfer *, const A *, \
                                                A *, int, int, int);                                    \
    template __global__ void xfer_up_task<A, 4>(const hm_task *, const hm_step *, const hm_xfer *, const A *, \
                                                A *, int, int, int);                                    \
    template __global__ void xfer_up_task<A, 8>(const hm_task *, const hm_step *, const hm_xfer *, const A *, \
                                                A *, int, int, int);                                    \
    template __global__ void xfer_down_task<A, 1>(const hm_task *, const hm_step *, const hm_xfer *,        \
                                                  const A *, A *, int, int, int);                       \
    template __global__ void xfer_down_task<A, 2>(const hm_task *, const hm_step *, const hm_xfer *,        \
                                                  const A *, A *, int, int, int);                       \
    template __global__ void xfer_down_task<A, 4>(const hm_task *, const hm_step *, const hm_xfer *,        \
                                                  const A *, A *, int, int, int);                       \
    template __global__ void xfer_down_task<A, 8>(const hm_task *, const hm_step *, const hm_xfer *,        \
                                                  const A *, A *, int, int, int);
HM_INST_MV(double, double)
HM_INST_MV(float, float)
template __global__ void add_far<double>(MulArgs<double>, int64_t, const double *, int64_t);
template __global__ void add_far<float>(MulArgs<float>, int64_t, const float *, int64_t);

// ============================================================== direct sums

// out[q] = sum_j f(x[rows[q]], y[j]) b[j] in FP64 with double-double
// accumulation; one CTA per row.  An exact-as-possible dense evaluation used
// to state the error of the compressed product.
__global__ void direct_rows(int kid, const double *x, int64_t nx, const double *y, int64_t ny,
                           const double *b, const int64_t *rows, int64_t nrows, double *out)
{
    __shared__ double hs[32], ls[32];
    const int64_t q = blockIdx.x;
    if (q >= nrows) return;
    const int64_t row = rows[q];
    if (row < 0 || row >= nx) {           // invalid row index: report NaN
        if (threadIdx.x == 0) out[q] = __longlong_as_double(0x7ff8000000000000LL);
        return;
    }
    const double xi = x[row];
    double s = 0.0, c = 0.0;
    for (int64_t j = threadIdx.x; j < ny; j += blockDim.x) {
        const double f = kernel_eval(kid, xi, y[j]);
        const double p = __dmul_rn(f, b[j]);
        const double pe = fma(f, b[j], -p);
        const double t = __dadd_rn(s, p);
        const double bp = __dsub_rn(t, s);
        const double se = __dadd_rn(__dsub_rn(s, __dsub_rn(t, bp)), __dsub_rn(p, bp));
        s = t;
        c = __dadd_rn(c, __dadd_rn(se, pe));
    }
    // combine (s, c) pairs across the block
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int o = 16; o; o >>= 1) {
        const double s2 = __shfl_down_sync(0xffffffffu, s, o);
        const double c2 = __shfl_down_sync(0xffffffffu, c, o);
        const double t = __dadd_rn(s, s2);
        const double bp = __dsub_rn(t, s);
        const double se = __dadd_rn(__dsub_rn(s, __dsub_rn(t, bp)), __dsub_rn(s2, bp));
        s = t;
        c = __dadd_rn(__dadd_rn(c, c2), se);
    }
    if (lane == 0) { hs[wid] = s; ls[wid] = c; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double S = 0.0, C = 0.0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
            const double t = __dadd_rn(S, hs[k]);
            const double bp = __dsub_rn(t, S);
            const double se = __dadd_rn(__dsub_rn(S, __dsub_rn(t, bp)), __dsub_rn(hs[k], bp));
            S = t;
            C = __dadd_rn(__dadd_rn(C, ls[k]), se);
        }
        out[q] = __dadd_rn(S, C);
    }
}

}  // namespace hm
