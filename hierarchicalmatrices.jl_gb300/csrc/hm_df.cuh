// Device bodies of the double-float (HM_DF64) tree passes, for the stage kernels
// (hm_df.cu) and the two-launch schedule (hm_fused.cu).  Written for sm_103a.
#pragma once
#include "hm_async.cuh"
#include "hm_kernels.cuh"
#include "hm_tree.cuh"

namespace hm {
namespace {

__device__ __forceinline__ float2 df_split(double v)
{
    const float h = __double2float_rn(v);
    return make_float2(h, __double2float_rn(__dsub_rn(v, (double)h)));
}

// (sh, sl) += (ph + pl) (gh + gl)
__device__ __forceinline__ void df_fma(float &sh, float &sl, float ph, float pl, float gh, float gl)
{
    const float h = __fmul_rn(ph, gh);
    float e = __fmaf_rn(ph, gh, -h);
    e = __fmaf_rn(ph, gl, e);
    e = __fmaf_rn(pl, gh, e);
    const float s = __fadd_rn(sh, h);
    const float bp = __fsub_rn(s, sh);
    float t = __fadd_rn(__fsub_rn(sh, __fsub_rn(s, bp)), __fsub_rn(h, bp));
    t = __fadd_rn(t, __fadd_rn(sl, e));
    sh = __fadd_rn(s, t);
    sl = __fsub_rn(t, __fsub_rn(sh, s));
}

// (sh, sl) += sum over columns [c0, c1) of a segment's panel (ld rows, two per lane) times
// g[c * KB + q]; `groups`: low segments' columns dealt out to lane groups (ring_groups),
// the groups' sums in every group at the end.
template <int KB>
__device__ __forceinline__ void df_columns(const float2 *Pg, int ld, const float2 *g, int c0, int c1, bool groups,
                                           float (&sh)[2][KB], float (&sl)[2][KB])
{
    const int lane = threadIdx.x & 31;
    const int cg = groups ? ring_groups(ld) : 1, lanes = 32 / cg, lr = lane & (lanes - 1);
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int q = 0; q < KB; ++q) sh[j][q] = sl[j][q] = 0.f;
    const float4 *base = reinterpret_cast<const float4 *>(Pg + 2 * lr);
    const int64_t ld2 = ld / 2;                                // float4 (two pairs) per column step
    auto use = [&](const float4 &p, int cc) {
        const float2 *gc = g + cc * KB;
#pragma unroll
        for (int q = 0; q < KB; ++q) {
            const float2 gq = gc[q];
            df_fma(sh[0][q], sl[0][q], p.x, p.y, gq.x, gq.y);
            df_fma(sh[1][q], sl[1][q], p.z, p.w, gq.x, gq.y);
        }
    };
    if (cg > 1) {
        if (2 * lr < ld) {
            constexpr int U = 4;
            for (int c = c0 + lane / lanes; c < c1; c += U * cg) {
                float4 p[U];
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (c + u * cg < c1) p[u] = __ldcs(base + ld2 * (c + u * cg));
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (c + u * cg < c1) use(p[u], c + u * cg);
            }
        }
        for (int o = lanes; o < 32; o <<= 1) {
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int q = 0; q < KB; ++q) {
                    const float a = sh[j][q], so = __shfl_xor_sync(0xffffffffu, a, o);
                    const float l = __fadd_rn(sl[j][q], __shfl_xor_sync(0xffffffffu, sl[j][q], o));
                    float s, e;
                    two_sum(a, so, s, e);
                    const float t = __fadd_rn(e, l);
                    sh[j][q] = __fadd_rn(s, t);
                    sl[j][q] = __fsub_rn(t, __fsub_rn(sh[j][q], s));
                }
        }
    } else if (2 * lane < ld) {
        constexpr int U = KB <= 2 ? 16 : 8;                    // loads in flight per lane
        int c = c0;
        for (; c + U <= c1; c += U) {
            float4 p[U];
#pragma unroll
            for (int u = 0; u < U; ++u) p[u] = __ldcs(base + ld2 * (c + u));
#pragma unroll
            for (int u = 0; u < U; ++u) use(p[u], c + u);
        }
        for (; c < c1; ++c) use(__ldcs(base + ld2 * c), c);
    }
}

// One basis panel by one warp (leaf_up_df); xs: cap pairs of this warp.
__device__ __forceinline__ void leaf_panel_df(const MulArgs<double> &ma, const hm_vpanel P, const float2 *V, double *t,
                                              int r, int cap, float2 *xs)
{
    const int lane = threadIdx.x & 31;
    const float2 *Vp = V + P.off;
    const double *xsrc = ma.xin ? ma.xin : ma.x;
    double *xcopy = ma.xin ? const_cast<double *>(ma.x) : nullptr;
    const int nr = min((int)P.nrows, cap);
    for (int q = 0; q < ma.k; ++q) {
        for (int j = lane; j < P.nrows; j += 32) {
            const int64_t e = (P.row0 + j) * ma.incx + (int64_t)q * ma.ldx;
            const double v = xsrc[e];
            if (xcopy) xcopy[e] = v;
            if (j < nr) xs[j] = df_split(v);
        }
        __syncwarp();
        if (lane < P.width) {
            float sh = 0.f, sl = 0.f;
            int j = 0;
            for (; j + 8 <= nr; j += 8) {
                float2 v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) v[u] = Vp[(int64_t)(j + u) * P.ld + lane];
#pragma unroll
                for (int u = 0; u < 8; ++u) df_fma(sh, sl, v[u].x, v[u].y, xs[j + u].x, xs[j + u].y);
            }
            for (; j < nr; ++j) {
                const float2 v = Vp[(int64_t)j * P.ld + lane];
                df_fma(sh, sl, v.x, v.y, xs[j].x, xs[j].y);
            }
            // rows past the staged ones (panels longer than cap) straight from x
            for (j = nr; j < P.nrows; ++j) {
                const float2 v = Vp[(int64_t)j * P.ld + lane];
                const float2 xv = df_split(xsrc[(P.row0 + j) * ma.incx + (int64_t)q * ma.ldx]);
                df_fma(sh, sl, v.x, v.y, xv.x, xv.y);
            }
            t[((int64_t)P.slot * ma.k + q) * r + P.col0 + lane] = __dadd_rn((double)sh, (double)sl);
        }
        __syncwarp();
    }
}

// One row slot's far field by one warp (m2l_df_ring, rank 20); ring: NS blocks
// and ts: 32 pairs of this warp.
template <int NS>
__device__ __forceinline__ void m2l_row_df(const hm_m2l_row R, const hm_m2l_ent *ents, const float2 *F,
                                           const double *t, double *s, int k, float2 *ring, float2 *ts)
{
    constexpr int R20 = 20, BLK = R20 * R20;
    const int lane = threadIdx.x & 31;
    const int ne = R.end - R.begin;
    auto issue = [&](int i, int stage) {
        const hm_m2l_ent E = ents[R.begin + i];
        float2 *dst = ring + stage * BLK;
        const float2 *src = F + E.foff;
        if ((E.foff & 1) == 0) {
            for (int c = lane; c < BLK / 2; c += 32) async_copy16(dst + 2 * c, src + 2 * c);
        } else {
            for (int c = lane; c < BLK; c += 32) async_copy<8>(dst + c, src + c);
        }
    };
    for (int q = 0; q < k; ++q) {
        float sh = 0.f, sl = 0.f;
        double tc = 0.0;
        if (ne > 0 && lane < R20) tc = t[((int64_t)ents[R.begin].yslot * k + q) * R20 + lane];
#pragma unroll
        for (int i = 0; i < NS - 1; ++i) {
            if (i < ne) issue(i, i);
            async_commit();
        }
        for (int e = 0; e < ne; ++e) {
            const int ei = e + NS - 1;
            if (ei < ne) issue(ei, ei % NS);
            async_commit();
            asm volatile("cp.async.wait_group %0;" ::"n"(NS - 1) : "memory");
            if (lane < R20) ts[lane] = df_split(tc);
            __syncwarp();                                      // block e and the coefficients visible
            double tn = 0.0;
            if (e + 1 < ne && lane < R20) tn = t[((int64_t)ents[R.begin + e + 1].yslot * k + q) * R20 + lane];
            if (lane < R20) {
                const float2 *f = ring + (e % NS) * BLK + lane;
#pragma unroll
                for (int n = 0; n < R20; ++n) {
                    const float2 v = f[R20 * n];
                    df_fma(sh, sl, v.x, v.y, ts[n].x, ts[n].y);
                }
            }
            __syncwarp();                                      // the stage and ts are free again
            tc = tn;
        }
        async_wait_all();
        __syncwarp();
        if (lane < R20) s[((int64_t)R.slot * k + q) * R20 + lane] = __dadd_rn((double)sh, (double)sl);
    }
}

// One band task of one right-hand side by the CTA (xfer_df): the external
// inputs into the local vectors L, then the task's levels.
template <bool UP>
__device__ __forceinline__ void xfer_df_fetch(const TaskRecs &R, const double *coef, float2 *L, int r, int k, int q)
{
    const int nrec = R.nrec;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int rec = warp; rec < nrec; rec += nw) {
        const hm_xfer X = R.x[rec];
        if (lane >= r) continue;
#pragma unroll
        for (int c = 0; c < (UP ? 2 : 3); ++c) {
            int lc, slot;
            if (UP) {
                lc = c ? (X.pad >> 16) : (X.pad & 0xffff);
                slot = c ? X.c1 : X.c0;
                if (lc < nrec) continue;                       // produced by an earlier level of this task
            } else if (c < 2) {
                lc = 2 * rec + c;                              // children start from their far-field values
                slot = c ? X.c1 : X.c0;
            } else {
                lc = X.pad;
                slot = X.slot;
                if (lc < 2 * nrec) continue;                   // a child of an earlier level of this task
            }
            L[lc * r + lane] = df_split(coef[((int64_t)slot * k + q) * r + lane]);
        }
    }
}

template <bool UP, int RC>
__device__ __forceinline__ void xfer_df_levels(const TaskRecs &R, const float2 *Ts, double *coef, float2 *L, int rr,
                                               int k, int q)
{
    const int r = RC ? RC : rr;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int st = 0; st < R.nsteps; ++st) {
        const hm_step S = R.step[st];
        for (int e = S.e0 + warp; e < S.e1; e += nw) {
            const hm_xfer X = R.x[e];
            if (lane >= r) continue;
            if (UP) {
                const float2 *c0 = L + (X.pad & 0xffff) * r, *c1 = L + (X.pad >> 16) * r;
                float sh = 0.f, sl = 0.f;
#pragma unroll 4
                for (int mp = 0; mp < r; ++mp) {
                    const float2 a0 = Ts[mp * r + lane], a1 = Ts[r * r + mp * r + lane];
                    df_fma(sh, sl, a0.x, a0.y, c0[mp].x, c0[mp].y);
                    df_fma(sh, sl, a1.x, a1.y, c1[mp].x, c1[mp].y);
                }
                L[e * r + lane] = make_float2(sh, sl);
                coef[((int64_t)X.slot * k + q) * r + lane] = __dadd_rn((double)sh, (double)sl);
            } else {
                const float2 *p = L + X.pad * r;
                float2 *o0 = L + (2 * e) * r, *o1 = o0 + r;
                float h0 = o0[lane].x, l0 = o0[lane].y, h1 = o1[lane].x, l1 = o1[lane].y;
#pragma unroll 4
                for (int m = 0; m < r; ++m) {
                    const float2 t0 = Ts[lane * r + m], t1 = Ts[r * r + lane * r + m];
                    df_fma(h0, l0, t0.x, t0.y, p[m].x, p[m].y);
                    df_fma(h1, l1, t1.x, t1.y, p[m].x, p[m].y);
                }
                o0[lane] = make_float2(h0, l0);
                o1[lane] = make_float2(h1, l1);
                coef[((int64_t)X.c0 * k + q) * r + lane] = __dadd_rn((double)h0, (double)l0);
                coef[((int64_t)X.c1 * k + q) * r + lane] = __dadd_rn((double)h1, (double)l1);
            }
        }
        __syncthreads();
    }
}

}  // namespace
}  // namespace hm
