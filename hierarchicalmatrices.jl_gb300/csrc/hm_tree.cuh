// Device bodies of the tree passes and of a row segment's sums, for the stage
// kernels (one launch per stage, hm_kernels.cu, hm_df.cu) and the two-launch
// schedule of small matrices (hm_fused.cu).  Written for sm_103a.
#pragma once
#include "hm_async.cuh"
#include "hm_kernels.cuh"
#include "hm_plan.h"

namespace hm {
namespace {

// N consecutive values from 16-byte aligned shared memory, as 16-byte loads
// where N values fill them (the chunks of right-hand sides below are stored
// right-hand side fastest, so that one step's N values are adjacent).
template <int N, typename A>
__device__ __forceinline__ void ld_vec(const A *p, A *v)
{
    if constexpr (sizeof(A) == 4 && N % 4 == 0) {
#pragma unroll
        for (int i = 0; i < N / 4; ++i) {
            const float4 w = reinterpret_cast<const float4 *>(p)[i];
            v[4 * i] = w.x; v[4 * i + 1] = w.y; v[4 * i + 2] = w.z; v[4 * i + 3] = w.w;
        }
    } else if constexpr (sizeof(A) == 8 && N % 2 == 0) {
#pragma unroll
        for (int i = 0; i < N / 2; ++i) {
            const double2 w = reinterpret_cast<const double2 *>(p)[i];
            v[2 * i] = w.x; v[2 * i + 1] = w.y;
        }
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = p[i];
    }
}

// Adds `n` consecutive partial slots of lane's column in order, eight loads in
// flight, for one right-hand side.
template <typename A>
__device__ __forceinline__ A sum_parts(const A *sums, int64_t first, int n, int k, int q, int width, int lane)
{
    A v = A(0);
    const A *p = sums + (first * k + q) * width + lane;
    const int64_t step = (int64_t)k * width;
    int i = 0;
    for (; i + 8 <= n; i += 8) {
        A u[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) u[j] = __ldcg(p + (i + j) * step);
#pragma unroll
        for (int j = 0; j < 8; ++j) v += u[j];
    }
    for (; i < n; ++i) v += __ldcg(p + i * step);
    return v;
}

// True in every lane of the warp that arrives last of `n` at *count, which is
// set back to zero for the next product; the others' writes are then visible.
__device__ __forceinline__ bool last_arrival(int *count, int n, int lane)
{
    __threadfence();
    __syncwarp();
    int old = 0;
    if (lane == 0) {
        old = atomicAdd(count, 1);
        if (old == n - 1) *count = 0;
    }
    old = __shfl_sync(0xffffffffu, old, 0);
    __threadfence();
    return old == n - 1;
}

// t[slot][col0 + m] = (V^T x)[m] for each explicit basis panel.  One warp
// per panel, looping over chunks of QC right-hand sides; lane m owns column m
// of the row-major panel (width <= 32, row stride ld).  With at most 16
// columns 32 / width rows go at once, one per lane group, and the groups are
// added at the end (an FP64 warp instruction takes 64 cycles of its pipe
// whatever lanes are active).  Panels of more than 128 rows (the low-rank
// factors of a user-assembled matrix) come as parts of at most 128 rows, one
// warp each, whose sums the last warp of a group to finish adds in part order
// (hm_vpart): one warp per 8,192-row panel took 1.30 ms of a 16,384-row FP64
// HODLR product, latency of one serial FP64 chain with 508 of 608
// sub-partitions idle.  Panels of up to cap
// rows and wcap columns (the handle's largest, up to 128 rows) are staged
// once in shared memory (cp.async) and the chunks' x values double-buffered
// beside them; longer panels are read directly.  Plain FMA accumulation
// (the coefficients feed only the far field).  Coefficients of a slot are r
// apart per right-hand side (kt of them in all, ma.k of them here); those past a block of lower rank are set to zero
// (hm_vpanel.zeros), because the far-field blocks read all r.
// smem: leaf_up_warp_bytes of this warp.
template <typename S, typename A, int QC>
__device__ __forceinline__ void leaf_panel(const MulArgs<S> &ma, int kt, const hm_vpanel P, const hm_vpart part,
                                           const S *V, A *t, int r, int cap, int wcap, unsigned char *smem,
                                           const LeafParts<A> &lp)
{
    const int lane = threadIdx.x & 31;
    const int pw = P.width;
    const S *Vp = V + P.off;
    const int k = ma.k;
    // right-hand sides read from xin (and copied into x as they pass) or from x
    const S *xsrc = ma.xin ? ma.xin : ma.x;
    S *xcopy = ma.xin ? const_cast<S *>(ma.x) : nullptr;
    // a whole panel's sums are its coefficients, a part's go to its partial slot
    A *out = part.nparts ? lp.sums + (int64_t)part.part * k * lp.width : t + (int64_t)P.slot * kt * r + P.col0;
    const int ldo = part.nparts ? lp.width : r;
    auto store = [&](int q0, int qc, PlainAcc<A> *acc) {
        if (lane < pw + P.zeros) {
#pragma unroll
            for (int qq = 0; qq < QC; ++qq)
                if (qq < qc) out[(int64_t)(q0 + qq) * ldo + lane] = lane < pw ? acc[qq].value() : A(0);
        }
    };
    if (P.nrows <= cap && P.ld == pw && pw <= wcap) {
        // the panel once; x chunks of QC right-hand sides double-buffered,
        // row major xs[b][j * QC + qq] (lanes walk rows)
        S *Vs = reinterpret_cast<S *>(smem);
        A *xs = reinterpret_cast<A *>(Vs + cap * wcap);
        const int nel = P.nrows * pw;
        if (sizeof(S) * nel % 16 == 0 && (P.off * sizeof(S)) % 16 == 0) {
            const char *src = reinterpret_cast<const char *>(Vp);
            char *dst = reinterpret_cast<char *>(Vs);
            for (int i = lane; i < (int)(nel * sizeof(S) / 16); i += 32) async_copy16(dst + 16 * i, src + 16 * i);
        } else {
            for (int i = lane; i < nel; i += 32) async_copy<sizeof(S)>(Vs + i, Vp + i);
        }
        auto fetch = [&](int q0, int b) {
            const int qc = min(QC, k - q0);
            A *d = xs + b * cap * QC;
#pragma unroll
            for (int qq = 0; qq < QC; ++qq)
                for (int j = lane; j < P.nrows; j += 32) {
                    const int64_t e = (P.row0 + j) * ma.incx + (int64_t)(q0 + qq) * ma.ldx;
                    if (qq >= qc) {
                        d[j * QC + qq] = A(0);
                    } else if (xcopy) {
                        // host-mapped source: plain loads, stored here and into x
                        const S v = xsrc[e];
                        d[j * QC + qq] = (A)v;
                        xcopy[e] = v;
                    } else {
                        async_copy<sizeof(A)>(d + j * QC + qq, ma.x + e);
                    }
                }
            async_commit();
        };
        fetch(0, 0);
        for (int q0 = 0, b = 0; q0 < k; q0 += QC, b ^= 1) {
            if (q0 + QC < k) {
                fetch(q0 + QC, b ^ 1);
                asm volatile("cp.async.wait_group 1;" ::: "memory");
            } else {
                async_wait_all();
            }
            __syncwarp();
            PlainAcc<A> acc[QC];
#pragma unroll
            for (int qq = 0; qq < QC; ++qq) acc[qq].zero();
            const A *xb = xs + b * cap * QC;
            auto row = [&](int j, int m) {
                const A v = (A)Vs[j * pw + m];
                A xv[QC];
                ld_vec<QC>(xb + j * QC, xv);
#pragma unroll
                for (int qq = 0; qq < QC; ++qq) acc[qq].add(v, xv[qq]);
            };
            if (pw > 16) {
                if (lane < pw)
                    for (int j = 0; j < P.nrows; ++j) row(j, lane);
            } else {
                const int groups = 32 / pw, jr = lane / pw, m = lane % pw;
                if (jr < groups)
                    for (int j = jr; j < P.nrows; j += groups) row(j, m);
#pragma unroll
                for (int qq = 0; qq < QC; ++qq) {         // add the row groups, in order
                    A v = acc[qq].s;
                    for (int g = 1; g < groups; ++g) v += __shfl_sync(0xffffffffu, acc[qq].s, (lane + g * pw) & 31);
                    acc[qq].s = v;
                }
            }
            store(q0, min(QC, k - q0), acc);
            __syncwarp();                                 // buffer b is refilled next
        }
    } else {
        for (int q0 = 0; q0 < k; q0 += QC) {
            const int qc = min(QC, k - q0);
            PlainAcc<A> acc[QC];
#pragma unroll
            for (int qq = 0; qq < QC; ++qq) acc[qq].zero();
            if (lane < pw) {
                const S *col = Vp + lane;
                for (int j = 0; j < P.nrows; ++j) {
                    const A v = (A)col[(int64_t)j * P.ld];
#pragma unroll
                    for (int qq = 0; qq < QC; ++qq)
                        if (qq < qc) acc[qq].add(v, (A)xsrc[(P.row0 + j) * ma.incx + (int64_t)(q0 + qq) * ma.ldx]);
                }
            }
            if (xcopy)
                for (int qq = 0; qq < qc; ++qq)
                    for (int j = lane; j < P.nrows; j += 32) {
                        const int64_t e = (P.row0 + j) * ma.incx + (int64_t)(q0 + qq) * ma.ldx;
                        xcopy[e] = xsrc[e];
                    }
            store(q0, qc, acc);
        }
    }
    if (part.nparts && last_arrival(lp.count + part.group, part.nparts, lane)) {
        A *tp = t + (int64_t)P.slot * kt * r + P.col0 + lane;
        A *gp = lp.sums + (int64_t)(part.gpart + part.group - part.group0) * k * lp.width + lane;
        if (lane < pw + P.zeros) {                             // (the parts hold the zeros too)
            for (int q = 0; q < k; ++q) {
                const A v = sum_parts(lp.sums, part.part0, part.nparts, k, q, lp.width, lane);
                if (part.ngroups == 1) tp[(int64_t)q * r] = v;
                else gp[(int64_t)q * lp.width] = v;
            }
        }
        __syncwarp();
        if (part.ngroups > 1 && last_arrival(lp.count + part.panel, part.ngroups, lane) && lane < pw + P.zeros)
            for (int q = 0; q < k; ++q)
                tp[(int64_t)q * r] = sum_parts(lp.sums, part.gpart, part.ngroups, k, q, lp.width, lane);
    }
}

// One band task's records in shared memory.  A level walk that reads its steps
// and records from global memory pays two dependent L2 round trips per level,
// more than the level's arithmetic; they are constant, so a kernel stages them
// before it waits for its inputs.
constexpr int kTaskRecs = (1 << kBandLevels) - 1;
struct TaskRecs {
    hm_xfer x[kTaskRecs];
    hm_step step[kBandLevels];      // record ranges of the levels, relative to x
    int nrec, nsteps;
};
// Fills R for one task by the CTA (a barrier is needed before it is read).
__device__ __forceinline__ void load_task(const hm_task *task, const hm_step *steps, const hm_xfer *ents, TaskRecs &R)
{
    const hm_task tk = *task;
    const int e0 = steps[tk.step0].e0, nrec = steps[tk.step1 - 1].e1 - e0, ns = tk.step1 - tk.step0;
    const int tid = threadIdx.x;
    if (tid < nrec) R.x[tid] = ents[e0 + tid];
    if (tid < ns) {
        const hm_step st = steps[tk.step0 + tid];
        R.step[tid] = hm_step{st.e0 - e0, st.e1 - e0};
    }
    if (tid == 0) { R.nrec = nrec; R.nsteps = ns; }
}

// Band tasks with shared-memory-resident coefficients, one CTA per (task,
// chunk of QC right-hand sides): the task's external inputs (and T) are fetched
// once with cp.async, every level then
// reads and writes shared memory only, with a CTA barrier between levels;
// each coefficient the task produces is also written to global memory.
// Task-local numbering (records' pad, set by the planner): upward, record i
// produces local i and reads locals pad & 0xffff, pad >> 16; downward,
// record i's children are locals 2i, 2i + 1 and its parent is local pad.
// Upward, L holds r x QC values per local, right-hand side fastest
// (L[local][m][qq]); downward QC x r (L[local][qq][m]).
template <typename A, int QC>
__device__ __forceinline__ void xfer_up_fetch(const TaskRecs &R, const A *t, A *L, int r, int k, int q0)
{
    const int qc = min(QC, k - q0);
    // external children: warps take records, lanes coefficients
    for (int rec = threadIdx.x >> 5; rec < R.nrec; rec += blockDim.x >> 5) {
        const hm_xfer X = R.x[rec];
        const int ln = threadIdx.x & 31;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int lc = c ? (X.pad >> 16) : (X.pad & 0xffff);
            if (lc < R.nrec || ln >= r) continue;         // produced by an earlier level of this task
            const A *src = t + ((int64_t)(c ? X.c1 : X.c0) * k + q0) * r + ln;
            A *d = L + (int64_t)lc * QC * r + ln * QC;
#pragma unroll
            for (int qq = 0; qq < QC; ++qq) {
                if (qq < qc) async_copy<sizeof(A)>(d + qq, src + (int64_t)qq * r);
                else d[qq] = A(0);
            }
        }
    }
}

// The level walks and the far-field rows take the rank as a template argument
// RC (20, the rank of FP64 compression; 0: any, read at run time): with the
// inner loops unrolled their shared-memory loads issue ahead of the FMAs that
// use them: the level walks are latency bound (a 100,003 x 77,777 FP32 matrix
// with 3 right-hand sides 84.6 -> 74.6 us per product, n = 2^20 with one 233 ->
// 226 us).
// f(e, m) for every output m of the records e of a step: a warp per record, lane m;
// FP64 rank 20 a thread per output, 160 of them for eight records (an FP64 warp
// instruction takes as long for 20 lanes as for 32).
template <typename A, int RC, typename F>
__device__ __forceinline__ void task_outputs(const hm_step S, int r, F f)
{
    if constexpr (sizeof(A) == 8 && RC == 20) {
        for (int u = threadIdx.x; u < (S.e1 - S.e0) * RC; u += blockDim.x) f(S.e0 + u / RC, u % RC);
    } else {
        const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
        if (lane >= r) return;
        for (int e = S.e0 + (threadIdx.x >> 5); e < S.e1; e += nw) f(e, lane);
    }
}

template <typename A, int QC, int RC>
__device__ __forceinline__ void xfer_up_levels(const TaskRecs &R, const A *Ts, A *t, A *L, int rr, int k, int q0)
{
    const int r = RC ? RC : rr;
    const int qc = min(QC, k - q0);
    for (int st = 0; st < R.nsteps; ++st) {
        const hm_step S = R.step[st];
        task_outputs<A, RC>(S, r, [&](int e, int lane) {
            const hm_xfer X = R.x[e];
            const A *c0 = L + (int64_t)(X.pad & 0xffff) * QC * r;
            const A *c1 = L + (int64_t)(X.pad >> 16) * QC * r;
            A *out = L + (int64_t)e * QC * r;
            // one sum per child: an FMA per term (a0 v0 + a1 v1 in one expression
            // is three operations), and neither sum is rounded more often than
            // when the pair was added first
            A s0[QC], s1[QC];
#pragma unroll
            for (int qq = 0; qq < QC; ++qq) s0[qq] = s1[qq] = 0;
#pragma unroll(RC ? RC : 4)
            for (int mp = 0; mp < r; ++mp) {
                const A a0 = Ts[mp * r + lane], a1 = Ts[r * r + mp * r + lane];
                A v0[QC], v1[QC];
                ld_vec<QC>(c0 + mp * QC, v0);
                ld_vec<QC>(c1 + mp * QC, v1);
#pragma unroll
                for (int qq = 0; qq < QC; ++qq) {
                    s0[qq] = fma(a0, v0[qq], s0[qq]);
                    s1[qq] = fma(a1, v1[qq], s1[qq]);
                }
            }
#pragma unroll
            for (int qq = 0; qq < QC; ++qq) {
                const A sum = s0[qq] + s1[qq];
                out[lane * QC + qq] = sum;
                if (qq < qc) t[((int64_t)X.slot * k + q0 + qq) * r + lane] = sum;
            }
        });
        __syncthreads();
    }
}

template <typename A, int QC>
__device__ __forceinline__ void xfer_down_fetch(const TaskRecs &R, const A *s, A *L, int r, int k, int q0)
{
    const int qc = min(QC, k - q0);
    // children start from their far-field (m2l) coefficients; external parents as computed
    // warps take records, lanes coefficients
    for (int rec = threadIdx.x >> 5; rec < R.nrec; rec += blockDim.x >> 5) {
        const hm_xfer X = R.x[rec];
        const int ln = threadIdx.x & 31;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            int lc, slot;
            if (c < 2) {
                lc = 2 * rec + c;
                slot = c ? X.c1 : X.c0;
            } else {
                lc = X.pad;
                slot = X.slot;
                if (lc < 2 * R.nrec) continue;            // a child of an earlier level of this task
            }
            if (ln >= r) continue;
            const A *src = s + ((int64_t)slot * k + q0) * r + ln;
            A *d = L + (int64_t)lc * QC * r + ln;
#pragma unroll
            for (int qq = 0; qq < QC; ++qq) {
                if (qq < qc) async_copy<sizeof(A)>(d + qq * r, src + (int64_t)qq * r);
                else d[qq * r] = A(0);
            }
        }
    }
}

template <typename A, int QC, int RC>
__device__ __forceinline__ void xfer_down_levels(const TaskRecs &R, const A *Ts, A *s, A *L, int rr, int k, int q0)
{
    const int r = RC ? RC : rr;
    const int qc = min(QC, k - q0);
    for (int st = 0; st < R.nsteps; ++st) {
        const hm_step S = R.step[st];
        task_outputs<A, RC>(S, r, [&](int e, int lane) {
            const hm_xfer X = R.x[e];
            const A *p = L + (int64_t)X.pad * QC * r;
            A *o0 = L + (int64_t)(2 * e) * QC * r;
            A *o1 = o0 + QC * r;
            A a0[QC], a1[QC];
#pragma unroll
            for (int qq = 0; qq < QC; ++qq) { a0[qq] = 0; a1[qq] = 0; }
            const A *Tl = Ts + lane * r, *Tr = Tl + r * r;
            if constexpr (RC % 4 == 0 && RC > 0) {
                // rows of T and of the parent in 16-byte loads
#pragma unroll
                for (int m = 0; m < RC; m += 4) {
                    A t0[4], t1[4];
                    ld_vec<4>(Tl + m, t0);
                    ld_vec<4>(Tr + m, t1);
#pragma unroll
                    for (int qq = 0; qq < QC; ++qq) {
                        A v[4];
                        ld_vec<4>(p + qq * RC + m, v);
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            a0[qq] += t0[u] * v[u];
                            a1[qq] += t1[u] * v[u];
                        }
                    }
                }
            } else {
#pragma unroll 4
                for (int m = 0; m < r; ++m) {
                    const A t0 = Tl[m], t1 = Tr[m];
#pragma unroll
                    for (int qq = 0; qq < QC; ++qq) {
                        const A v = p[qq * r + m];
                        a0[qq] += t0 * v;
                        a1[qq] += t1 * v;
                    }
                }
            }
#pragma unroll
            for (int qq = 0; qq < QC; ++qq) {
                const A v0 = o0[qq * r + lane] + a0[qq], v1 = o1[qq * r + lane] + a1[qq];
                o0[qq * r + lane] = v0;
                o1[qq * r + lane] = v1;
                if (qq < qc) {
                    s[((int64_t)X.c0 * k + q0 + qq) * r + lane] = v0;
                    s[((int64_t)X.c1 * k + q0 + qq) * r + lane] = v1;
                }
            }
        });
        __syncthreads();
    }
}

// Far field: s[slot][m] = sum_e sum_n F_e[m + r n] t[yslot_e][n]
// (the F stage of src/algebra.jl:258-265, grouped by row cluster).  One warp
// per (row slot, chunk of up to QC right-hand sides).  The r x r blocks of the
// row and the column coefficients they multiply are double-buffered in
// shared memory with cp.async: block e + 1 is in flight while block e is
// used for every right-hand side of the chunk.  Lane m accumulates row m.
// smem: m2l_warp_bytes of this warp.  m2l_first copies the first block, which
// does not depend on the upward pass: a kernel calls it before it waits.
template <typename S>
__device__ __forceinline__ void m2l_block(const S *F, int fstride, int64_t foff, S *dst)
{
    const char *src = reinterpret_cast<const char *>(F + foff);
    for (int i = threadIdx.x & 31; i < (int)(fstride * sizeof(S) / 16); i += 32)
        async_copy16(reinterpret_cast<char *>(dst) + 16 * i, src + 16 * i);
}
template <typename S>
__device__ __forceinline__ void m2l_first(const hm_m2l_row R, const hm_m2l_ent *ents, const S *F, int fstride,
                                          unsigned char *smem)
{
    if (R.begin < R.end) m2l_block(F, fstride, ents[R.begin].foff, reinterpret_cast<S *>(smem));
}
template <typename S, typename A, int QC, int RC>
__device__ __forceinline__ void m2l_row(const hm_m2l_row R, int q0, const hm_m2l_ent *ents, const S *F, int fstride,
                                        const A *t, A *s, int rr, int k, unsigned char *smem)
{
    const int r = RC ? RC : rr;
    // two F blocks (fstride values of S) and two column-coefficient chunks (QC * HM_RMAX of A)
    S *Fb = reinterpret_cast<S *>(smem);
    A *Tb = reinterpret_cast<A *>(Fb + 2 * fstride);
    const int lane = threadIdx.x & 31;
    const int qc = min(QC, k - q0);
    auto fetch = [&](int e, int buf) {
        const hm_m2l_ent E = ents[e];
        if (e > R.begin) m2l_block(F, fstride, E.foff, Fb + buf * fstride);      // the first: m2l_first
        A *tb = Tb + buf * QC * HM_RMAX;
        if (lane < r) {
            const A *src = t + ((int64_t)E.yslot * k + q0) * r + lane;
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
    if (R.begin < R.end) fetch(R.begin, 0);
    for (int e = R.begin; e < R.end; ++e) {
        const int buf = (e - R.begin) & 1;
        if (e + 1 < R.end) {
            fetch(e + 1, buf ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            async_wait_all();
        }
        __syncwarp();
        const S *fb = Fb + buf * fstride;
        const A *tb = Tb + buf * QC * HM_RMAX;
        if (lane < r) {
#pragma unroll(RC ? RC : 4)
            for (int n = 0; n < r; ++n) {
                const A f = (A)fb[lane + r * n];
#pragma unroll
                for (int qq = 0; qq < QC; ++qq) acc[qq] += f * tb[qq * HM_RMAX + n];
            }
        }
        __syncwarp();                         // buffer buf is refilled by the next fetch
    }
    if (lane < r) {
#pragma unroll
        for (int qq = 0; qq < QC; ++qq)
            if (qq < qc) s[((int64_t)R.slot * k + q0 + qq) * r + lane] = acc[qq];
    }
}

// Compensated sums of one row segment's columns for KB right-hand sides.
template <typename A, int KB>
struct SegAcc;
template <typename A>
struct SegAcc<A, 1> {
    Acc<A> a;
    __device__ __forceinline__ void zero() { a.zero(); }
    __device__ __forceinline__ void add(A p, const A *g) { a.add(p, g[0]); }
    __device__ __forceinline__ void fold() {}
    __device__ __forceinline__ A hi(int) const { return a.s_hi(); }
    __device__ __forceinline__ A lo(int) const { return a.s_lo(); }
    __device__ __forceinline__ A merged(int, A so, A co) const { return a.merged(so, co); }
    // adds the lane's o away (FP64: plain sums)
    __device__ __forceinline__ void absorb(int o) { a.s = a.s + __shfl_xor_sync(0xffffffffu, a.s, o); }
};
template <typename A, int KB>
struct SegAcc {
    A part[KB], h[KB], l[KB];
    __device__ __forceinline__ void zero()
    {
#pragma unroll
        for (int q = 0; q < KB; ++q) { part[q] = 0; h[q] = 0; l[q] = 0; }
    }
    __device__ __forceinline__ void add(A p, const A *g)
    {
#pragma unroll
        for (int q = 0; q < KB; ++q) part[q] = fma(p, g[q], part[q]);
    }
    __device__ __forceinline__ void fold()   // end of a piece: compensated fold of the partial sums
    {
#pragma unroll
        for (int q = 0; q < KB; ++q) {
            const A t = h[q] + part[q];
            const A bp = t - h[q];
            l[q] += (h[q] - (t - bp)) + (part[q] - bp);
            h[q] = t;
            part[q] = 0;
        }
    }
    __device__ __forceinline__ A hi(int q) const { return h[q]; }
    __device__ __forceinline__ A lo(int q) const { return l[q]; }
    __device__ __forceinline__ A merged(int q, A so, A co) const
    {
        const A t = h[q] + so;
        const A bp = t - h[q];
        return t + (((h[q] - (t - bp)) + (so - bp)) + (l[q] + co));
    }
    __device__ __forceinline__ void absorb(int o)
    {
#pragma unroll
        for (int q = 0; q < KB; ++q) {
            const A so = __shfl_xor_sync(0xffffffffu, h[q], o), co = __shfl_xor_sync(0xffffffffu, l[q], o);
            const A t = h[q] + so, bp = t - h[q];
            l[q] = (l[q] + co) + ((h[q] - (t - bp)) + (so - bp));
            h[q] = t;
        }
    }
};


// Columns of a segment that ring_part takes at once: lane groups of 32 / that many
// lanes, two rows a lane.
__device__ __forceinline__ int ring_groups(int ld) { return ld > 32 ? 1 : ld > 16 ? 2 : ld > 8 ? 4 : 8; }
// The groups' (hi, lo) sums of two rows and KB right-hand sides added into every group
// of `lanes` lanes (TwoSum: the same in each of them).
template <int KB, typename H, typename L>
__device__ __forceinline__ void ring_combine(int lanes, H hi, L lo)
{
    for (int o = lanes; o < 32; o <<= 1) {
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int q = 0; q < KB; ++q) {
                const float h = hi(i, q), so = __shfl_xor_sync(0xffffffffu, h, o);
                const float l = lo(i, q) + __shfl_xor_sync(0xffffffffu, lo(i, q), o);
                const float t = h + so, bp = t - h;
                hi(i, q) = t;
                lo(i, q) = l + ((h - (t - bp)) + (so - bp));
            }
    }
}

// The rows of a segment (<= 64) a lane sums: with one or two FP32 right-hand
// sides lanes 0-15 and 16-31 take alternate columns, each lane four
// consecutive rows (one 16-byte load per column; lanes 0-15 hold the sums);
// otherwise every lane two rows.
template <typename S, int KB>
struct SegRows {
    static constexpr bool quad = sizeof(S) == 4 && KB < 4;
    static constexpr int per_lane = quad ? 4 : 2;
    // row j of this lane, or past every segment where the lane holds no sums
    static __device__ __forceinline__ int row(int j)
    {
        const int lane = threadIdx.x & 31;
        if constexpr (quad) return lane < 16 ? 4 * lane + j : 1 << 20;
        else return 2 * lane + j;
    }
};

// Gathers the right-hand sides of a segment's near-field (FAR = false) or
// far-field columns into shared memory (g[c * KB + q]) and waits for this
// lane's copies.  The part's pieces are one contiguous column run [c0, c1) of
// the panel; false (and an empty run) when there are none.
template <typename S, typename A, bool FAR, int KB>
__device__ __forceinline__ bool seg_gather(const MulArgs<S> &ma, const hm_seg &G, const hm_piece *pieces, const A *s,
                                           const A *t, int r, A *g, int &c0, int &c1)
{
    const int lane = threadIdx.x & 31, k = ma.k;
    int col = 0;
    c0 = -1;
    c1 = 0;
    for (int pc = 0; pc < G.npieces; ++pc) {
        const hm_piece Q = pieces[G.piece0 + pc];
        const bool take = FAR ? (Q.kind != HM_PIECE_X) : (Q.kind == HM_PIECE_X);
        if (take) {
            if (c0 < 0) c0 = col;
            const A *coef = Q.kind == HM_PIECE_TCOEF ? t : s;
            // fire-and-forget copies into shared memory for every piece, one
            // wait after the loop (no load-to-store round trip per piece)
            const int n = Q.width * KB;
            for (int i = lane; i < n; i += 32) {
                const int c = i / KB, q = i % KB;
                A *d = g + (col + c) * KB + q;
                if (q >= k) {
                    *d = A(0);
                } else if constexpr (FAR) {
                    async_copy<sizeof(A)>(d, coef + ((int64_t)Q.src * k + q) * r + c);
                } else if constexpr (sizeof(S) == sizeof(A)) {
                    async_copy<sizeof(A)>(d, ma.x + (Q.src + c) * ma.incx + (int64_t)q * ma.ldx);
                } else {
                    *d = (A)ma.x[(Q.src + c) * ma.incx + (int64_t)q * ma.ldx];
                }
            }
            c1 = col + Q.width;
        }
        col += Q.width;
    }
    async_wait_all();
    if (c0 >= 0) return true;
    c0 = c1 = 0;
    return false;
}

// val[q][j] = sum over columns [c0, c1) of P[row j][c] g[c * KB + q] for this
// lane's rows (SegRows), FMA partial sums folded with TwoSum every 64 columns.
template <typename S, typename A, int KB>
__device__ __forceinline__ void seg_columns(const S *Pg, int ld, const A *g, int c0, int c1,
                                            A (&val)[KB][SegRows<S, KB>::per_lane])
{
    const int lane = threadIdx.x & 31;
    constexpr int FOLD = 64;              // columns between compensated folds (KB > 1)
    if constexpr (sizeof(S) == 4 && KB >= 4) {
        // four or more right-hand sides: each value loaded feeds KB FMAs, so
        // two rows per lane (float2) and every column in turn, which halves
        // the accumulators of the four-row form (3 KB values per row) and lets
        // twice as many warps hide the loads' latency
        SegAcc<A, KB> a0, a1;
        a0.zero(); a1.zero();
        if (2 * lane < ld) {
            const float2 *base = reinterpret_cast<const float2 *>(Pg + 2 * lane);
            const int64_t ld2 = ld / 2;
            for (int cb = c0; cb < c1; cb += FOLD) {
                const int ce = min(c1, cb + FOLD);
                int c = cb;
                for (; c + 16 <= ce; c += 16) {      // 16 loads in flight per lane
                    float2 p[16];
#pragma unroll
                    for (int u = 0; u < 16; ++u) p[u] = __ldcs(base + ld2 * (c + u));
#pragma unroll
                    for (int u = 0; u < 16; ++u) { a0.add(p[u].x, g + (c + u) * KB); a1.add(p[u].y, g + (c + u) * KB); }
                }
                for (; c + 8 <= ce; c += 8) {
                    float2 p[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) p[u] = __ldcs(base + ld2 * (c + u));
#pragma unroll
                    for (int u = 0; u < 8; ++u) { a0.add(p[u].x, g + (c + u) * KB); a1.add(p[u].y, g + (c + u) * KB); }
                }
                for (; c + 4 <= ce; c += 4) {
                    float2 p[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) p[u] = __ldcs(base + ld2 * (c + u));
#pragma unroll
                    for (int u = 0; u < 4; ++u) { a0.add(p[u].x, g + (c + u) * KB); a1.add(p[u].y, g + (c + u) * KB); }
                }
                for (; c < ce; ++c) {
                    const float2 p0 = __ldcs(base + ld2 * c);
                    a0.add(p0.x, g + c * KB); a1.add(p0.y, g + c * KB);
                }
                a0.fold(); a1.fold();
            }
        }
#pragma unroll
        for (int q = 0; q < KB; ++q) { val[q][0] = a0.merged(q, 0, 0); val[q][1] = a1.merged(q, 0, 0); }
    } else if constexpr (sizeof(S) == 4) {
        const int rg = lane & 15, h = lane >> 4;
        SegAcc<A, KB> acc[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[j].zero();
        if (4 * rg < ld) {
            const float4 *base = reinterpret_cast<const float4 *>(Pg + 4 * rg);
            const int64_t ld4 = ld / 4;
            auto add4 = [&](const float4 &p, const A *gu) {
                acc[0].add(p.x, gu); acc[1].add(p.y, gu); acc[2].add(p.z, gu); acc[3].add(p.w, gu);
            };
            for (int cb = c0; cb < c1; cb += FOLD) {
                const int ce = min(c1, cb + FOLD);
                int c = cb + ((h - cb) & 1);             // this half's columns have parity h
                for (; c + 14 < ce; c += 16) {
                    float4 p[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) p[u] = __ldcs(base + ld4 * (c + 2 * u));
#pragma unroll
                    for (int u = 0; u < 8; ++u) add4(p[u], g + (c + 2 * u) * KB);
                }
                for (; c + 6 < ce; c += 8) {           // tails in batches: fewer dependent round trips
                    float4 p[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) p[u] = __ldcs(base + ld4 * (c + 2 * u));
#pragma unroll
                    for (int u = 0; u < 4; ++u) add4(p[u], g + (c + 2 * u) * KB);
                }
                for (; c + 2 < ce; c += 4) {
                    const float4 p0 = __ldcs(base + ld4 * c), p1 = __ldcs(base + ld4 * (c + 2));
                    add4(p0, g + c * KB);
                    add4(p1, g + (c + 2) * KB);
                }
                for (; c < ce; c += 2) add4(__ldcs(base + ld4 * c), g + c * KB);
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[j].fold();
            }
        }
#pragma unroll
        for (int q = 0; q < KB; ++q)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const A so = __shfl_xor_sync(0xffffffffu, acc[j].hi(q), 16);
                const A co = __shfl_xor_sync(0xffffffffu, acc[j].lo(q), 16);
                val[q][j] = acc[j].merged(q, so, co);
            }
    } else {
        SegAcc<A, KB> a0, a1;
        a0.zero(); a1.zero();
        const int64_t ld2 = ld / 2;
        // FP64: a low segment's columns are dealt out to lane groups (an FP64 warp
        // instruction takes 64 cycles however few lanes are live).  Near field of
        // n = 2^20 random points, one right-hand side: 514 -> 393 us,
        // of a 2^16 grid (32-row segments) 61 -> 37
        const int cg = ring_groups(ld);
        if (cg > 1) {
            const int lanes = 32 / cg, lr = lane & (lanes - 1), grp = lane / lanes;
            const double2 *base = reinterpret_cast<const double2 *>(Pg + 2 * lr);
            for (int cb = c0; cb < c1; cb += FOLD) {
                const int ce = min(c1, cb + FOLD);
                if (2 * lr < ld) {
                    for (int c = cb + grp; c < ce; c += 8 * cg) {
                        double2 p[8];
#pragma unroll
                        for (int u = 0; u < 8; ++u)
                            if (c + u * cg < ce) p[u] = __ldcs(base + ld2 * (c + u * cg));
#pragma unroll
                        for (int u = 0; u < 8; ++u)
                            if (c + u * cg < ce) {
                                a0.add(p[u].x, g + (c + u * cg) * KB);
                                a1.add(p[u].y, g + (c + u * cg) * KB);
                            }
                    }
                }
                a0.fold(); a1.fold();
            }
            for (int o = lanes; o < 32; o <<= 1) {
                a0.absorb(o);
                a1.absorb(o);
            }
        } else if (2 * lane < ld) {
            const double2 *base = reinterpret_cast<const double2 *>(Pg + 2 * lane);
            for (int cb = c0; cb < c1; cb += FOLD) {
                const int ce = min(c1, cb + FOLD);
                int c = cb;
                for (; c + 8 <= ce; c += 8) {
                    double2 p[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) p[u] = __ldcs(base + ld2 * (c + u));
#pragma unroll
                    for (int u = 0; u < 8; ++u) { a0.add(p[u].x, g + (c + u) * KB); a1.add(p[u].y, g + (c + u) * KB); }
                }
                for (; c < ce; ++c) {
                    const double2 p0 = __ldcs(base + ld2 * c);
                    a0.add(p0.x, g + c * KB); a1.add(p0.y, g + c * KB);
                }
                a0.fold(); a1.fold();
            }
        }
#pragma unroll
        for (int q = 0; q < KB; ++q) { val[q][0] = a0.merged(q, 0, 0); val[q][1] = a1.merged(q, 0, 0); }
    }
}

}  // namespace
}  // namespace hm
