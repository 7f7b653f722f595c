// Tensor-core (tcgen05) row-segment panels for many right-hand sides, FP32
// storage.  Written for sm_103a.
//
// For one row segment (nrows <= 64 rows, panel P of nrows x width, column-
// major with leading dimension ld) and a chunk of up to 128 right-hand sides,
// an item computes
//     Y[row][q] (+)= sum_c P[row][c] G[q][c],
// where G holds the gathered [s ; x pieces] entries of the chunk.  The MMA is
// D = A B with A = G (M = 128 right-hand sides x K) and B = P^T (K x N = 64
// rows), both stored K-major in shared memory, D (128 x 64, FP32) in tensor
// memory.  FP32 accuracy comes from splitting every FP32 value exactly into
// three BF16 pieces, v = v_h + v_m + v_l (round-to-nearest at each step;
// 3 x 8 significant bits cover FP32's 24), and summing the six products
//     G_h P_h + G_h P_m + G_m P_h + G_m P_m + G_h P_l + G_l P_h
// with FP32 accumulation (the dropped terms are below 2^-24 relative).  The
// panel's pieces are one operand of up to 192 rows, so the six products are three
// MMAs, G_h (P_h, P_m, P_l), G_m (P_h, P_m) and G_l P_h, into three tensor-memory
// blocks added at the end: the tensor core rounds each accumulation relative to
// the running sum, so the corrections (2^-8 of it) must not ride on the large one.
//
// Items (segment, chunk of 128 right-hand sides) run through one persistent CTA
// per SM of four roles, joined by mbarriers only, so that no role waits for
// another one's round trip:
//   table warp     publishes the next items' columns (the address of each column's
//                  first right-hand side) and prefetches their panels into L2 (a
//                  panel is one contiguous run);
//   16 producer    in two groups, each filling every other 64-column chunk: load G
//   warps          and P into registers (lanes along the columns of a right-hand
//                  side, the rows of the panel: whole lines), split them and write
//                  the BF16 pieces into a ring of operand stages;
//   MMA warp       issues a stage's MMAs and frees it by tcgen05.commit;
//   4 epilogue     read the finished accumulators (two sets in tensor memory, so
//   warps          the next item's MMAs run meanwhile), transpose through shared
//                  memory and write y.
// Measured (ms per call of the panel stage): 32 right-hand sides at n = 2^19 0.436
// -> 0.201, 256 at n = 2^18 0.584 -> 0.319.  The form before loaded, split and
// multiplied a chunk between CTA barriers with 24% of the warps active, and its
// load instructions touched eight lines each.  What bounds it now: the producers'
// wait for a chunk's loads, which the registers of 22 warps leave no room to issue a
// chunk ahead (32 right-hand sides: issue slots 43% busy, of which the splitting itself, 11
// instructions per two values, is a quarter, tensor pipe 37%; a second register set
// measured 0.245 ms).
//
// Operand layout (SWIZZLE_128B, K-major, 16-bit): a row's 64 columns are 128 bytes,
// 8-row groups 1,024 bytes apart, the 16-byte columns of row i permuted by XOR
// with i mod 8.  Rows past the live right-hand sides read whatever follows; their
// results are never read.
#include "hm_kernels.cuh"
#include "hm_async.cuh"

#include <cuda_bf16.h>

namespace hm {

namespace {

constexpr int TC_M = 128;          // right-hand sides per CTA (MMA M)
constexpr int TC_N = 64;           // rows per segment (MMA N)
constexpr int TC_KC = 64;          // columns per K chunk (a 128-byte row of BF16)
constexpr int TC_PRODUCERS = 16;   // producer warps (warps 6 .. 21; 0 .. 3 epilogue, 4 MMA, 5 tables)
constexpr int TC_FIRST = 6;
constexpr int TC_GROUP = 8;                            // warps that fill a chunk
constexpr int TC_GROUPS = TC_PRODUCERS / TC_GROUP;
constexpr int TC_P_PIECE = TC_N * 128;                 // one BF16 piece of a chunk's panel
constexpr int TC_P_BYTES = 3 * TC_P_PIECE;
constexpr int TC_SET = 3 * TC_N;                       // tensor-memory columns of one accumulator set
constexpr int TC_TMEM = 512;                           // two sets, allocated as a power of two
constexpr int TC_YS = 65;                              // row stride of the epilogue's transpose
constexpr int TC_MAX_STAGES = 6, TC_MAX_TABLES = 4;
static_assert(TC_THREADS == (TC_FIRST + TC_PRODUCERS) * 32, "roles");

struct TcItem {                    // what the producers need of an item
    int64_t poff;
    int width, ld;
};
struct TcShared {
    uint64_t full[TC_MAX_STAGES], empty[TC_MAX_STAGES];    // operand stages: written / read by the MMAs
    uint64_t tab_full[TC_MAX_TABLES], tab_empty[TC_MAX_TABLES];   // column tables
    uint64_t acc_full[2], acc_empty[2];                    // accumulator sets
    uint64_t never;                                        // nothing arrives on it (stall hook)
    TcItem item[TC_MAX_TABLES];
    uint32_t tmem_base;
    int abort;                                             // a role gave up: the others leave too
};

// A stage: the pieces of G (8-row groups of 1,024 bytes), then those of P.
__host__ __device__ constexpr int tc_stage_bytes(int groups) { return 3 * groups * 1024 + TC_P_BYTES; }
__host__ __device__ constexpr size_t tc_fixed_bytes()
{
    return (sizeof(TcShared) + 127) / 128 * 128 + sizeof(float) * 128 * TC_YS;
}

// (a, b) = h + m + l exactly, each a BF16 pair (round to nearest at every
// step); the pairs are packed as stored: a in the low half.
__device__ __forceinline__ void split3x2(float a, float b, uint32_t &h, uint32_t &m, uint32_t &l)
{
    const __nv_bfloat162 h2 = __floats2bfloat162_rn(a, b);
    const float2 hf = __bfloat1622float2(h2);
    const float ra = a - hf.x, rb = b - hf.y;
    const __nv_bfloat162 m2 = __floats2bfloat162_rn(ra, rb);
    const float2 mf = __bfloat1622float2(m2);
    const __nv_bfloat162 l2 = __floats2bfloat162_rn(ra - mf.x, rb - mf.y);
    h = *reinterpret_cast<const uint32_t *>(&h2);
    m = *reinterpret_cast<const uint32_t *>(&m2);
    l = *reinterpret_cast<const uint32_t *>(&l2);
}

// Shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups 1,024
// bytes apart, descriptor version 1.
__device__ __forceinline__ uint64_t umma_desc(const void *p)
{
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr(p) & 0x3FFFF) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// Instruction descriptor (kind::f16): D FP32, A and B BF16, both K-major, M x N.
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int m, int n)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// Called by a whole converged warp; one lane (elect.sync, the same one each time)
// issues.  Descriptors then stay in uniform registers: issued from a one-thread
// branch each MMA paid six moves into them, about 130 cycles.
__device__ __forceinline__ void umma_bf16(uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, int acc)
{
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "elect.sync _|e, 0xffffffff;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(dtmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
        : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t *bar)
{
    asm volatile(
        "{\n\t.reg .pred e;\n\t"
        "elect.sync _|e, 0xffffffff;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_addr(bar))
        : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 16 consecutive FP32 columns of this warp's 32 TMEM lanes of an accumulator
// set's three blocks, summed.
__device__ __forceinline__ void tmem_sum16(uint32_t a, float *v)
{
    uint32_t r[48];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%48];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%49];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%32, %33, %34, %35, %36, %37, %38, %39, %40, %41, %42, %43, %44, %45, %46, %47}, [%50];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]),
          "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]), "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47])
        : "r"(a), "r"(a + TC_N), "r"(a + 2 * TC_N)
        : "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i)
        v[i] = __uint_as_float(r[i]) + (__uint_as_float(r[16 + i]) + __uint_as_float(r[32 + i]));
}

// Waits for a phase of `bar` (a whole warp; the answer is the same in every
// lane); false when another role gave up, or once limit_ns has passed (then
// *abort is set).  SLEEP: between tests the warp sleeps about that many
// nanoseconds, so that the roles that mostly wait leave the issue slots to the
// producers.  The global timer, slow to read, is left alone for the first 32 tests.
template <int SLEEP>
__device__ __forceinline__ bool tc_wait(uint64_t *bar, uint32_t parity, unsigned long long limit_ns, int *abort)
{
    bool got = mbar_test(bar, parity);
    if (!got) {
        uint64_t t0 = 0;
        for (;;) {
#pragma unroll 1
            for (int i = 0; i < 32 && !got; ++i) {
                if (SLEEP) __nanosleep(SLEEP);
                got = mbar_test(bar, parity);
            }
            if (got || *reinterpret_cast<volatile int *>(abort)) break;
            const uint64_t now = global_ns();
            if (!t0) t0 = now;
            else if (now - t0 > limit_ns) {
                atomicExch(abort, 1);
                break;
            }
        }
    }
    return __all_sync(0xffffffffu, got);
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

// Two words (four consecutive columns) of each BF16 piece to dst, dst + piece, dst + 2 piece.
__device__ __forceinline__ void split_store(const float (&v)[4], unsigned char *dst, int piece)
{
    uint2 h, m, l;
    split3x2(v[0], v[1], h.x, m.x, l.x);
    split3x2(v[2], v[3], h.y, m.y, l.y);
    *reinterpret_cast<uint2 *>(dst) = h;
    *reinterpret_cast<uint2 *>(dst + piece) = m;
    *reinterpret_cast<uint2 *>(dst + 2 * piece) = l;
}

}  // namespace

// Stages, table buffers and shared memory for k right-hand sides and panels of
// at most maxw columns; stages == 0 when it does not fit.
TcPlan expand_tc_plan(int k, int maxw)
{
    constexpr size_t kMax = 227 * 1024;
    TcPlan p;
    p.groups = ((k < TC_M ? k : TC_M) + 7) / 8;
    const size_t table = ((size_t)maxw * sizeof(const float *) + 127) / 128 * 128, stage = tc_stage_bytes(p.groups);
    for (int least = 2; least >= 1; --least) {             // one stage only for panels of thousands of columns
        for (p.tables = TC_MAX_TABLES; p.tables >= 1; --p.tables) {
            const size_t used = tc_fixed_bytes() + p.tables * table + 1024;    // the ring starts on a 1,024-byte boundary
            const size_t fit = used < kMax ? (kMax - used) / stage : 0;
            p.stages = (int)(fit < TC_MAX_STAGES ? fit : TC_MAX_STAGES);
            p.smem = used + p.stages * stage;
            if (p.stages >= least) return p;
        }
    }
    p.stages = 0;
    return p;
}

template <bool VEC, int NJ>
__global__ void __launch_bounds__(TC_THREADS, 1)
    expand_tc(MulArgs<float> ma, const hm_seg *segs, int nsegs, const hm_piece *pieces, const float *P, const float *s,
              const float *t, int r, int maxw, TcPlan plan, int *status, unsigned long long wait_ns, int stall)
{
    extern __shared__ __align__(128) unsigned char tc_smem_raw[];
    TcShared &S = *reinterpret_cast<TcShared *>(tc_smem_raw);
    float *Ys = reinterpret_cast<float *>(tc_smem_raw + (sizeof(TcShared) + 127) / 128 * 128);
    unsigned char *tables = tc_smem_raw + tc_fixed_bytes();
    const int table_bytes = (int)(((size_t)maxw * sizeof(const float *) + 127) / 128 * 128);
    unsigned char *ring = tables + (size_t)plan.tables * table_bytes;
    ring += (1024u - (smem_addr(ring) & 1023u)) & 1023u;
    // A parity tells a barrier's neighbouring phases apart only: two groups need two
    // stages (a group's previous chunk was then let in after the fill two before
    // its next one was read); on a single stage one group works.
    const int ngroups = plan.stages > 1 ? TC_GROUPS : 1;
    const int gpiece = plan.groups * 1024, stage_bytes = tc_stage_bytes(plan.groups);
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    // items in order: segment, then chunk of right-hand sides; a CTA takes every
    // gridDim.x-th.  (The step as quotient and remainder: a 64-bit division per item and
    // role cost each of them some 500 cycles.)
    const int nqc = (ma.k + TC_M - 1) / TC_M;
    const int dseg = (int)gridDim.x / nqc, dqi = (int)gridDim.x % nqc;
    struct Cursor {
        int seg, qi;
    };
    auto advance = [&](Cursor &c) {
        c.seg += dseg;
        c.qi += dqi;
        if (c.qi >= nqc) { c.qi -= nqc; ++c.seg; }
    };
    Cursor at_item{(int)blockIdx.x / nqc, (int)blockIdx.x % nqc};

    if (warp == 4) {               // tensor memory: two sets of (h h products, corrections) x 64 FP32 columns
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&S.tmem_base)),
                     "r"(TC_TMEM)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int i = 0; i < plan.stages; ++i) {
            mbar_init(&S.full[i], TC_GROUP);
            mbar_init(&S.empty[i], 1);
        }
        for (int i = 0; i < plan.tables; ++i) {
            mbar_init(&S.tab_full[i], 1);
            mbar_init(&S.tab_empty[i], ngroups * TC_GROUP);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&S.acc_full[i], 1);
            mbar_init(&S.acc_empty[i], 4);
        }
        mbar_init(&S.never, 1);
        S.abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = S.tmem_base;
    uint64_t *pending = nullptr;   // MMA thread: the barrier of the last commit
    uint32_t pending_parity = 0;

    if (warp >= TC_FIRST) {
        // ---- producers.  Group `grp` of eight warps fills every other chunk by itself:
        // a warp's way through a chunk (table, loads, wait, split, fence, arrival) is
        // a chain of about 1,000 cycles whatever its share, so all warps on every
        // (32-column) chunk took 2,000 cycles a chunk.  Lane (qs, c16) of warp gw takes
        // right-hand sides 2 gw + qs + 16 j, columns 4 c16 .. + 3 of the chunk; of the
        // panel rows 16 (gw / 2) + lane / 2, columns 8 (gw % 2 + 2 i) + 4 (lane % 2) .. + 3.
        const int grp = (warp - TC_FIRST) / TC_GROUP, gw = (warp - TC_FIRST) % TC_GROUP, qs = lane >> 4, c16 = lane & 15;
        const int prow = 16 * (gw >> 1) + (lane >> 1), pcol = 8 * (gw & 1) + 4 * (lane & 1);
        const int q0l = 2 * gw + qs;
        // byte of (row, column 4 c): 16-byte columns swizzled by the row within its group of 8
        auto at = [](int row, int c) { return (row >> 3) * 1024 + (row & 7) * 128 + (((c >> 1) ^ (row & 7)) << 4) + (c & 1) * 8; };
        const int gdst = at(q0l, c16);                         // rows 16 apart: 2,048 bytes apart
        const int pdst = at(prow, pcol >> 2);                  // columns 16 i on: pdst ^ (32 i)
        int slot = 0, ch = grp, nch = 0, qc = 0, stage = grp;
        uint32_t tab_phase = 0, phase = 0;
        TcItem it{};
        const float *const *cols = nullptr;
        bool have = false, ok = grp < ngroups;               // have: the item's table is open
        for (; stage >= plan.stages; stage -= plan.stages) phase ^= 1;
        while (ok) {
            // this group's next chunk, through the tables of the items it has no chunk of
            while (ch >= nch) {
                if (have) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&S.tab_empty[slot]);
                    ch -= nch;
                    advance(at_item);
                    if (++slot == plan.tables) { slot = 0; tab_phase ^= 1; }
                }
                if (at_item.seg >= nsegs || !tc_wait<20>(&S.tab_full[slot], tab_phase, wait_ns, &S.abort)) { ok = false; break; }
                have = true;
                it = S.item[slot];
                cols = reinterpret_cast<const float *const *>(tables + (size_t)slot * table_bytes);
                nch = (it.width + TC_KC - 1) / TC_KC;
                qc = min(TC_M, ma.k - at_item.qi * TC_M);
            }
            if (!ok) break;
            const int left = it.width - ch * TC_KC;            // columns of the item from this chunk on
            float p[4][4], g[NJ][4];
            const float *pp = P + it.poff + (int64_t)(ch * TC_KC + pcol) * it.ld + prow;
            if (left >= TC_KC && it.ld == TC_N) {              // a whole chunk of a whole segment
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int u = 0; u < 4; ++u) p[i][u] = __ldcs(pp + (16 * i + u) * TC_N);
            } else {
                const int pleft = prow < it.ld ? left - pcol : 0;
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int u = 0; u < 4; ++u) p[i][u] = 16 * i + u < pleft ? __ldcs(pp + (16 * i + u) * it.ld) : 0.f;
            }
            const int gc = 4 * c16;
            if constexpr (VEC) {
                // four columns of one piece, 16-byte aligned: one load per right-hand side
                const uintptr_t e = gc < left ? reinterpret_cast<uintptr_t>(cols[ch * TC_KC + gc]) : 0;
                const int64_t st = (e & 1 ? (int64_t)r : ma.ldx) * (int64_t)sizeof(float);     // bit 0: coefficients
                const char *b = reinterpret_cast<const char *>(e & ~(uintptr_t)3) + q0l * st;
                const int64_t st16 = 16 * st;
#pragma unroll
                for (int j = 0; j < NJ; ++j, b += st16) {
                    if (2 * gw + 16 * j >= qc) break;          // no live right-hand side in this warp's rows
                    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (e && q0l + 16 * j < qc) v = *reinterpret_cast<const float4 *>(b);
                    g[j][0] = v.x; g[j][1] = v.y; g[j][2] = v.z; g[j][3] = v.w;
                }
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uintptr_t e = gc + i < left ? reinterpret_cast<uintptr_t>(cols[ch * TC_KC + gc + i]) : 0;
                    const int64_t st = (e & 1 ? (int64_t)r : ma.ldx) * (int64_t)sizeof(float);
                    const char *b = reinterpret_cast<const char *>(e & ~(uintptr_t)3) + q0l * st;
                    const int64_t st16 = 16 * st;
#pragma unroll
                    for (int j = 0; j < NJ; ++j, b += st16) {
                        if (2 * gw + 16 * j >= qc) break;
                        g[j][i] = e && q0l + 16 * j < qc ? *reinterpret_cast<const float *>(b) : 0.f;
                    }
                }
            }
            if (!tc_wait<20>(&S.empty[stage], phase ^ 1, wait_ns, &S.abort)) break;
            unsigned char *sg = ring + (size_t)stage * stage_bytes, *sp = sg + 3 * gpiece;
            // columns up to the last step of 16 the MMAs take
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (16 * i < left) split_store(p[i], sp + (pdst ^ (i << 5)), TC_P_PIECE);
            if (4 * c16 < ((left + 15) & ~15)) {
#pragma unroll
                for (int j = 0; j < NJ; ++j)
                    if (2 * gw + 16 * j < qc) split_store(g[j], sg + gdst + j * 2048, gpiece);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");               // visible to the tensor core
            __syncwarp();
            if (lane == 0) mbar_arrive(&S.full[stage]);
            ch += ngroups;
            for (stage += ngroups; stage >= plan.stages; stage -= plan.stages) phase ^= 1;
        }
    } else if (warp == 5) {
        // ---- column tables: the address of each column's right-hand side q0 (bit 0 set
        // for coefficients).  Lane i holds piece i of the item; the next item's segment and
        // pieces are loaded while this one's table is written (a load in line per
        // piece, about 0.6 us each, made this warp the bottleneck: 6.8 us an item).
        int slot = 0;
        uint32_t phase = 0;
        auto seg_at = [&](const Cursor &c) { return c.seg < nsegs ? segs[c.seg] : hm_seg{}; };
        auto piece_of = [&](const hm_seg &G, int i) { return i < G.npieces ? pieces[G.piece0 + i] : hm_piece{0, HM_PIECE_X, 0}; };
        Cursor ahead = at_item;
        advance(ahead);
        hm_seg G = seg_at(at_item), Gn = seg_at(ahead);
        hm_piece Q = piece_of(G, lane);
        for (; at_item.seg < nsegs; advance(at_item)) {
            advance(ahead);
            const hm_seg G2 = seg_at(ahead);
            const hm_piece Qn = piece_of(Gn, lane);
            if (!tc_wait<50>(&S.tab_empty[slot], phase ^ 1, wait_ns, &S.abort)) break;
            const int q0 = at_item.qi * TC_M;
            const float **cols = reinterpret_cast<const float **>(tables + (size_t)slot * table_bytes);
            if (lane == 0) {
                S.item[slot] = TcItem{G.poff, G.width, G.ld};
                const uint32_t bytes = (uint32_t)G.ld * (uint32_t)G.width * 4u;
                if (bytes)
                    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(P + G.poff), "r"(bytes) : "memory");
            }
            int col = 0;
            for (int p0 = 0; p0 < G.npieces; p0 += 32) {
                if (p0) Q = piece_of(G, p0 + lane);
                const bool x = Q.kind == HM_PIECE_X;
                const float *base = x ? ma.x + Q.src * ma.incx + (int64_t)q0 * ma.ldx
                                      : (Q.kind == HM_PIECE_TCOEF ? t : s) + ((int64_t)Q.src * ma.k + q0) * r;
                const uintptr_t e = reinterpret_cast<uintptr_t>(base) | (x ? 0u : 1u);
                const int64_t inc = x ? ma.incx * (int64_t)sizeof(float) : (int64_t)sizeof(float);
                for (int i = 0; i < min(32, G.npieces - p0); ++i) {
                    const int w = __shfl_sync(0xffffffffu, Q.width, i);
                    const uintptr_t ei = __shfl_sync(0xffffffffu, (unsigned long long)e, i);
                    const int64_t inci = __shfl_sync(0xffffffffu, (long long)inc, i);
                    for (int c = lane; c < w; c += 32) cols[col + c] = reinterpret_cast<const float *>(ei + c * inci);
                    col += w;
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&S.tab_full[slot]);
            if (++slot == plan.tables) { slot = 0; phase ^= 1; }
            G = Gn;
            Gn = G2;
            Q = Qn;
        }
    } else if (warp == 4) {
        // ---- MMAs (the warp stays converged: umma_bf16)
        const uint32_t idesc1 = umma_idesc_bf16(TC_M, TC_N), idesc2 = umma_idesc_bf16(TC_M, 2 * TC_N),
                       idesc3 = umma_idesc_bf16(TC_M, 3 * TC_N);
        int stage = 0, set = 0;
        uint32_t phase = 0, set_phase = 0;
        bool ok = true, first = stall != 0;
        int width = __shfl_sync(0xffffffffu, at_item.seg < nsegs ? segs[at_item.seg].width : 0, 0);
        const uint64_t ring_desc = umma_desc(ring);
        const uint32_t dstage = (uint32_t)stage_bytes >> 4, dpiece = (uint32_t)gpiece >> 4;
        while (at_item.seg < nsegs && ok) {
            const int w = width, nch = (w + TC_KC - 1) / TC_KC;
            advance(at_item);
            if (at_item.seg < nsegs) width = __shfl_sync(0xffffffffu, segs[at_item.seg].width, 0);
            if (nch == 0) continue;
            if (!tc_wait<20>(&S.acc_empty[set], set_phase ^ 1, wait_ns, &S.abort)) break;
            const uint32_t acc = tmem + (uint32_t)set * TC_SET;
            for (int ch = 0; ch < nch; ++ch) {
                uint64_t *bar = first ? &S.never : &S.full[stage];
                if (!tc_wait<0>(bar, first ? 0 : phase, wait_ns, &S.abort)) { ok = false; break; }
                first = false;
                tc_fence_after();
                // the panel's pieces h, m, l are one operand of 64 to 192 rows; descriptors by
                // additions to the start address (built anew they cost the thread
                // about 100 cycles per MMA)
                const uint64_t gh = ring_desc + stage * dstage, ph = gh + 3 * dpiece;
                const int nks = min(TC_KC, w - ch * TC_KC + 15) >> 4;
#pragma unroll
                for (int ks = 0; ks < TC_KC / 16; ++ks) {
                    if (ks >= nks) break;
                    umma_bf16(acc, gh + 2 * ks, ph + 2 * ks, idesc3, ch > 0 || ks > 0 ? 1 : 0);        // h (h, m, l)
                    umma_bf16(acc + TC_N, gh + dpiece + 2 * ks, ph + 2 * ks, idesc2, 1);               // m (h, m)
                    umma_bf16(acc + TC_N, gh + 2 * dpiece + 2 * ks, ph + 2 * ks, idesc1, 1);           // l h
                }
                umma_commit(&S.empty[stage]);
                pending = &S.empty[stage];
                pending_parity = phase;
                if (++stage == plan.stages) { stage = 0; phase ^= 1; }
            }
            if (!ok) break;
            umma_commit(&S.acc_full[set]);
            pending = &S.acc_full[set];
            pending_parity = set_phase;
            if ((set ^= 1) == 0) set_phase ^= 1;
        }
        // all MMAs done before this CTA's shared and tensor memory go
        if (pending) mbar_wait(pending, pending_parity, kDrainLimitNs);
    } else {
        // ---- epilogue: warp w holds right-hand sides 32 w .. + 31 of an item, lane l one of them
        float *yw = Ys + warp * 32 * TC_YS;
        int set = 0;
        uint32_t set_phase = 0;
        hm_seg Gn = at_item.seg < nsegs ? segs[at_item.seg] : hm_seg{};
        while (at_item.seg < nsegs) {
            const hm_seg G = Gn;
            const int q0 = at_item.qi * TC_M, nq = min(32, ma.k - q0 - 32 * warp);
            advance(at_item);
            if (at_item.seg < nsegs) Gn = segs[at_item.seg];
            if (G.width > 0) {
                if (!tc_wait<100>(&S.acc_full[set], set_phase, wait_ns, &S.abort)) break;
                tc_fence_after();
                if (nq > 0) {
                    const uint32_t acc = tmem + (uint32_t)set * TC_SET + ((uint32_t)(warp * 32) << 16);
#pragma unroll
                    for (int c0 = 0; c0 < TC_N; c0 += 16) {
                        float v[16];
                        tmem_sum16(acc + c0, v);
#pragma unroll
                        for (int i = 0; i < 16; ++i) yw[lane * TC_YS + c0 + i] = v[i];
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&S.acc_empty[set]);
                if ((set ^= 1) == 0) set_phase ^= 1;
            }
            // rows lane and lane + 32 of eight right-hand sides at a time
            float *yp = ma.y + (G.row0 + lane) * ma.incy + (int64_t)(q0 + 32 * warp) * ma.ldy;
            const bool r0 = lane < G.nrows, r1 = lane + 32 < G.nrows, zero = G.width == 0;   // no columns: zero rows
            for (int qb = 0; qb < nq; qb += 8) {
                float v0[8], v1[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    v0[i] = zero ? 0.f : yw[(qb + i) * TC_YS + lane];
                    v1[i] = zero ? 0.f : yw[(qb + i) * TC_YS + lane + 32];
                }
                if (ma.accumulate) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        if (qb + i >= nq) break;
                        const float *o = yp + (qb + i) * ma.ldy;
                        if (r0) v0[i] += o[0];
                        if (r1) v1[i] += o[32 * ma.incy];
                    }
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    if (qb + i >= nq) break;
                    float *o = yp + (qb + i) * ma.ldy;
                    if (r0) o[0] = v0[i];
                    if (r1) o[32 * ma.incy] = v1[i];
                }
            }
            __syncwarp();                                      // yw is free again
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (tid == 0 && S.abort) atomicExch(status, HM_DEV_WAIT_TIMEOUT);
    if (warp == 4)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TC_TMEM) : "memory");
}

#define HM_INST_TC(VEC, NJ)                                                                                      \
    template __global__ void expand_tc<VEC, NJ>(MulArgs<float>, const hm_seg *, int, const hm_piece *,         \
                                                const float *, const float *, const float *, int, int, TcPlan, \
                                                int *, unsigned long long, int);
HM_INST_TC(true, 2) HM_INST_TC(false, 2) HM_INST_TC(true, 4) HM_INST_TC(false, 4) HM_INST_TC(true, 8) HM_INST_TC(false, 8)

}  // namespace hm
