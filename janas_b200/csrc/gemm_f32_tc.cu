// out[n, m] = A[n, k] . W[m, k]^T in float32 on the fifth-generation tensor cores.
//
// A float times 2^24 is the exact sum of three bfloat16 (24 bits of mantissa in three times eight, each rest rounded to
// nearest: hi, mid, lo; the factor keeps the last part of the smallest float above the smallest normal bfloat16, which
// has the exponents of a float), so the product of two floats is nine products of bfloat16, each exact in float32.  The
// six largest are added up; the three left out are below 2^-26 of the product.  They are tcgen05 MMAs, 128 features by
// tokens by 16 of k, with float32 accumulators in tensor memory.  A segment's sum is taken times 2^-48 at its end.
//
// Every output value is computed by one fixed recipe, whatever n is, so that a row's result is the same bits
// however the tokens are cut into steps: k is cut into blocks of 64 at fixed places; a block's accumulator takes the
// small products first (weight's part, token's part: hi lo, mid mid, lo hi, then hi mid, mid hi, then hi hi; all of the
// block's k for one pair, then the next), so that only the last four MMAs round at the size of the sum; the blocks' sums
// of a segment are added in ascending order by ordinary additions, and so are the segments' sums.  (The
// tensor core cuts off what does not fit instead of rounding; over all of a segment that bias would show.)
//
// The weights are floats in memory.  TMA brings boxes of 128 features x 32 of k into a ring; four warps take them
// apart, a thread a feature, and put the three parts into tensor memory, from where the MMAs read them: shared
// memory is read and written once per weight and holds no second copy.  The tokens' parts are the MMAs' other
// operand, in shared memory.  For few tokens some warps of the CTA make them from the floats; for many a kernel
// ahead of this one does it once, instead of every tile of features again, and TMA brings them.
//
// What bounds it: few tokens, the stores of the next block's parts into tensor memory beside a block's MMAs (24 MMAs of 16
// tokens take 590 cycles alone, about 1,000 beside the stores; a block some 1,600 with all of it, its 32 KB of weights
// 1,400 at the memory's full rate); many, the MMAs: 1,920 cycles a block of 160 tokens, of 2,150 that it takes.  One
// B200, microseconds, weights from memory, all kernels of a call; in brackets gemm_simt.cu, which took these products
// before:
//   tokens          6144 x 2560   2560 x 4096   19456 x 2560   2560 x 9728   151936 x 2560
//       8           17.5 (21.2)   14.8 (15.1)   47.6 (52.6)    24.2 (29.5)   306 to 324 (272)
//      64           22.6 (67.4)   19.1 (45.9)   59.6 (208)     31.0 (118)    380 (1,150)
//     300           56.2 (271)    44.7 (171)    170 (724)      82.3 (414)    1,270 (5,290)
// The error against 64 bits is 1.0e-7 to 1.3e-7 of the result (2.9e-7 to 3.0e-7), also where all of a token or of a
// feature is small.
//
// A sum that is not finite is taken again from the floats by plain multiply-adds: an infinity has no parts, and neither
// has a float from 2^104 up; a finite sum of finite products gets there from 2^80 up, or where it overflows on the way.
//
// The reference computes y = W x with rows of W as output features (src/llm/model_load.c:452); its products are
// over quantized blocks and are not reproduced.
#include "kernels.h"
#include "tc_common.cuh"

namespace jb {

constexpr int F_BK = 64;                       // k of a block
constexpr int F_M = 128;                       // features of a tile
constexpr int BOX_K = 32;                      // k of a box of weights: 128 bytes of float, one swizzle row
constexpr int BOX_BYTES = F_M * BOX_K * 4;
static_assert(BOX_K * 4 == 128 && F_BK * 2 == 128, "boxes of tensor_map_2d");
constexpr int A_COLS = 3 * F_BK / 2;           // tensor-memory columns of a block's weights: three parts, two values a column

__device__ int g_gemm_f32_tc_error;            // 0, or the code of the first wait that ran out

// FEW: the few tokens of a decode step, whose parts the CTA makes itself.
template <int BN> struct F32Cfg {
    static constexpr bool FEW = BN <= 32;
    static constexpr int PART_BYTES = BN * F_BK * 2;            // one part of a block's tokens
    static constexpr int BUFS = BN <= 64 ? 3 : 2;               // blocks of weights' parts in tensor memory
    static constexpr int B_SLOTS = FEW ? 3 : BN == 160 ? 7 : 9; // tokens' parts in shared memory: FEW by blocks, else by parts
    static constexpr int SLOT_BYTES = FEW ? 3 * PART_BYTES : PART_BYTES;
    static constexpr int BOXES = BN == 160 ? 5 : BN == 128 ? 4 : BN == 96 ? 6 : BN == 64 ? 9 : 10;
    static constexpr int CONV_WARPS = BN <= 96 ? 8 : 4, EPI_WARPS = FEW ? 4 : 8;
    static constexpr int TOK_WARPS = FEW ? BN / 4 : 0;          // FEW: make the tokens' parts
    static constexpr int THREADS = 32 * (4 + CONV_WARPS + EPI_WARPS + TOK_WARPS);
    static constexpr int COLS = BN * 4 / EPI_WARPS;             // token columns of an epilogue thread
    static constexpr int BARS = 2 * (BOXES + BUFS + B_SLOTS + 1);
    static constexpr int SMEM_BYTES = BOXES * BOX_BYTES + B_SLOTS * SLOT_BYTES + 1024 /* alignment */ + 8 * BARS + 16;
    static_assert(BUFS * A_COLS + 2 * BN <= 512, "the blocks of weights and two accumulators");
    static_assert(SMEM_BYTES <= 227 * 1024, "shared memory of a CTA");
};

// What a CTA works on: a tile over all of k (its sums go to out), or a segment of a tile (its sums go to part[(tile - whole) segments + segment][BN][128]).
struct F32Work {
    int n, m, k;
    int n_tiles, segments, seg_blocks, blocks;      // token tiles, segments of k, blocks of one, blocks of k
    int whole;                          // tiles taken over all of k
    int units;                          // those tiles, and the others' segments
};

struct Ring {
    uint32_t at = 0, parity = 0;
    __device__ void next(uint32_t places)
    {
        if (++at == places) {
            at = 0;
            parity ^= 1;
        }
    }
};

// The CTA's blocks in the order in which every role takes them.
struct F32Cursor {
    const F32Work &w;
    int u, tile, seg, segs_end, kb, kb_end;
    __device__ explicit F32Cursor(const F32Work &work) : w(work), u(blockIdx.x)
    {
        if (valid())
            open();
    }
    __device__ bool valid() const { return u < w.units; }
    __device__ bool whole() const { return u < w.whole; }
    __device__ bool last() const { return kb + 1 == kb_end; }          // of its segment
    // blocks that the CTA still has, this one included
    __device__ int left() const
    {
        int n = 0;
        for (F32Cursor c = *this; c.valid();) {
            n += min(w.blocks, c.segs_end * w.seg_blocks) - c.kb;
            c.u += gridDim.x;
            if (c.valid())
                c.open();
        }
        return n;
    }
    __device__ int m0() const { return tile / w.n_tiles * F_M; }
    __device__ int n0(int bn) const { return tile % w.n_tiles * bn; }
    __device__ void open()
    {
        if (u < w.whole) {
            tile = u;
            seg = 0;
            segs_end = w.segments;
        } else {
            int v = u - w.whole;
            tile = w.whole + v / w.segments;
            seg = v % w.segments;
            segs_end = seg + 1;
        }
        kb = seg * w.seg_blocks;
        kb_end = min(w.blocks, kb + w.seg_blocks);
    }
    __device__ void next()
    {
        if (++kb < kb_end)
            return;
        if (++seg < segs_end) {
            kb_end = min(w.blocks, kb + w.seg_blocks);
        } else {
            u += gridDim.x;
            if (valid())
                open();
        }
    }
};

// d += a . b over a block's k (64: four MMAs; first: d starts from zero), a in tensor memory (lane: row, a column: two
// values of k), b in shared memory.  By a whole warp (see tc_mma4).
__device__ __forceinline__ void tc_mma_ts_block(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                                uint32_t accumulate)
{
    asm volatile(
        "{\n\t"
        ".reg .pred p, q;\n\t"
        ".reg .b32 a1, a2, a3;\n\t"
        ".reg .b64 b1, b2, b3;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "add.u32 a1, %1, 8;\n\t"
        "add.u32 a2, %1, 16;\n\t"
        "add.u32 a3, %1, 24;\n\t"
        "add.u64 b1, %2, 2;\n\t"
        "add.u64 b2, %2, 4;\n\t"
        "add.u64 b3, %2, 6;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], b1, %3, 1;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], b2, %3, 1;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], b3, %3, 1;\n\t"
        "}\n"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void tc_st8(uint32_t taddr, const uint32_t *r)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};"
                 ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(taddr)
                 : "memory");
}

__device__ __forceinline__ void tc_ld16_nowait(uint32_t taddr, uint32_t *r)
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}

// Both operands' factor, and what takes both out of a sum again.
constexpr float F_UP = 16777216.0f, F_DOWN = 1.0f / F_UP / F_UP;

// The parts of two floats times F_UP, the first in the lower halves.
__device__ __forceinline__ uint32_t bf16_pair(float lo, float hi)
{
    uint32_t d;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
}
__device__ __forceinline__ void parts_of(float x, float y, uint32_t &p0, uint32_t &p1, uint32_t &p2)
{
    const f32x2 minus = pair2(-1.0f, -1.0f);
    f32x2 v = mul2(pair2(x, y), pair2(F_UP, F_UP));
    auto rest = [&](uint32_t p) { return fma2(pair2(__uint_as_float(p << 16), __uint_as_float(p & 0xffff0000u)), minus, v); };
    split2(v, x, y);
    p0 = bf16_pair(x, y);
    v = rest(p0);
    split2(v, x, y);
    p1 = bf16_pair(x, y);
    v = rest(p1);
    split2(v, x, y);
    p2 = bf16_pair(x, y);
}

// A segment (k0 <= k < k1, multiples of four) of four tokens for a lane's feature, where sums were not finite: by
// multiply-adds, even and odd k in a chain each.  a: the first token, rows of k floats, `last` the last that there is; bad:
// the sums to make, a bit a token; to, step: where they go, added to what is there or not.  A token's NaN makes all of its
// sums one, and a run that went wrong has little else: looked for first, without the weights, of which every lane reads a
// row of its own.  One B200, us, 320 rows of 12288 x 2048 (one segment; finite 120, gemm_simt.cu 393): all NaN 3,020, all
// infinite 8,700; 300 of 2560 x 9728 (98, 433) 1,190 and 3,170; 8 of those (46, 47) 94 and 270.  A token and a feature
// at a time, as it was: 46,100, 17,500 and 1,040.
__device__ __noinline__ void plain_sums(const float *a, int k, int last, int a_vec, const float *w, int k0, int k1,
                                        uint32_t bad, float *to, size_t step, bool add)
{
    const float *row[4];
#pragma unroll
    for (int t = 0; t < 4; t++)
        row[t] = a + (size_t)min(t, last) * k;
    bool nan[4] = {};
    if (a_vec) {
#pragma unroll 2
        for (int i = k0; i < k1; i += 4)
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const float4 v = load4(row[t] + i);
                nan[t] |= isnan(v.x) | isnan(v.y) | isnan(v.z) | isnan(v.w);
            }
    } else {
#pragma unroll 4
        for (int i = k0; i < k1; i++)
#pragma unroll
            for (int t = 0; t < 4; t++)
                nan[t] |= isnan(row[t][i]);
    }
    float s0[4], s1[4];
    bool sums = false;
#pragma unroll
    for (int t = 0; t < 4; t++) {
        s0[t] = s1[t] = nan[t] ? __int_as_float(0x7fffffff) : 0.0f;
        sums |= !nan[t] && (bad >> t & 1);
    }
    if (sums) {
#pragma unroll 1
        for (int i = k0; i < k1; i += 4) {
            const float4 u = load4(w + i);
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const float *p = row[t] + i;
                const float4 v = a_vec ? load4(p) : make_float4(p[0], p[1], p[2], p[3]);
                s0[t] = fmaf(v.x, u.x, s0[t]);
                s1[t] = fmaf(v.y, u.y, s1[t]);
                s0[t] = fmaf(v.z, u.z, s0[t]);
                s1[t] = fmaf(v.w, u.w, s1[t]);
            }
        }
    }
#pragma unroll
    for (int t = 0; t < 4; t++, to += step)
        if (bad >> t & 1)
            *to = add ? *to + (s0[t] + s1[t]) : s0[t] + s1[t];
}

template <int BN>
__global__ void __launch_bounds__(F32Cfg<BN>::THREADS, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a,
                   const float *A, const float *__restrict__ W, float *out, float *part, const F32Work work,
                   int a_vec, int early)
{
    using Cfg = F32Cfg<BN>;
    constexpr int BOXES = Cfg::BOXES, BUFS = Cfg::BUFS, SLOTS = Cfg::B_SLOTS;
    constexpr bool FEW = Cfg::FEW;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *b_smem = smem + BOXES * BOX_BYTES;
    uint64_t *bars = (uint64_t *)(b_smem + SLOTS * Cfg::SLOT_BYTES);
    uint32_t *tmem_slot = (uint32_t *)(bars + Cfg::BARS);
    volatile int *abort = (volatile int *)(tmem_slot + 1);
    // a box of weights is there, may be overwritten; a block's parts of weights are in tensor memory; its MMAs are
    // through; the tokens' parts are in shared memory, may be overwritten (FEW: when the MMAs are through); an
    // accumulator has been read
    const uint32_t w_full = smem_u32(bars), w_empty = w_full + 8 * BOXES, a_full = w_empty + 8 * BOXES,
                   done = a_full + 8 * BUFS, b_full = done + 8 * BUFS, b_empty = b_full + 8 * SLOTS,
                   acc_empty = b_empty + 8 * SLOTS;
    int warp = (int)warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        prefetch_tensor_map(&map_w);
        if (!FEW)
            prefetch_tensor_map(&map_a);
        for (int s = 0; s < BOXES; s++) {
            mbar_init(w_full + 8 * s, 1);
            mbar_init(w_empty + 8 * s, 4);
        }
        for (int b = 0; b < BUFS; b++) {
            mbar_init(a_full + 8 * b, 4);
            mbar_init(done + 8 * b, 1);
        }
        for (int b = 0; b < SLOTS; b++) {
            mbar_init(b_full + 8 * b, FEW ? Cfg::TOK_WARPS : 1);
            mbar_init(b_empty + 8 * b, 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(acc_empty + 8 * b, Cfg::EPI_WARPS);
        }
        *abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = warp_uniform(*tmem_slot), tmem_acc = tmem + BUFS * A_COLS;
    pdl_trigger();

    // Every role walks the CTA's blocks with a cursor, and the places of a ring with a Ring: the place of the use that is
    // next, and its phase's parity.  full(): that use's own phase; empty(): the end of the use before it in the same
    // place (a barrier that is new takes the phase before its first for complete).
    int *const err = &g_gemm_f32_tc_error;
    auto full = [&](uint32_t bars0, const Ring &r, int code) { return mbar_wait(bars0 + 8 * r.at, r.parity, abort, err, code); };
    auto empty = [&](uint32_t bars0, const Ring &r, int code) { return mbar_wait(bars0 + 8 * r.at, r.parity ^ 1, abort, err, code); };

    if (warp == 0) {
        if (lane == 0) {
            // -------------------------------------------------- weights by TMA
            // (they do not depend on the kernel ahead: the ring fills while that one ends)
            if (!early)
                pdl_wait();
            Ring box;
            int asked = 0;
            bool ok = true;
            for (F32Cursor c(work); ok && c.valid(); c.next()) {
#pragma unroll
                for (int h = 0; h < F_BK / BOX_K; h++) {
                    ok = ok && empty(w_empty, box, 1);
                    if (ok) {
                        mbar_expect_tx(w_full + 8 * box.at, BOX_BYTES);
                        tma_load_2d(smem_u32(smem) + box.at * BOX_BYTES, &map_w, w_full + 8 * box.at,
                                    c.kb * F_BK + h * BOX_K, c.m0());
                        box.next(BOXES);
                        asked++;
                    }
                }
            }
            if (*abort) {
                // the loads in flight: the last one of every place, once, with the limit
                volatile int never = 0;
                for (int b = asked > BOXES ? asked - BOXES : 0; b < asked; b++)
                    mbar_wait(w_full + 8 * (b % BOXES), (b / BOXES) & 1, &never, err, 5);
            }
        }
    } else if (warp == 1) {
        {
            // ------------------------------------------------------------ MMAs
            // (the lanes wait side by side; a wait that runs out raises *abort, and all of them leave)
            auto all = [](bool ok) { return __all_sync(0xffffffffu, ok); };
            constexpr uint32_t idesc = instr_desc_bf16(F_M, BN, false);
            const uint32_t slots = smem_u32(b_smem);
            Ring buf, accum, slot;
            // what a block needs besides its MMAs' issue is kept short: nothing runs on the tensor core meanwhile
            for (int left = F32Cursor(work).left(); left > 0; left--) {
                const uint32_t wt = tmem + buf.at * A_COLS, acc = tmem_acc + accum.at * BN;
                // all of the block's k for part pw of the weights and the tokens' part at bt
                auto products = [&](int pw, uint32_t bt, bool first) {
                    tc_mma_ts_block(acc, wt + pw * (F_BK / 2), smem_desc_sw128(bt, 16, 1024), idesc, !first);
                };
                // (asked together; one after the other only if one is not there yet)
                bool ready = mbar_try(a_full + 8 * buf.at, buf.parity) & mbar_try(acc_empty + 8 * accum.at, accum.parity ^ 1) &
                             mbar_try(b_full + 8 * slot.at, slot.parity);
                if (!all(ready) && !all(full(a_full, buf, 2) && empty(acc_empty, accum, 2) && full(b_full, slot, 2)))
                    break;
                tc_fence_after();
                if constexpr (FEW) {
                    const uint32_t hi = slots + slot.at * Cfg::SLOT_BYTES, mid = hi + Cfg::PART_BYTES, lo = mid + Cfg::PART_BYTES;
                    products(0, lo, true);
                    products(1, mid, false);
                    products(2, hi, false);
                    products(0, mid, false);
                    products(1, hi, false);
                    products(0, hi, false);
                    slot.next(SLOTS);
                } else {
                    // the tokens' parts come as lo, mid, hi, each in a slot of its own, and go as early as they can
                    products(0, slots + slot.at * Cfg::SLOT_BYTES, true);
                    tc_commit_warp(b_empty + 8 * slot.at);
                    slot.next(SLOTS);
                    const uint32_t mid = slots + slot.at * Cfg::SLOT_BYTES, mid_bar = b_empty + 8 * slot.at;
                    if (!all(full(b_full, slot, 2)))
                        break;
                    tc_fence_after();
                    products(1, mid, false);
                    slot.next(SLOTS);
                    const uint32_t hi = slots + slot.at * Cfg::SLOT_BYTES;
                    if (!all(full(b_full, slot, 2)))
                        break;
                    tc_fence_after();
                    products(2, hi, false);
                    products(0, mid, false);
                    tc_commit_warp(mid_bar);
                    products(1, hi, false);
                    products(0, hi, false);
                    tc_commit_warp(b_empty + 8 * slot.at);
                    slot.next(SLOTS);
                }
                tc_commit_warp(done + 8 * buf.at);
                buf.next(BUFS);
                accum.next(2);
            }
            if (all(*abort != 0)) {
                // the MMAs in flight, with the limit, before the tensor memory is given back: one more commit,
                // onto the barrier of the use that is still open
                volatile int never = 0;
                tc_commit_warp(done + 8 * buf.at);
                mbar_wait(done + 8 * buf.at, buf.parity, &never, err, 6);
            }
        }
    } else if (warp < 4) {
        if constexpr (!FEW) {
            // ------------------------------------------------ tokens' parts by TMA
            if (warp == 2 && lane == 0) {
                pdl_wait();
                Ring slot;
                int asked = 0;
                bool ok = true;
                for (F32Cursor c(work); ok && c.valid(); c.next()) {
#pragma unroll
                    for (int j = 0; j < 3; j++) {          // lo, mid, hi
                        ok = ok && empty(b_empty, slot, 3);
                        if (ok) {
                            mbar_expect_tx(b_full + 8 * slot.at, Cfg::PART_BYTES);
                            tma_load_2d(smem_u32(b_smem) + slot.at * Cfg::PART_BYTES, &map_a, b_full + 8 * slot.at,
                                        c.kb * F_BK, (2 - j) * work.n + c.n0(BN));
                            slot.next(SLOTS);
                            asked++;
                        }
                    }
                }
                if (*abort) {
                    volatile int never = 0;
                    for (int u = asked > SLOTS ? asked - SLOTS : 0; u < asked; u++)
                        mbar_wait(b_full + 8 * (u % SLOTS), (u / SLOTS) & 1, &never, err, 5);
                }
            }
        }
    } else if (warp < 4 + Cfg::CONV_WARPS) {
        // -------------------------------------------------- weights' parts into tensor memory
        // (with eight warps two groups of four take turns)
        constexpr int GROUPS = Cfg::CONV_WARPS / 4;
        const int group = (warp - 4) / 4, r = (warp & 3) * 32 + lane;         // r: this thread's feature of the tile
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
        bool ok = true;
        Ring buf, box;
        const int blocks = F32Cursor(work).left();
        for (int i = 0; ok && i < blocks; i++) {
            if (GROUPS > 1 && i % GROUPS != group) {
                buf.next(BUFS);
                box.next(BOXES);
                box.next(BOXES);
                continue;
            }
            ok = empty(done, buf, 4);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok)
                break;
            tc_fence_after();
            uint32_t to = tmem + lanes + buf.at * A_COLS;
            static_assert(F_BK == 2 * BOX_K, "two boxes a block");
#pragma unroll
            for (int h = 0; h < 2; h++) {
                ok = full(w_full, box, 4);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok)
                    break;
                const uint8_t *row = smem + box.at * BOX_BYTES + r * 128;
#pragma unroll
                for (int g = 0; g < 2; g++) {              // 16 values at a time
                    uint32_t p0[8], p1[8], p2[8];
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        float4 v = *reinterpret_cast<const float4 *>(row + (((g * 4 + c) ^ (r & 7)) << 4));
                        parts_of(v.x, v.y, p0[2 * c], p1[2 * c], p2[2 * c]);
                        parts_of(v.z, v.w, p0[2 * c + 1], p1[2 * c + 1], p2[2 * c + 1]);
                    }
                    uint32_t at = to + h * 16 + g * 8;
                    tc_st8(at, p0);
                    tc_st8(at + F_BK / 2, p1);
                    tc_st8(at + F_BK, p2);
                }
                __syncwarp();
                if (lane == 0)
                    mbar_arrive(w_empty + 8 * box.at);
                box.next(BOXES);
            }
            tc_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0 && ok)
                mbar_arrive(a_full + 8 * buf.at);
            buf.next(BUFS);
        }
    } else if (FEW && warp >= 4 + Cfg::CONV_WARPS + Cfg::EPI_WARPS) {
        if constexpr (FEW) {
            // ------------------------------------------ tokens' parts from the floats
            // a thread has four values of k of two tokens (all of them are one tile's); the next blocks' are on their way
            constexpr int ROWS = 2 * Cfg::TOK_WARPS, AHEAD = 4;
            static_assert(2 * ROWS == BN, "two tokens a thread");
            const int t = threadIdx.x - 32 * (4 + Cfg::CONV_WARPS + Cfg::EPI_WARPS), row = t >> 4, c4 = t & 15;
            const float *const p0 = A + (size_t)row * work.k + c4 * 4, *const p1 = p0 + (size_t)ROWS * work.k;
            const bool have0 = row < work.n, have1 = row + ROWS < work.n;
            float4 next[AHEAD][2];
            F32Cursor ahead(work);
            auto load = [&](const float *p, bool have) {
                int at = ahead.kb * F_BK;
                p += at;
                if (!have || !ahead.valid() || at + c4 * 4 >= work.k)             // (k is a multiple of four)
                    return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                return a_vec ? *reinterpret_cast<const float4 *>(p) : make_float4(p[0], p[1], p[2], p[3]);
            };
            pdl_wait();
#pragma unroll
            for (int d = 0; d < AHEAD; d++) {
                next[d][0] = load(p0, have0);
                next[d][1] = load(p1, have1);
                if (ahead.valid())
                    ahead.next();
            }
            F32Cursor c(work);
            Ring buf;
            static_assert(BUFS == SLOTS, "a block's tokens go with its weights");
            bool ok = true;
            while (ok && c.valid()) {
                // (unrolled, so that every block has registers of its own: moving a value waits for its load)
#pragma unroll
                for (int d = 0; d < AHEAD; d++) {
                    if (!c.valid())
                        break;
                    ok = empty(done, buf, 3);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok)
                        break;
                    uint8_t *dst = b_smem + buf.at * Cfg::SLOT_BYTES + row * 128 + (((c4 >> 1) ^ (row & 7)) << 4) + ((c4 & 1) << 3);
#pragma unroll
                    for (int j = 0; j < 2; j++) {              // (ROWS is a multiple of eight: the swizzle is the same)
                        uint2 p[3];
                        parts_of(next[d][j].x, next[d][j].y, p[0].x, p[1].x, p[2].x);
                        parts_of(next[d][j].z, next[d][j].w, p[0].y, p[1].y, p[2].y);
#pragma unroll
                        for (int q = 0; q < 3; q++)
                            *reinterpret_cast<uint2 *>(dst + q * Cfg::PART_BYTES + j * ROWS * 128) = p[q];
                        next[d][j] = load(j == 0 ? p0 : p1, j == 0 ? have0 : have1);
                    }
                    if (ahead.valid())
                        ahead.next();
                    c.next();
                    fence_async_smem();
                    __syncwarp();
                    if (lane == 0)
                        mbar_arrive(b_full + 8 * buf.at);
                    buf.next(BUFS);
                }
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue
        // a thread has one feature and COLS tokens
        constexpr int COLS = Cfg::COLS;
        const int q = warp & 3, c0 = (warp - 4 - Cfg::CONV_WARPS) / 4 * COLS;
        const uint32_t from = tmem_acc + ((uint32_t)(q * 32) << 16) + c0;
        pdl_wait();                         // no store before the kernel before this one is done
        F32Cursor cur(work);
        bool ok = true;
        Ring buf, accum;
        for (; ok && cur.valid(); cur.next()) {
            // a segment: its blocks' sums added up
            float sum[COLS];
#pragma unroll
            for (int c = 0; c < COLS; c++)
                sum[c] = 0.0f;
#pragma unroll 1
            for (bool last = false; !last; cur.kb += !last) {
                ok = full(done, buf, 7);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok)
                    break;
                tc_fence_after();
#pragma unroll
                for (int c = 0; c < COLS; c += 16) {
                    uint32_t v[16];
                    tc_ld16_nowait(from + accum.at * BN + c, v);
                    tc_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; j++)
                        sum[c + j] += __uint_as_float(v[j]);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0)
                    mbar_arrive(acc_empty + 8 * accum.at);
                buf.next(BUFS);
                accum.next(2);
                last = cur.last();
            }
            const int f0 = cur.m0(), f = f0 + q * 32 + lane, n0 = cur.n0(BN) + c0, rows = min(COLS, work.n - n0);
            if (!ok || f >= work.m)
                continue;
            const bool whole = cur.whole(), add = whole && cur.seg > 0;
            float *p = whole ? out + (size_t)n0 * work.m + f
                             : part + (((size_t)(cur.tile - work.whole) * work.segments + cur.seg) * BN + c0) * F_M + (f - f0);
            const size_t step = whole ? work.m : F_M;
            uint32_t bad[(COLS + 31) / 32] = {};
            float *to = p;
#pragma unroll
            for (int c = 0; c < COLS; c += 8) {
                float had[8];
                float *at = to;
#pragma unroll
                for (int j = 0; j < 8; j++, at += step)
                    had[j] = add && c + j < rows ? *at : 0.0f;
#pragma unroll
                for (int j = 0; j < 8; j++, to += step)
                    if (c + j < rows) {
                        float v = sum[c + j];
                        if (fabsf(v) <= 3.402823466e38f) {
                            v *= F_DOWN;
                            *to = add ? had[j] + v : v;
                        } else {
                            bad[(c + j) / 32] |= 1u << ((c + j) % 32);
                        }
                    }
            }
#pragma unroll
            for (int w = 0; w < (COLS + 31) / 32; w++)
                while (bad[w]) {
                    const int g = (__ffs(bad[w]) - 1) & ~3, c = w * 32 + g;
                    plain_sums(A + (size_t)(n0 + c) * work.k, work.k, rows - c - 1, a_vec, W + (size_t)f * work.k,
                               cur.seg * work.seg_blocks * F_BK, min(work.k, (cur.seg + 1) * work.seg_blocks * F_BK),
                               bad[w] >> g & 15, p + (size_t)c * step, step, add);
                    bad[w] &= ~(15u << g);
                }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                     ::"r"(tmem), "r"(512u) : "memory");
    }
}

// The three parts of A [n, k] as matrices [n, kp] one after the other (kp: k up to a multiple of eight; the rest zeros).
// Four values a thread.
__global__ void __launch_bounds__(256)
f32_parts_kernel(const float *A, bf16 *__restrict__ planes, int n, int k, int kp, int a_vec)
{
    pdl_trigger();
    int fours = kp / 4;
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    pdl_wait();
    if (i >= (size_t)n * fours)
        return;
    size_t r = i / fours;
    int c = (int)(i - r * fours) * 4;
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const float *p = A + r * k + c;
    if (c < k)                                              // (k is a multiple of four)
        v = a_vec ? *reinterpret_cast<const float4 *>(p) : make_float4(p[0], p[1], p[2], p[3]);
    uint2 q[3];
    parts_of(v.x, v.y, q[0].x, q[1].x, q[2].x);
    parts_of(v.z, v.w, q[0].y, q[1].y, q[2].y);
#pragma unroll
    for (int j = 0; j < 3; j++)
        *reinterpret_cast<uint2 *>(planes + ((size_t)j * n + r) * kp + c) = q[j];
}

// The segments' sums of the tiles that were shared out, added in ascending order: four features of a token a thread.
__global__ void __launch_bounds__(256)
f32_join_kernel(const float *part, float *__restrict__ out, int n, int m, int n_tiles, int whole, int segments, int BN)
{
    pdl_trigger();
    int per_tile = BN * F_M / 4;
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    int tile = (int)(i / per_tile), at = (int)(i - (size_t)tile * per_tile), c = at / (F_M / 4), f4 = at % (F_M / 4) * 4;
    int r = (tile + whole) % n_tiles * BN + c, f = (tile + whole) / n_tiles * F_M + f4;
    pdl_wait();
    if (r >= n || f >= m)           // (tiles past the last have features past the last)
        return;
    const float *p = part + ((size_t)tile * segments * BN + c) * F_M + f4;
    const size_t step = (size_t)BN * F_M;
    float4 t = load4(p);
    for (int s = 1; s < segments; s += 8) {
        float4 v[8];
#pragma unroll
        for (int u = 0; u < 8; u++)
            if (s + u < segments)
                v[u] = load4(p + (s + u) * step);
#pragma unroll
        for (int u = 0; u < 8; u++)
            if (s + u < segments) {
                t.x += v[u].x;
                t.y += v[u].y;
                t.z += v[u].z;
                t.w += v[u].w;
            }
    }
    float *o = out + (size_t)r * m + f;
    if (m % 4 == 0) {
        store4(o, t);
    } else {
        const float e[4] = {t.x, t.y, t.z, t.w};
        for (int j = 0; j < 4 && f + j < m; j++)
            o[j] = e[j];
    }
}

// ------------------------------------------------------------------ host side
// Tokens of a tile: the least padding, and of equals the wider tile (a weight is taken apart once a tile).
static int f32_tile(int n)
{
    if (n <= 16)
        return 16;
    if (n <= 32)
        return 32;
    const int choices[4] = {160, 128, 96, 64};
    int best = 0;
    long long best_t = 0;
    for (int bn : choices) {
        long long t = (long long)((n + bn - 1) / bn) * (bn + 32);       // (32: what a tile costs besides)
        if (best == 0 || t < best_t) {
            best_t = t;
            best = bn;
        }
    }
    return best;
}

// Blocks of k of a segment, by the weight alone: so many segments that the feature tiles' segments are at most as many
// as the SMs (148), of four blocks at least; eight blocks where the tiles alone are more.  One tile of tokens then takes
// one round of about equal pieces (8 tokens, us, segments of eight blocks in brackets: 2560 x 4096 14.4 (18.5), 2560 x 9728
// 23.2 (27.4), 6144 x 2560 16.9 (19.4), 512 x 2560 7.8 (10.3)).
static int f32_seg_blocks(int m, int k)
{
    int tiles = (m + F_M - 1) / F_M, blocks = (k + F_BK - 1) / F_BK;
    if (tiles > 148)
        return 8;
    int segments = 148 / tiles, len = (blocks + segments - 1) / segments;
    return len < 4 ? 4 : len;
}

// How the next rows of a call are taken: `rows` of them, all at once where the scratch is enough for that.  A row's bits
// do not depend on it.
struct F32Plan {
    int rows, bn, seg_blocks, segments;
    long long whole, rest;              // tiles taken over all of k, and shared out by segments
    long long plane_floats, part_floats;
    long long floats() const { return plane_floats + part_floats; }
};

static F32Plan f32_pass(int rows, int m, int k, bool share)
{
    F32Plan p;
    p.rows = rows;
    p.bn = f32_tile(rows);
    p.seg_blocks = f32_seg_blocks(m, k);
    p.segments = ((k + F_BK - 1) / F_BK + p.seg_blocks - 1) / p.seg_blocks;
    long long tiles = ((long long)m + F_M - 1) / F_M * (((long long)rows + p.bn - 1) / p.bn), places = sm_count();
    // tiles that fill every SM are taken whole; the rest is shared out by segments where that ends earlier
    p.rest = tiles % places;
    if (!share || (p.rest * p.segments + places - 1) / places >= p.segments)
        p.rest = 0;
    p.whole = tiles - p.rest;
    p.part_floats = p.rest * p.segments * p.bn * F_M;
    p.plane_floats = p.bn > 32 ? (3ll * rows * ((k + 7) / 8 * 8) / 2 + 63) / 64 * 64 : 0;
    return p;
}

// The scratch that a call asks for at most.  Planes (6 bytes a value) and shared segments of all rows at once would take
// 184 MB for 2,048 rows of 2560 x 9728; two passes of 1,024 rows take 65 MB and, by rounds of tiles, the same time.
constexpr long long F32_SCRATCH = 18ll << 20;           // floats

// The next pass of n rows with `have` floats of scratch: equal passes, as few as fit; up to 32 rows need none.
static F32Plan f32_plan(int n, int m, int k, long long have)
{
    for (int passes = 1;; passes++) {
        int rows = passes == 1 ? n : (int)(((long long)n + passes - 1) / passes + 31) / 32 * 32;
        if (rows > n)
            rows = n;
        F32Plan p = f32_pass(rows, m, k, true);
        if (p.floats() <= have)
            return p;
        if (rows <= 32)
            return f32_pass(rows, m, k, false);
    }
}

template <int BN>
static int f32_launch(const CUtensorMap &map_w, const CUtensorMap &map_a, const float *A, const float *W, float *out,
                      float *part, const F32Work &work, int a_vec, int early, cudaStream_t st)
{
    using Cfg = F32Cfg<BN>;
    static unsigned long long allowed = 0;
    if (!allow_dynamic_smem(gemm_f32_tc_kernel<BN>, Cfg::SMEM_BYTES, allowed))
        return JB_ELAUNCH;
    int places = sm_count();
    launch(gemm_f32_tc_kernel<BN>, (unsigned)(work.units < places ? work.units : places), Cfg::THREADS, Cfg::SMEM_BYTES,
           st, map_w, map_a, A, W, out, part, work, a_vec, early);
    return launch_status();
}

}  // namespace jb

using namespace jb;

// Whether this kernel takes a product; says nothing about n, so that a row's bits do not depend on the batch.  That costs
// a step of 1 to 8 rows a little where the weight has few tiles and moderate k, or is a head: in a captured chain of norm
// and product, us, this kernel and gemm_simt.cu, 1 / 8 / 16 / 32 rows: 2560 x 4096 15.7 / 16.8 / 17.2 / 19.3 and
// 14.9 / 15.4 / 20.9 / 35.2; 2048 x 6144 16.5 / 18.0 / 18.6 / 20.2 and 15.7 / 16.1 / 21.6 / 35.7; 4096 x 2560 14.2 /
// 15.0 / 15.6 / 17.0 and 14.1 / 14.6 / 20.1 / 34.3; a head of 151,936 x 2560 269 to 290 / 264 to 284 / 293 / 318 to 345
// and 266 / 270 / 367 / 620 (by box: it is the clock's, the plain kernel's is the memory's).  Everything else measured is
// ahead from one row on (19456 x 2560 46 / 47 / 48 / 55 and 50 / 53 / 72 / 110), all of them are from 16 rows on, and a
// prompt takes a quarter of the time.  A whole 36-layer step of 8 rows: 5.73 ms, 5.83 by plain multiply-adds.
// Smaller weights are left to the plain kernel: at 8 tokens 512 x 1024 takes 7.3 us (7.8 there) and 1000 x 1028 7.5 (7.8), but
// 512 x 512 7.2 (6.7), 2560 x 512 7.4 (6.8) and 256 x 256 5.4 (3.9).  Longer rows too: a tile whose sums are all infinite
// takes the epilogue some 4,500 cycles a k (23 ms at 9,728), and the others' waits end after 2 * 10^9.
extern "C" int jb_gemm_f32_tc_ok(const void *W, int m, int k)
{
    return m >= 512 && k >= 1024 && k % 4 == 0 && (uintptr_t)W % 16 == 0 && k <= 1 << 17;
}

// Floats of scratch that a call asks for (0: none; it makes do with less, or with none, at some cost in time), and kernels
// that it launches with `have` of them.
extern "C" long long jb_gemm_f32_tc_scratch(int n, int m, int k)
{
    long long most = 0;
    for (int r0 = 0; r0 < n && m > 0 && k > 0;) {
        F32Plan p = f32_plan(n - r0, m, k, F32_SCRATCH);
        most = p.floats() > most ? p.floats() : most;
        r0 += p.rows;
    }
    return most;
}
extern "C" int jb_gemm_f32_tc_launches(int n, int m, int k, long long have)
{
    int kernels = 0;
    for (int r0 = 0; r0 < n && m > 0 && k > 0;) {
        F32Plan p = f32_plan(n - r0, m, k, have);
        kernels += 1 + (p.plane_floats > 0) + (p.rest > 0);
        r0 += p.rows;
    }
    return kernels;
}

static int f32_run(const F32Plan &p, const float *A, const float *W, float *out, int m, int k, float *scratch, int early,
                   cudaStream_t st)
{
    const int n = p.rows;
    F32Work work;
    work.n = n;
    work.m = m;
    work.k = k;
    work.n_tiles = (n + p.bn - 1) / p.bn;
    work.segments = p.segments;
    work.seg_blocks = p.seg_blocks;
    work.blocks = (k + F_BK - 1) / F_BK;
    if (p.whole + p.rest * p.segments > 0x7fffffffll || 3ll * n > 0x7fffffffll)
        return JB_EINVAL;
    work.whole = (int)p.whole;
    work.units = (int)(p.whole + p.rest * p.segments);
    const int a_vec = (uintptr_t)A % 16 == 0, kp = (k + 7) / 8 * 8;
    CUtensorMap map_w, map_a;
    if (!tensor_map_2d(W, m, k, F_M, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, &map_w))
        return JB_EINVAL;
    map_a = map_w;
    float *part = p.part_floats > 0 ? scratch + p.plane_floats : nullptr;
    if (p.plane_floats > 0) {
        if (!tensor_map_2d(scratch, 3 * n, kp, p.bn, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, &map_a))
            return JB_EINVAL;
        launch(f32_parts_kernel, (unsigned)(((size_t)n * (kp / 4) + 255) / 256), 256, 0, st, A, (bf16 *)scratch, n, k, kp,
               a_vec);
        if (cudaGetLastError() != cudaSuccess)
            return JB_ELAUNCH;
    }
    int rc;
#define JB_FP(B) rc = f32_launch<B>(map_w, map_a, A, W, out, part, work, a_vec, early, st)
    switch (p.bn) {
    case 16: JB_FP(16); break;
    case 32: JB_FP(32); break;
    case 64: JB_FP(64); break;
    case 96: JB_FP(96); break;
    case 128: JB_FP(128); break;
    default: JB_FP(160); break;
    }
#undef JB_FP
    if (rc != JB_OK || p.rest == 0)
        return rc;
    launch(f32_join_kernel, (unsigned)(((size_t)p.rest * p.bn * (F_M / 4) + 255) / 256), 256, 0, st, (const float *)part, out,
           n, m, work.n_tiles, work.whole, work.segments, p.bn);
    return launch_status();
}

// scratch: `have` floats, 16-byte aligned; jb_gemm_f32_tc_scratch says how many are worth having, and the results do not
// depend on it.  early: as jb_gemm_simt.
extern "C" int jb_gemm_f32_tc(const void *A, const void *W, float *out, int n, int m, int k, float *scratch,
                              long long have, int early, cudaStream_t st)
{
    if (n <= 0 || m <= 0)
        return JB_OK;
    if (!jb_gemm_f32_tc_ok(W, m, k) || (uintptr_t)A % 4 || (uintptr_t)out % 4 || (uintptr_t)scratch % 16)
        return JB_EINVAL;
    if (scratch == nullptr || have < 0)
        have = 0;
    int rc = JB_OK;
    for (int r0 = 0; r0 < n && rc == JB_OK;) {
        F32Plan p = f32_plan(n - r0, m, k, have);
        rc = f32_run(p, (const float *)A + (size_t)r0 * k, (const float *)W, out + (size_t)r0 * m, m, k, scratch, early, st);
        r0 += p.rows;
    }
    return rc;
}

extern "C" int jb_gemm_f32_tc_error(void)
{
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_gemm_f32_tc_error, sizeof v) != cudaSuccess)
        return JB_ELAUNCH;
    if (v != 0)
        cudaMemcpyToSymbol(g_gemm_f32_tc_error, &zero, sizeof zero);
    return v;
}
