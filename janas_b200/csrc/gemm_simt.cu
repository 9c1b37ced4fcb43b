// out[n, m] = A[n, k] . W[m, k]^T with plain float multiply-adds.
//
// This is the matrix product of the true 32-bit path for weights that are small
// or whose rows TMA does not take (the others: gemm_f32_tc.cu), and the fallback
// for shapes and type mixes the bfloat16 tensor-core kernel refuses.  Every output value is
// computed by one fixed recipe, whatever n is and wherever the row lies in the
// batch, so a row's result is the same bits however the tokens are cut into
// steps: k is cut into segments of SEG values at fixed places; within a segment
// the products of even k and of odd k are added by one chain of fmaf each, in
// ascending order from zero, and the two sums are added; the segments' sums are
// added in ascending order.  One kernel follows the recipe for every shape: a
// block walks one or more segments of a tile of rows and features.  Where tiles
// alone leave the SMs without work, the segments are shared out over blocks, which
// leave their sums in scratch for a second kernel that adds them in order.
// A and W are float or bfloat16 (widened exactly); no reduced-precision matrix
// mode is involved.
//
// The reference computes y = W x with rows of W as output features
// (src/llm/model_load.c:452, src/llm/model_attn.c:234-255); its products are
// over quantized blocks and are not reproduced.
#include "common.cuh"
#include "kernels.h"

namespace jb {

constexpr int BK = 64;        // k of a stage
constexpr int SEG = 512;      // k of a segment
static_assert(SEG % BK == 0, "segments end where stages end");
// values a row of a stage takes in shared memory: a multiple of 16 bytes, and neighbouring rows start in other banks
template <typename T> constexpr int ROW = BK + 16 / (int)sizeof(T);

// Four consecutive values of a row in shared memory as two pairs.
__device__ __forceinline__ void pairs(const float *p, f32x2 &lo, f32x2 &hi)
{
    ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(p);
    lo = v.x;
    hi = v.y;
}
__device__ __forceinline__ void pairs(const bf16 *p, f32x2 &lo, f32x2 &hi)
{
    uint2 u = *reinterpret_cast<const uint2 *>(p);
    lo = (f32x2)(u.x & 0xffff0000u) << 32 | u.x << 16;
    hi = (f32x2)(u.y & 0xffff0000u) << 32 | u.y << 16;
}

// Asks for ROWS rows of BK values from k0 on, src[row0 + r][k0 ..], to be put into a stage, BYTES (4, 8 or 16) at a
// time; 2 bytes: values loaded and stored, sixteen of a thread on their way together.  Rows from `have` on and values
// from kb on become zeros; k and kb are multiples of what a copy takes.
template <typename T, int ROWS, int THREADS, int BYTES>
__device__ __forceinline__ void fetch_by(T *stage, const T *__restrict__ src, long long row0, int have, int k,
                                         int k0, int kb)
{
    constexpr int V = BYTES / sizeof(T), PER = BK / V, STEP = THREADS / PER, N = ROWS / STEP;
    static_assert(THREADS % PER == 0 && ROWS % STEP == 0, "a thread has the same place in every STEP-th row");
    int r = threadIdx.x / PER, c = threadIdx.x % PER * V;
    const T *p = src + (row0 + r) * (size_t)k + k0 + c;
    int rows = k0 + c < kb ? (int)min(have - row0, (long long)ROWS) - r : 0;
    T *dst = stage + r * ROW<T> + c;
    if constexpr (BYTES == 2) {
        constexpr int B = N < 16 ? N : 16;
#pragma unroll 1
        for (int i = 0; i < N; i += B) {
            T v[B];
#pragma unroll
            for (int u = 0; u < B; u++) {
                v[u] = (i + u) * STEP < rows ? *p : from_f<T>(0.0f);
                p += STEP * (size_t)k;
            }
#pragma unroll
            for (int u = 0; u < B; u++)
                dst[(i + u) * STEP * ROW<T>] = v[u];
        }
    } else {
        constexpr int UNROLL = BYTES == 16 || N < 8 ? N : 8;
        uint32_t to = (uint32_t)__cvta_generic_to_shared(dst);
#pragma unroll UNROLL
        for (int i = 0; i < N; i++) {
            bool in = i * STEP < rows;
            const T *from = in ? p : src;
            if constexpr (BYTES == 16)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(from), "r"(in ? 16 : 0)
                             : "memory");
            else
                asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(to), "l"(from), "n"(BYTES),
                             "r"(in ? BYTES : 0)
                             : "memory");
            p += STEP * (size_t)k;
            to += STEP * ROW<T> * (int)sizeof(T);
        }
    }
}

// bytes: what copy_bytes said.
template <typename T, int ROWS, int THREADS>
__device__ __forceinline__ void fetch(T *stage, const T *__restrict__ src, long long row0, int have, int k,
                                      int k0, int kb, int bytes)
{
    if (bytes == 16)
        fetch_by<T, ROWS, THREADS, 16>(stage, src, row0, have, k, k0, kb);
    else if (bytes == 8)
        fetch_by<T, ROWS, THREADS, 8>(stage, src, row0, have, k, k0, kb);
    else if (sizeof(T) == 4 || bytes == 4)
        fetch_by<T, ROWS, THREADS, 4>(stage, src, row0, have, k, k0, kb);
    else if constexpr (sizeof(T) == 2)
        fetch_by<T, ROWS, THREADS, 2>(stage, src, row0, have, k, k0, kb);
}

// A block's threads stand TX along the features and TY along the rows; a thread owns the rows
// ty + TY i (i < RT) and the features tx + TX j (j < CT) of the block's tile.  Along k, four values of a row
// or feature come out of shared memory in one access and feed CT or RT pairs of multiply-adds.
// KEEP: the sum over the segments stays in registers (else in shared memory, each thread its own).
template <int RT, int CT, int TX, int TY, int ST> struct SimtTile {
    static constexpr int R = RT, C = CT, X = TX, Y = TY, STAGES = ST;
    static constexpr bool KEEP = RT * CT <= 16;
    static constexpr int ROWS = RT * TY, FEATS = CT * TX, THREADS = TX * TY;
    template <typename TA, typename TW> static constexpr int smem()
    {
        return ST * (ROW<TA> * ROWS * (int)sizeof(TA) + ROW<TW> * FEATS * (int)sizeof(TW)) + (KEEP ? 0 : ROWS * FEATS * 4);
    }
};

// grid: x row tiles and feature tiles, the row tiles next to each other (so that the blocks that read the
// same weights run at the same time), z groups of segments.  With one group the sums of a block's
// segments stay with its threads and `out` is the result; else each segment's sums go to
// out[segment][n][m].
template <typename TA, typename TW, typename Tile, bool PARTS>
__global__ void __launch_bounds__(Tile::THREADS, Tile::ROWS == 64 ? 2 : 1)
gemm_simt_kernel(const TA *A, const TW *__restrict__ W, float *__restrict__ out, int n, int m, int k, int row_tiles,
                 int a_bytes, int w_bytes, bool early)
{
    constexpr int RT = Tile::R, CT = Tile::C, TX = Tile::X, TY = Tile::Y, ST = Tile::STAGES, THREADS = Tile::THREADS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TW *Ws = reinterpret_cast<TW *>(smem_raw);
    TA *As = reinterpret_cast<TA *>(Ws + ST * ROW<TW> * Tile::FEATS);
    float *Ts = reinterpret_cast<float *>(As + ST * ROW<TA> * Tile::ROWS);
    pdl_trigger();
    int tid = threadIdx.x;
    // a warp's lanes stand eight along the features and four along the rows where both run, lane bits
    // 0, 2, 4 and 1, 3: neighbours (i ^ 1, i ^ 2) then ask for the same 16 bytes, and an access to shared
    // memory takes fewer turns
    int tx, ty;
    if constexpr (TY % 4 == 0) {
        int w = tid >> 5, l = tid & 31;
        tx = ((l & 1) | (l >> 1 & 2) | (l >> 2 & 4)) + 8 * (w % (TX / 8));
        ty = ((l >> 1 & 1) | (l >> 2 & 2)) + 4 * (w / (TX / 8));
    } else {
        tx = tid % TX;
        ty = tid / TX;
    }
    long long n0 = (long long)(blockIdx.x % row_tiles) * Tile::ROWS, m0 = (long long)(blockIdx.x / row_tiles) * Tile::FEATS;
    int segments = (k + SEG - 1) / SEG;
    int s0 = (int)((long long)segments * blockIdx.z / gridDim.z);
    int s1 = (int)((long long)segments * (blockIdx.z + 1) / gridDim.z);
    int ka = s0 * SEG, kb = min(k, s1 * SEG);
    int steps = (kb - ka + BK - 1) / BK;
    auto fetch_w = [&](int s) {
        fetch<TW, Tile::FEATS, THREADS>(Ws + (s % ST) * ROW<TW> * Tile::FEATS, W, m0, m, k, ka + s * BK, kb, w_bytes);
    };
    auto fetch_a = [&](int s) {
        fetch<TA, Tile::ROWS, THREADS>(As + (s % ST) * ROW<TA> * Tile::ROWS, A, n0, n, k, ka + s * BK, kb, a_bytes);
    };
    // early: the first stages' weights are on their way while the kernel before this one ends
    if (!early)
        pdl_wait();
#pragma unroll 1
    for (int s = 0; s < ST - 1; s++)
        if (s < steps)
            fetch_w(s);
    if (early)
        pdl_wait();
#pragma unroll 1
    for (int s = 0; s < ST - 1; s++) {
        if (s < steps)
            fetch_a(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    f32x2 acc[RT][CT];
    float total[Tile::KEEP ? RT : 1][Tile::KEEP ? CT : 1];
#pragma unroll
    for (int i = 0; i < RT; i++)
#pragma unroll
        for (int j = 0; j < CT; j++) {
            acc[i][j] = 0;
            if (Tile::KEEP)
                total[i][j] = 0.0f;
        }
    for (int s = 0; s < steps; s++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
        __syncthreads();                 // stage s is there for all, and all are done with stage s - 1
        if (s + ST - 1 < steps) {
            fetch_w(s + ST - 1);
            fetch_a(s + ST - 1);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        const TW *ws = Ws + (s % ST) * ROW<TW> * Tile::FEATS + tx * ROW<TW>;
        const TA *as = As + (s % ST) * ROW<TA> * Tile::ROWS + ty * ROW<TA>;
#pragma unroll
        for (int kk = 0; kk < BK; kk += 4) {
            f32x2 w0[CT], w1[CT];
#pragma unroll
            for (int j = 0; j < CT; j++)
                pairs(ws + j * TX * ROW<TW> + kk, w0[j], w1[j]);
#pragma unroll
            for (int i = 0; i < RT; i++) {
                f32x2 a0, a1;
                pairs(as + i * TY * ROW<TA> + kk, a0, a1);
#pragma unroll
                for (int j = 0; j < CT; j++)
                    acc[i][j] = fma2(a0, w0[j], acc[i][j]);
#pragma unroll
                for (int j = 0; j < CT; j++)
                    acc[i][j] = fma2(a1, w1[j], acc[i][j]);
            }
        }
        if ((s + 1) % (SEG / BK) == 0 || s + 1 == steps) {
            // a segment ends
            int seg = s0 + s / (SEG / BK);
#pragma unroll
            for (int i = 0; i < RT; i++) {
                long long r = n0 + ty + TY * i;
#pragma unroll
                for (int j = 0; j < CT; j++) {
                    float v = sum2(acc[i][j]);
                    acc[i][j] = 0;
                    if (PARTS) {
                        long long c = m0 + tx + TX * j;
                        if (r < n && c < m)
                            out[((size_t)seg * n + r) * m + c] = v;
                    } else if (Tile::KEEP) {
                        total[i][j] = seg == 0 ? v : total[i][j] + v;
                    } else {
                        float *t = Ts + (i * CT + j) * THREADS + tid;
                        *t = seg == 0 ? v : *t + v;
                    }
                }
            }
        }
    }
    if (!PARTS) {
#pragma unroll
        for (int i = 0; i < RT; i++) {
            long long r = n0 + ty + TY * i;
#pragma unroll
            for (int j = 0; j < CT; j++) {
                long long c = m0 + tx + TX * j;
                if (r < n && c < m)
                    out[(size_t)r * m + c] = Tile::KEEP ? total[i][j] : Ts[(i * CT + j) * THREADS + tid];
            }
        }
    }
}

// out = ((part[0] + part[1]) + part[2]) + ...: the segments' sums in ascending order, V
// neighbours a thread.
template <int V>
__global__ void __launch_bounds__(256)
gemm_simt_join_kernel(const float *part, float *__restrict__ out, long long count, int segments)
{
    pdl_trigger();
    pdl_wait();
    long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * V;
    if (i >= count)
        return;
    if constexpr (V == 4) {
        float4 t = load4(part + i);
        for (int s = 1; s < segments; s += 4) {
            float4 v[4];
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (s + u < segments)
                    v[u] = load4(part + (size_t)(s + u) * count + i);
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (s + u < segments) {
                    t.x += v[u].x;
                    t.y += v[u].y;
                    t.z += v[u].z;
                    t.w += v[u].w;
                }
        }
        store4(out + i, t);
    } else {
        float t = part[i];
        for (int s = 1; s < segments; s++)
            t = t + part[(size_t)s * count + i];
        out[i] = t;
    }
}

// Which tile: rows up to 8, 16 and 32 stand in one tile, so that a weight is read once; more rows in tiles of 64, or of
// 16 or 8 where those of 64 would be few (simt_rows).
//
// Up to 16 rows the weights' bytes are the bound.  A narrow tile (64 features) leaves room for three blocks on an SM,
// each with two stages of 16 KB on their way; every multiply-add takes its weight from shared memory, and the reads of
// weights (twice per block of 8 rows) are what is fullest.  From 32 rows on the multiply-adds are the bound
// (72.7 TFLOP/s is what this instruction gives); four to eight rows and four features a thread, the stage
// unrolled whole, were the fastest of the tiles tried (8 x 8 a thread, more blocks of fewer registers).
// One B200, float, microseconds (before: blocks of 64 x 64 with 16 values of k a stage, or of 128 features and
// 16 rows), weights from memory, with the second kernel where k is shared out:
//   rows 8:   6144 x 2560  20.3 (80.3)   2560 x 4096  14.7 (77.3)   19456 x 2560  50.2 (113)   151936 x 2560  272 (702)
//   rows 16:  6144 x 2560  28.1 (89.4)   2560 x 4096  19.9 (75.2)   19456 x 2560  70.0 (115)   151936 x 2560  361 (725)
//   rows 64:  6144 x 2560  68.5 (181)    2560 x 4096  45.5 (200)    19456 x 2560  207 (369)    2560 x 9728  117 (472)
//   rows 300: 6144 x 2560  271 (383)     2560 x 4096  172 (309)     19456 x 2560  724 (1,057)  2560 x 9728  414 (729)
// and 2,048 rows run at 47 TFLOP/s (31).  The error against 64 bits is 2.9e-7 of the result (4.1e-7): a chain is
// half as long.
typedef SimtTile<4, 2, 32, 2, 3> Rows8;
typedef SimtTile<4, 4, 16, 4, 3> Rows16;
typedef SimtTile<8, 4, 32, 4, 2> Rows32;
typedef SimtTile<8, 4, 16, 8, 2> Rows64;
static_assert(Rows8::FEATS == Rows64::FEATS && Rows16::FEATS == Rows64::FEATS, "simt_groups counts so");

static int simt_segments(int k) { return (k + SEG - 1) / SEG; }

// Rows of the tile that n rows go with.  A single segment cannot be shared out over blocks: 17 to 32 rows are then two
// tiles of 16, whose blocks are half as long (24 rows, float, us: 96 x 100 3.1 against 5.2, 2560 x 512 11.1 against 17.2, 20000 x 512 26
// against 31; a head of 151,936 features, which fills the chip either way, 143 against 127).
// With more segments one tile is ahead where there are many (2560 x 9728 49 against 69, 6144 x 2560 33 against 46).
//
// More rows: tiles of 64 unless those of 16 or 8 are well ahead, which they are where few tiles of 64 leave the chip
// idle (a block walks its k alone, and one of 8 rows does in 0.4 of the time).  The estimate, in microseconds for a
// segment of 512: what a block alone takes beside others, and what each block takes of the chip's time; both measured.
// One B200, us, float, before (tiles of 64) -> now: 96 x 96, 132 rows 5.0 -> 2.1; 448 x 96, 132 rows 5.3 -> 2.4; 96 x 224,
// 132 rows 8.7 -> 3.6; 512 x 512, 64 rows 16.3 -> 6.4; 2560 x 512, 132 rows 28.7 -> 16.5; 8 x 2560, 300 rows 16.9 -> 11.5.
static int simt_rows(int n, int m, int k)
{
    if (n <= 8)
        return 8;
    if (n <= 16 || (n <= 32 && simt_segments(k) == 1))
        return 16;
    if (n <= 32)
        return 32;
    double columns = ((double)m + Rows64::FEATS - 1) / Rows64::FEATS * simt_segments(k);
    auto cost = [&](int rows, double alone, double each) { return alone + each * ((n + rows - 1) / rows) * columns; };
    double c8 = cost(8, 3.8, 0.022), c16 = cost(16, 5.4, 0.031), c64 = cost(64, 9.8, 0.108) * 0.8;
    return c8 < c16 && c8 < c64 ? 8 : c16 < c64 ? 16 : 64;
}

// Groups of segments: as few as give every SM the blocks that fit it at a time (by shared memory three of 8 or 16 rows,
// two of 64), and for tiles of 32 rows, of which two fit, twice as many.  8 | 16 rows, 2560 x 9728, float: 28.7 | 40.7
// us; counting four of them a SM, whose last round is nearly empty, 32.4 | 44.2.  24 rows, 2560 x 9728 and 19456 x 2560:
// 49 and 107; counting two of them a SM 74 and 121.  The sums that pass through scratch cost 8 bytes a segment, row and
// feature, the weights 4 bytes x 512 a segment and feature.
static int simt_groups(int n, int m, int k)
{
    int rows = simt_rows(n, m, k);
    int feats = rows == Rows32::ROWS ? Rows32::FEATS : Rows64::FEATS;
    long long tiles = ((long long)m + feats - 1) / feats * (((long long)n + rows - 1) / rows);
    long long want = (rows < 32 ? 3 : rows == 32 ? 4 : 2) * (long long)sm_count();
    int segments = simt_segments(k);
    if (tiles >= want)
        return 1;
    return (int)((want + tiles - 1) / tiles < segments ? (want + tiles - 1) / tiles : segments);
}

// The widest copy (16, 8 or 4 bytes; 2: none) that every row of k values from p on starts and ends at a multiple of,
// for each operand by itself.  One B200, 2,560 features, rows 8 | 300 | 1,000, microseconds (before: value by value
// unless both operands could go by 16 bytes):
//   float            k = 2561   16.9 (104)    131 (379)   390 (1,318)
//   bfloat16, float  k = 2564   15.6 (101)    130 (498)   392 (1,052)
//   bfloat16         k = 2561   34.5 (83.9)   206 (374)   570 (954)
template <typename T> static int copy_bytes(const void *p, int k)
{
    unsigned long long at = (unsigned long long)(uintptr_t)p | (unsigned long long)k * sizeof(T);
    return at % 16 == 0 ? 16 : at % 8 == 0 ? 8 : at % 4 == 0 ? 4 : 2;
}

template <typename TA, typename TW, typename Tile>
static bool simt_launch(const void *A, const void *W, float *out, int n, int m, int k, int groups,
                        bool early, cudaStream_t st)
{
    static unsigned long long done = 0, done_parts = 0;
    // (no more than four blocks an SM: bfloat16 weights would let seven in, and the SMs then end apart: 8 rows, float
    // by bfloat16, 6144 x 2560, 18.2 us against 14.3)
    constexpr int smem = Tile::template smem<TA, TW>() > (56 << 10) ? Tile::template smem<TA, TW>() : 56 << 10;
    long long row_tiles = ((long long)n + Tile::ROWS - 1) / Tile::ROWS;
    long long tiles = row_tiles * (((long long)m + Tile::FEATS - 1) / Tile::FEATS);
    if (tiles > 0x7fffffffll)
        return false;
    dim3 grid((unsigned)tiles, 1, groups);
    if (groups > 1) {
        if (!allow_dynamic_smem(gemm_simt_kernel<TA, TW, Tile, true>, smem, done_parts))
            return false;
        launch(gemm_simt_kernel<TA, TW, Tile, true>, grid, Tile::THREADS, smem, st, (const TA *)A, (const TW *)W, out,
               n, m, k, (int)row_tiles, copy_bytes<TA>(A, k), copy_bytes<TW>(W, k), early);
    } else {
        if (!allow_dynamic_smem(gemm_simt_kernel<TA, TW, Tile, false>, smem, done))
            return false;
        launch(gemm_simt_kernel<TA, TW, Tile, false>, grid, Tile::THREADS, smem, st, (const TA *)A, (const TW *)W, out,
               n, m, k, (int)row_tiles, copy_bytes<TA>(A, k), copy_bytes<TW>(W, k), early);
    }
    return true;
}

template <typename TA, typename TW>
static bool simt_pick(const void *A, const void *W, float *out, int n, int m, int k, int groups, bool early,
                      cudaStream_t st)
{
    int rows = simt_rows(n, m, k);
    if (rows == Rows8::ROWS)
        return simt_launch<TA, TW, Rows8>(A, W, out, n, m, k, groups, early, st);
    if (rows == Rows16::ROWS)
        return simt_launch<TA, TW, Rows16>(A, W, out, n, m, k, groups, early, st);
    if (rows == Rows32::ROWS)
        return simt_launch<TA, TW, Rows32>(A, W, out, n, m, k, groups, early, st);
    return simt_launch<TA, TW, Rows64>(A, W, out, n, m, k, groups, early, st);
}

}  // namespace jb

using namespace jb;

// Floats of scratch that jb_gemm_simt wants for this shape (0: none).
extern "C" long long jb_gemm_simt_scratch(int n, int m, int k)
{
    if (n <= 0 || m <= 0 || k <= 0 || simt_groups(n, m, k) <= 1)
        return 0;
    return (long long)simt_segments(k) * n * m;
}

// scratch: jb_gemm_simt_scratch(n, m, k) floats (may be null when that is 0).  early: W was complete before
// any kernel that may still run (a model's weights), so it may be read before the kernel ahead has ended.
extern "C" int jb_gemm_simt(const void *A, int a_dt, const void *W, int w_dt, float *out, int n,
                            int m, int k, float *scratch, int early, cudaStream_t st)
{
    if (n <= 0 || m <= 0)
        return JB_OK;
    if (k <= 0 || ((long long)n + 63) / 64 > 65535)
        return JB_EINVAL;
    int groups = simt_groups(n, m, k), segments = simt_segments(k);
    if (groups > 1 && scratch == nullptr)
        return JB_EINVAL;
    float *to = groups > 1 ? scratch : out;
    bool ok;
    if (a_dt == JB_F32 && w_dt == JB_F32)
        ok = simt_pick<float, float>(A, W, to, n, m, k, groups, early != 0, st);
    else if (a_dt == JB_F32 && w_dt == JB_BF16)
        ok = simt_pick<float, bf16>(A, W, to, n, m, k, groups, early != 0, st);
    else if (a_dt == JB_BF16 && w_dt == JB_F32)
        ok = simt_pick<bf16, float>(A, W, to, n, m, k, groups, early != 0, st);
    else if (a_dt == JB_BF16 && w_dt == JB_BF16)
        ok = simt_pick<bf16, bf16>(A, W, to, n, m, k, groups, early != 0, st);
    else
        return JB_EINVAL;
    if (!ok)
        return JB_ELAUNCH;
    if (groups > 1) {
        if (cudaGetLastError() != cudaSuccess)
            return JB_ELAUNCH;
        long long count = (long long)n * m;
        if (count % 4 == 0 && (uintptr_t)out % 16 == 0 && (uintptr_t)scratch % 16 == 0)
            launch(gemm_simt_join_kernel<4>, (unsigned)((count / 4 + 255) / 256), 256, 0, st, (const float *)scratch,
                   out, count, segments);
        else
            launch(gemm_simt_join_kernel<1>, (unsigned)((count + 255) / 256), 256, 0, st, (const float *)scratch, out,
                   count, segments);
    }
    return launch_status();
}
