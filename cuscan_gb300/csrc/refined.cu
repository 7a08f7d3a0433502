// bf16 tensor-core screening of the distance sweeps, with exact f32 re-evaluation.
//
// The kNN sweep and every Borůvka round first run a screening pass on the 5th-generation tensor
// cores: the points are rounded to bf16 once, in a pre-swizzled tiled copy, and one persistent
// CTA per SM computes 128 x 256 tiles of dot products with tcgen05.mma (fp32 accumulators in
// TMEM, operands streamed into shared memory by bulk async copies). From each dot product the
// epilogue forms a proven LOWER bound of the reference's f32 squared distance,
//
//     L_ij = (1 - C_B)(p_i + p_j) - 2 dot_ij - C_A m_i m_j  <=  d2_ij (sequential-FMA f32),
//
// where p = ||x||^2 (f32), m >= ||x||, C_A bounds the bf16 rounding of both operands and the
// tensor-core accumulation, and C_B the f32 rounding of norms, of the reference sum and of the
// epilogue arithmetic (see error_coefficients below). Per query row the M smallest bounds (for
// Borůvka: max(L, core_i, core_j) over other components) stay in registers. A second kernel
// re-evaluates those M candidates with the exact f32 direct-difference arithmetic and checks the
// result against the M-th bound: every pair outside the list has a lower bound >= that bound, so
// when it is larger than the selected exact value no outside pair can change the result. Rows
// that fail the check are re-run by the exact f32 kernels. The outputs are therefore bit
// identical to the plain path.
//
// Operand formats: bf16 of x; fp16 of x * 2^k (a power-of-two scale that brings the largest
// |x| into [2^14, 2^15)); and split bf16, x = hi + lo with hi = bf16(x) and lo = bf16(x - hi),
// whose dot product hi.hi' + hi.lo' + lo.hi' (three K blocks per 64 features) misses x.y by
// about 3 * 2^-16 |x||y| instead of 2^-7. A bf16-refined fit whose plain bf16 screen leaves too
// many kNN rows inconclusive screens again with split bf16 (d <= 64: three MMAs per block) or
// with scaled fp16 operands (wider rows: one MMA per block), and keeps that format for its
// Borůvka rounds. Rows of up to 256 features take the screens.
#include <cuda_bf16.h>

#include <cmath>
#include <type_traits>

#include "cells.cuh"
#include "common.cuh"
#include "forest.cuh"
#include "workspace.cuh"

namespace cuscan {

namespace {

constexpr int BM = 128;            // query rows per block = TMEM lanes
constexpr int BN = 256;            // reference rows per tile = MMA N
constexpr int EPI_WARPS = 8;            // two per TMEM lane quadrant
constexpr int HALF = 128;                // columns of a tile per epilogue warp
constexpr int THREADS = (2 + EPI_WARPS) * 32;
constexpr uint32_t KBLOCK_A = BM * 128;   // bytes of one 64-element K block of A (16 KiB)
constexpr uint32_t KBLOCK_B = BN * 128;   // bytes of one 64-element K block of B (32 KiB)
constexpr uint64_t WAIT_NS = 2000000000ull;  // bounded mbarrier waits: 2 s of wall time
constexpr uint32_t WAIT_POLLS = 1u << 22;      // poll bound of the abort-path drains
constexpr int VSTRIDE = 36;               // floats per lane in the hit staging area
constexpr int PB_STRIDE = 4 * HALF;       // kNN modes, per epilogue warp: [2][HALF] pb, [2][HALF] m
constexpr int BORUVKA_CAP = 32;           // Borůvka candidate slots per row half

struct Params {
    const uint8_t *xt;        // 16-bit tiles, pre-swizzled (see prep_rows_kernel)
    int nbk;                  // K blocks per tile row of the copy: kblocks, or 2 kblocks (split)
    int split;                // split bf16: blocks [0, kblocks) hold hi, [kblocks, 2 kblocks) lo
    // kNN sweeps: [0] tiles issued by all CTAs so far (see knn_tile), [1] query blocks taken
    unsigned long long *cursor;
    const float *pnorm;       // [n_pad] f32 squared norms (+inf on padding rows)
    const float *mnorm;       // [n_pad] norms rounded up (0 on padding rows)
    // column terms of this launch (screen_columns_kernel): (1 - C_B) p, cores in screen units
    // (Borůvka; 0 past n) and (min, min) of both over every 32-column chunk
    const float *colp;
    const float *colc;
    const float4 *cmin;       // [n_pad / 64]: two chunks per entry
    const float *core;        // [n] core distances (Borůvka)
    const int32_t *label;     // [n] component labels (Borůvka)
    const float *tile_mmax;   // [n_tiles] max m over each 256-row tile
    const int32_t *chunk_lo;  // [ceil(n/32)] label range of 32-row chunks (Borůvka)
    const int32_t *chunk_hi;
    const int32_t *tile_lo;   // [n_tiles] label range of 256-row tiles (Borůvka)
    const int32_t *tile_hi;
    int64_t n, n_tiles, n_qblocks, n_chunks;
    int kblocks, stages, stage_blocks;  // stage_blocks: K blocks per ring stage (divides nbk)
    // one-sided Borůvka: parts of every query block's tile order (screen_parts), each a work item of
    // its own (item qi = block qi / splits, part qi % splits; with several parts appends take their
    // slots with atomics and the row bounds are min-reduced)
    int splits;
    float c_a, one_minus_cb;
    int32_t *cand_ids;        // [n][M]
    float *cand_lb;           // [n][M]
    int *error;               // [0]: error flag; bytes 8..15: (qb, tile) pairs the MMA ran (u64)
    float *debug_tile;        // when set: the raw 128 x 256 accumulator of query block 0 x tile 0
    float *debug_chunk;       // with debug_tile: [128][8] the phase-1 maxima of its 32-column chunks
    float c_b;                // norm coefficient of the bound (upper bounds use it)
    uint32_t *cbound;         // Borůvka: per-component upper bound of the cheapest edge (f32 bits)
    int32_t *rowcnt;          // Borůvka: candidates appended per row half ([n][2])
    int cap;                  // Borůvka: candidate slots per row half
    uint32_t idesc;           // MMA instruction descriptor (bf16 or fp16 operands)
    float s2, inv_s2;         // operand scale squared (a power of two) and its inverse: the
                              // screen works in scaled units, inputs and outputs are raw
    float abs_c;              // absolute error term of the bound (fp16 subnormal rounding)
    // query rows (the A operand): the reference set itself, or a gathered subset
    const uint8_t *xq;        // 16-bit tiles of the query rows, same layout as xt
    const float *pq, *mq;     // their squared norms and rounded-up norms
    int64_t nq;               // query rows
    const int32_t *qpos;      // position of each query row in the reference order (null: same)
    const int32_t *qchunk_lo; // Borůvka: label range of 32-row chunks of gathered query rows
    const int32_t *qchunk_hi;
    const float *qthr;        // threshold mode: per-query upper bound of the k-th distance (raw)
    // symmetric Borůvka: per-row upper bounds of the cheapest cross edge (raw f32 bits) and the
    // per-row buffers that other query blocks append column-side pairs to
    uint32_t *urow;
    int32_t *colcnt;
    int32_t *colbuf;
    int capc;
    // one-sided Borůvka: per query row and column half, a lower bound of every cross-component
    // pair weight the row has (raw f32, rounded down)
    float *rowlb;
    // LIST: the tiles each query block visits ([n_qblocks][n_tiles], in order) and their number
    const uint16_t *vis;
    const int32_t *vis_count;
};

// Screen modes: kNN lists, Borůvka thresholds with shared component bounds, kNN thresholds.
constexpr int MODE_KNN_LIST = 0;
constexpr int MODE_BORUVKA = 1;
constexpr int MODE_KNN_THRESHOLD = 2;
// Borůvka over each unordered pair once: a query block visits its own tile (both halves see
// every pair inside it) and the tiles after it, testing each pair for its row and, through
// the column-side buffers, for its column.
constexpr int MODE_BORUVKA_SYM = 3;
constexpr int BORUVKA_COL_CAP = 64;  // column-side candidate slots per row
constexpr double SYM_UNBOUNDED_MAX = 0.25;  // largest share of unbounded rows for the symmetric screen
constexpr int64_t SYM_MIN_ROWS = 131072;     // smallest point set for the symmetric screen
constexpr double SYM_ACTIVE_MIN = 0.9;  // smallest share of screened rows for the symmetric screen
constexpr int KNN_CAP = 512;  // threshold-mode candidate slots per row half
constexpr int KNN_LIST = 22;  // kNN list entries per row half
static_assert(KNN_LIST <= BORUVKA_CAP, "the candidate buffer of the rounds holds the lists");
constexpr int RESCREEN_MIN_ROWS = 256;  // fewer inconclusive kNN rows go straight to exact f32
// A bf16-refined fit whose first kNN screen leaves more than this share of rows inconclusive
// screens again with tighter operands (split bf16, or scaled fp16 for rows too wide to split).
constexpr double TIGHTEN_TRIGGER = 0.15;
// Share of rows that choose_operands_by_cells expects to be inconclusive from which the first
// screen already uses the tightened operands.
constexpr double TIGHT_START = 0.25;
// kNN screens over lists of tiles: smallest fit, and the share of row pairs in cells too far apart to
// hold neighbours from which the lists are made (mixtures of separated clusters have 0.93 to 0.97,
// unit vectors about 0). At 100,000 x 64, 50 clusters and noise, the blocks visit a fifth of the
// tiles and the screen takes 1.60 ms instead of 2.46 ms (lists and balls 0.09 ms; the noise
// blocks visit all); 50,000 x 128: 0.41 instead of 0.65 ms. At 9,001 x 32, where half of the tiles
// stay, the two launches cost what the screen gains.
constexpr int64_t LIST_MIN_ROWS = 16384;
constexpr float LIST_MIN_APART = 0.6f;
// Status words of a screen: [0] error flag, [2..3] tile pairs (u64), [4] inconclusive rows listed by
// the re-rank, [5] spare.
constexpr int SCREEN_STATUS_WORDS = 8;
constexpr int STATUS_FALLBACKS = 4;
// Operand formats of the 16-bit copy.
constexpr int FMT_BF16 = 0;
constexpr int FMT_FP16 = 1;
constexpr int FMT_SPLIT = 2;

// ---- PTX wrappers ----
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
// Bounded wait: returns false (and raises the CTA abort flag and the error word) when the
// barrier does not flip within WAIT_NS nanoseconds, or as soon as another role has aborted.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, volatile int *abort,
                                          int *error) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = global_ns();
    for (uint32_t it = 1;; ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 255u) == 0u) {
            if (*abort) return false;
            if (global_ns() - t0 > WAIT_NS) break;
        }
    }
    *abort = 1;
    atomicExch(error, 1);
    return false;
}
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes,
                                         uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
        ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
// Shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t desc_sw128(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;            // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(1024 >> 4) << 32;  // stride byte offset
    d |= (uint64_t)1 << 46;            // descriptor version for tcgen05
    d |= (uint64_t)2 << 61;            // SWIZZLE_128B
    return d;
}
// Instruction descriptors of kind::f16: D f32, A and B both bf16 (format 1 in bits 7-9 and
// 10-12) or both fp16 (format 0), both K-major, M=128, N=256.
constexpr uint32_t IDESC_F16 = (1u << 4) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
constexpr uint32_t IDESC_BF16 = IDESC_F16 | (1u << 7) | (1u << 10);

__device__ __forceinline__ void mma_16bit(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc,
                                          uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}
__device__ __forceinline__ void mma_commit(uint64_t *bar) {
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
            smem_u32(bar))
        : "memory");
}
// Issue a 32-column TMEM load (no wait): the registers are valid only after tmem_ld_wait.
__device__ __forceinline__ void tmem_ld32_issue(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
        "%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
          "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
          "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
          "=r"(r[31])
        : "r"(taddr));
}
// Issue a 32-column TMEM load that also returns the largest of the 32 values (tcgen05.ld.red,
// sm_103a): the reduction rides on the load, so the chunk maxima of the screens cost no ALU
// work. mx and r are valid only after tmem_ld_wait_max. The maximum is exact (no rounding), the
// same value as a max.f32 tree over r.
__device__ __forceinline__ void tmem_ld32_max_issue(uint32_t taddr, uint32_t (&r)[32], float &mx) {
    asm volatile(
        "tcgen05.ld.red.sync.aligned.32x32b.x32.max.f32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,"
        "%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, %32, "
        "[%33];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
          "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
          "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
          "=r"(r[31]), "=f"(mx)
        : "r"(taddr));
}
// Wait for every issued TMEM load; the register operands tie r to the wait so the compiler
// cannot read them earlier.
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&r)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    asm volatile(""
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]),
                   "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]),
                   "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]),
                   "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]),
                   "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]),
                   "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31]));
}

// Byte offset of element (row r, column f < d_eff) in the tiled 16-bit copy: 256-row tiles, each
// split into 64-column K blocks of 256 rows x 128 bytes whose 16-byte chunks are XOR-swizzled
// by the row (the SWIZZLE_128B K-major layout), so one bulk copy lands a block ready for the
// MMA. d_eff is d_pad, or 2 d_pad for split copies (the lo parts in columns d_pad + f).
__host__ __device__ __forceinline__ uint64_t tiled_offset(int64_t r, int f, int d_eff) {
    const int64_t t = r >> 8;
    const int rr = (int)(r & 255);
    const int kb = f >> 6, c = f & 63;
    const int chunk = (c >> 3) ^ (rr & 7);
    return (uint64_t)t * (uint64_t)(BN * d_eff * 2) + (uint64_t)kb * KBLOCK_B +
           (uint64_t)rr * 128 + (uint64_t)chunk * 16 + (uint64_t)(c & 7) * 2;
}

// Order-preserving map of f32 values to u32 (for integer warp reductions) and back.
__device__ __forceinline__ uint32_t f2ord(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ord2f(uint32_t o) {
    return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}
// Everything a screen needs of a set of rows, one block per 256-row tile: the 16-bit tiled copy of
// the (scaled) rows (bf16, fp16 of x * scale, scale a power of two, or split bf16: hi in columns
// [0, d_pad), lo = bf16(x - hi) in [d_pad, 2 d_pad)), their squared norms and rounded-up norms, the
// tile's largest norm and, with labels, the label ranges of its 32-row chunks and of the tile.
// Row r is row rowmap[r] of x (r itself when rowmap is null); rows >= n are zero with norm +inf.
// Eight lanes share a row, eight features each per step, so the rows are read once with
// consecutive addresses; separate kernels for the copy, the norms (one thread per row), the
// tile statistics and the label ranges took 22 us per round of a 9,001 x 32 fit.
constexpr int PREP_THREADS = 1024;
template <int FMT>
__global__ void __launch_bounds__(PREP_THREADS)
    prep_rows_kernel(const float *__restrict__ x, int64_t n, int d, int d_pad, float scale,
                     const int32_t *__restrict__ rowmap, int vec4, uint8_t *__restrict__ xt,
                     float *__restrict__ pnorm, float *__restrict__ mnorm,
                     float *__restrict__ tile_mmax, const int32_t *__restrict__ label,
                     int32_t *__restrict__ chunk_lo, int32_t *__restrict__ chunk_hi,
                     int32_t *__restrict__ tile_lo, int32_t *__restrict__ tile_hi) {
    __shared__ float warp_max[PREP_THREADS / 32];
    __shared__ int32_t range_lo[BN / 32], range_hi[BN / 32];
    const int tid = threadIdx.x, lane = tid & 31, sub = tid & 7;
    const int64_t row0 = (int64_t)blockIdx.x * BN;
    const int d_eff = FMT == FMT_SPLIT ? 2 * d_pad : d_pad;
    float mmax = 0.0f;
#pragma unroll
    for (int rr = 0; rr < BN; rr += PREP_THREADS / 8) {
        const int64_t r = row0 + rr + (tid >> 3);
        const bool valid = r < n;
        const float *src = x + (valid ? (rowmap ? (int64_t)rowmap[r] : r) : 0) * d;
        float acc = 0.0f;
        for (int g = sub; g < d_pad / 8; g += 8) {
            const int f0 = g * 8;
            float v[8];
            if (vec4 && valid && f0 + 8 <= d) {
                const float4 a = *reinterpret_cast<const float4 *>(src + f0);
                const float4 b = *reinterpret_cast<const float4 *>(src + f0 + 4);
                v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
                v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
            } else {
#pragma unroll
                for (int q = 0; q < 8; ++q) v[q] = valid && f0 + q < d ? src[f0 + q] : 0.0f;
            }
            __align__(16) uint16_t h[8];
            __align__(16) uint16_t l[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const float sv = v[q] * scale;
                acc = __fmaf_rn(sv, sv, acc);
                if constexpr (FMT == FMT_FP16) {
                    h[q] = __half_as_ushort(__float2half_rn(sv));
                } else {
                    const __nv_bfloat16 hi = __float2bfloat16_rn(v[q]);
                    h[q] = __bfloat16_as_ushort(hi);
                    // v - hi is exact in f32 (hi is within a factor of two of v)
                    if constexpr (FMT == FMT_SPLIT)
                        l[q] = __bfloat16_as_ushort(
                            __float2bfloat16_rn(v[q] - __bfloat162float(hi)));
                }
            }
            *reinterpret_cast<uint4 *>(xt + tiled_offset(r, f0, d_eff)) =
                *reinterpret_cast<const uint4 *>(h);
            if constexpr (FMT == FMT_SPLIT)
                *reinterpret_cast<uint4 *>(xt + tiled_offset(r, d_pad + f0, d_eff)) =
                    *reinterpret_cast<const uint4 *>(l);
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        // rounded-up norm, widened by 2^-20 so it bounds the true norm despite the f32 sum
        const float m = valid ? __fmul_ru(__fsqrt_ru(acc), 1.0f + 0x1p-20f) : 0.0f;
        if (sub == 0) {
            pnorm[r] = valid ? acc : CUSCAN_INF;
            mnorm[r] = m;
        }
        mmax = fmaxf(mmax, m);
    }
    if (label && tid < BN) {
        // a warp per 32-row chunk; chunks past the end have the empty range
        const int64_t r = row0 + tid;
        const int32_t l = r < n ? label[rowmap ? (int64_t)rowmap[r] : r] : 0;
        const int32_t lo = __reduce_min_sync(0xffffffffu, r < n ? l : INT32_MAX);
        const int32_t hi = __reduce_max_sync(0xffffffffu, r < n ? l : INT32_MIN);
        if (lane == 0) {
            range_lo[tid >> 5] = lo;
            range_hi[tid >> 5] = hi;
            if (r < n) {
                chunk_lo[r >> 5] = lo;
                chunk_hi[r >> 5] = hi;
            }
        }
    }
    if (tile_mmax) {
        mmax = ord2f(__reduce_max_sync(0xffffffffu, f2ord(mmax)));
        if (lane == 0) warp_max[tid >> 5] = mmax;
        __syncthreads();
        if (tid == 0) {
            float mx = 0.0f;
            for (int w = 0; w < PREP_THREADS / 32; ++w) mx = fmaxf(mx, warp_max[w]);
            tile_mmax[blockIdx.x] = mx;
            if (label) {
                int32_t lo = INT32_MAX, hi = INT32_MIN;
                for (int c = 0; c < BN / 32; ++c) {
                    lo = min(lo, range_lo[c]);
                    hi = max(hi, range_hi[c]);
                }
                tile_lo[blockIdx.x] = lo;
                tile_hi[blockIdx.x] = hi;
            }
        }
    }
}

// Largest |x| over all coordinates (non-negative floats order like their bit patterns).
__global__ void absmax_kernel(const float *__restrict__ x, int64_t count,
                              unsigned int *__restrict__ out) {
    float m = 0.0f;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count;
         i += (int64_t)gridDim.x * blockDim.x)
        m = fmaxf(m, fabsf(x[i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, __float_as_uint(m));
}

// Before a screen launch: its column terms, computed once instead of by every epilogue warp that
// reads the columns: colp = (1 - C_B) p (+inf on padding rows), colc = core * s2 (Borůvka; 0
// past n), and for every 32-column chunk (min colp, min colc) (0 for colc in the kNN modes); and
// its cleared counters: the status words, the cursor, the append counts of the query rows and, for
// split blocks, their bounds (+inf). One thread per padded row; n_pad is a multiple of the
// 256-thread block.
__global__ void screen_columns_kernel(const float *__restrict__ pnorm,
                                      const float *__restrict__ core, int64_t n,
                                      float one_minus_cb, float s2, float *__restrict__ colp,
                                      float *__restrict__ colc, float2 *__restrict__ cmin,
                                      int *__restrict__ status,
                                      unsigned long long *__restrict__ cursor,
                                      int2 *__restrict__ rowcnt, float2 *__restrict__ rowlb,
                                      int64_t nq) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j < SCREEN_STATUS_WORDS) status[j] = 0;
    if (j < 2) cursor[j] = 0ull;
    if (j < nq) {
        if (rowcnt) rowcnt[j] = make_int2(0, 0);
        if (rowlb) rowlb[j] = make_float2(CUSCAN_INF, CUSCAN_INF);
    }
    const float p = pnorm[j] * one_minus_cb;
    colp[j] = p;
    float c = 0.0f;
    if (core) {
        c = j < n ? core[j] * s2 : 0.0f;
        colc[j] = c;
    }
    float pm = p, cm = c;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        pm = fminf(pm, __shfl_xor_sync(0xffffffffu, pm, o));
        cm = fminf(cm, __shfl_xor_sync(0xffffffffu, cm, o));
    }
    if ((threadIdx.x & 31) == 0) cmin[j >> 5] = make_float2(pm, cm);
}

// Order in which query block qb visits the reference tiles. Every order starts with a window of
// WARM tiles around the block's own tile: in cell-sorted data these hold the block's nearest
// neighbours, so the per-row thresholds tighten at once.
//
// Borůvka rounds (tile_order) go on cyclically from the window. Their blocks skip different
// tiles, and the tiles they run stay in L2 anyway (one to two GB of DRAM reads per round at
// 500,000 points), so the cheapest order wins there.
//
// The kNN sweeps (knn_tile) run every tile for every block. After the window a block enters one
// cyclic order of the other tiles that all CTAs share, at the rotation `rot` the producer takes
// from the tile cursor when the block starts: the average position of the CTAs. Blocks started
// at different times then stream the same tiles and share them in L2. Without the rotation the
// CTAs drift apart over the waves of the persistent loop and the sweep reads the copy from
// DRAM about a thousand times over.
constexpr int64_t WARM = 4;

__device__ __forceinline__ float warp_max_f(float v) {
    return ord2f(__reduce_max_sync(0xffffffffu, f2ord(v)));
}
__device__ __forceinline__ float warp_min_f(float v) {
    return ord2f(__reduce_min_sync(0xffffffffu, f2ord(v)));
}

__device__ __forceinline__ int64_t window_start(const Params &P, int64_t qb) {
    const int64_t w = P.n_tiles < WARM ? P.n_tiles : WARM;
    const int64_t first = P.qpos ? (int64_t)P.qpos[qb * BM] : qb * BM;
    int64_t a = first / BN - w / 2;
    if (a < 0) a = 0;
    if (a > P.n_tiles - w) a = P.n_tiles - w;
    return a;
}
__device__ __forceinline__ int64_t tile_order(const Params &P, int64_t a, int64_t i) {
    const int64_t t = a + i;
    return t < P.n_tiles ? t : t - P.n_tiles;
}
// n tiles, window [a, a + w), rotation r < n - w (r = 0 when n <= WARM).
__device__ __forceinline__ int32_t knn_tile(int32_t n, int32_t a, int32_t r, int32_t i) {
    const int32_t w = n < (int32_t)WARM ? n : (int32_t)WARM;
    if (i < w) return a + i;
    int32_t j = i - w + r;
    if (j >= n - w) j -= n - w;
    return j < a ? j : j + w;
}

// Tiles query block qb visits and the i-th of them. The symmetric Borůvka mode visits the
// block's own tile and then every later tile in order; the other modes visit every tile
// (tile_order).
template <bool SYM>
__device__ __forceinline__ int64_t vis_count(const Params &P, int64_t qb) {
    return SYM ? P.n_tiles - (qb >> 1) : P.n_tiles;
}
template <bool SYM>
__device__ __forceinline__ int64_t vis_tile(const Params &P, int64_t qb, int64_t wa, int64_t i) {
    return SYM ? (qb >> 1) + i : tile_order(P, wa, i);
}

// Label range of query block qb (4 chunks of 32 rows).
__device__ __forceinline__ void qblock_range(const Params &P, int64_t qb, int32_t &lo,
                                             int32_t &hi) {
    // gathered query rows keep the order of their components, so most of their blocks have one
    // label too and skip their own component's tiles; without label ranges they skip none
    if (P.qpos && !P.qchunk_lo) {
        lo = INT32_MIN;
        hi = INT32_MAX;
        return;
    }
    const int32_t *clo = P.qpos ? P.qchunk_lo : P.chunk_lo;
    const int32_t *chi = P.qpos ? P.qchunk_hi : P.chunk_hi;
    const int64_t chunks = P.qpos ? (P.nq + 31) / 32 : P.n_chunks;
    lo = INT32_MAX;
    hi = INT32_MIN;
    for (int64_t c = qb * 4; c < qb * 4 + 4 && c < chunks; ++c) {
        lo = min(lo, clo[c]);
        hi = max(hi, chi[c]);
    }
}

template <bool BORUVKA>
__device__ __forceinline__ bool tile_skipped(const Params &P, int64_t t, int32_t qlo, int32_t qhi) {
    if (!BORUVKA) return false;
    return qlo == qhi && P.tile_lo[t] == qlo && P.tile_hi[t] == qlo;
}

template <int M>
__device__ __forceinline__ void list_insert(float (&L)[M], int (&J)[M], float x, int j) {
#pragma unroll
    for (int s = M - 1; s >= 0; --s) {
        const bool here = x < L[s];
        const bool prev = (s > 0) ? (x < L[s > 0 ? s - 1 : 0]) : false;
        if (here) {
            if (prev) {
                L[s] = L[s > 0 ? s - 1 : 0];
                J[s] = J[s > 0 ? s - 1 : 0];
            } else {
                L[s] = x;
                J[s] = j;
            }
        }
    }
}

// LIST (kNN lists): the blocks visit the tiles of their lists (visit_lists_kernel), not every tile.
template <int M, int MODE, bool LIST>
__global__ void __launch_bounds__(THREADS, 1) screen_kernel(const Params P) {
    constexpr bool BORUVKA = MODE == MODE_BORUVKA || MODE == MODE_BORUVKA_SYM;
    constexpr bool SYM = MODE == MODE_BORUVKA_SYM;
    constexpr bool THRESH = MODE == MODE_KNN_THRESHOLD;
    constexpr bool APPEND = BORUVKA || THRESH;  // threshold modes append to per-row buffers
    constexpr bool ROT = !BORUVKA && !LIST;     // kNN sweeps: rotated shared tile order
    constexpr bool CLAIM = !BORUVKA;            // and blocks from a global counter
    // kNN sweeps: the column terms of each tile are copied into the warp's shared slots, where
    // the list insertions read them (Borůvka screens read them from global memory)
    constexpr bool STAGE = !BORUVKA;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t a_bytes = (uint32_t)P.nbk * KBLOCK_A;
    const uint32_t b_bytes = (uint32_t)P.nbk * KBLOCK_B;  // one tile of the copy
    uint8_t *sA = smem;
    // Ring of reference tiles. A stage holds a whole tile of up to two 64-column K blocks, one
    // block of a wider one, so that rows of up to 256 features (four blocks of A, 64 KB) still
    // leave three stages. One wait and commit per block for every width measured 118.2 ms against
    // 102.7 ms at 500,000 x 128: the MMAs of a tile start when its TMEM buffer frees, and the
    // waits between them add to that chain.
    uint8_t *sB = smem + a_bytes;
    const uint32_t stage_bytes = (uint32_t)P.stage_blocks * KBLOCK_B;
    float *pbuf = (float *)(sB + (size_t)P.stages * stage_bytes);  // [EPI_WARPS][PB_STRIDE]
    float *vstage = pbuf + EPI_WARPS * PB_STRIDE;                    // [EPI_WARPS][32][VSTRIDE]
    uint64_t *bars = (uint64_t *)(vstage + EPI_WARPS * 32 * VSTRIDE);
    uint64_t *full = bars;
    uint64_t *empty = bars + P.stages;
    uint64_t *a_full = bars + 2 * P.stages;
    uint64_t *a_empty = a_full + 1;
    uint64_t *t_full = a_full + 2;   // [2]
    uint64_t *t_empty = a_full + 4;  // [2]
    uint64_t *done = a_full + 6;     // MMA drain on the abort path
    // kNN sweeps: ring of the blocks the producer took and their rotations
    uint64_t *rot_full = a_full + 7;    // [4] the producer published a block
    uint64_t *rot_empty = a_full + 11;  // [4] the MMA warp and every epilogue warp have read it
    uint32_t *tmem_slot = (uint32_t *)(a_full + 15);
    volatile int *abort = (volatile int *)(tmem_slot + 1);
    int32_t *rot_val = (int32_t *)(tmem_slot + 2);  // [4] rotations
    int64_t *rot_blk = (int64_t *)(tmem_slot + 6);  // [4] query blocks (n_qblocks: none left)

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < P.stages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(a_full, 1);
        mbar_init(a_empty, 1);
        mbar_init(done, 1);
        for (int b = 0; b < 2; ++b) {
            mbar_init(&t_full[b], 1);
            mbar_init(&t_empty[b], EPI_WARPS);
        }
        for (int r = 0; r < 4; ++r) {
            mbar_init(&rot_full[r], 1);
            mbar_init(&rot_empty[r], EPI_WARPS + 1);
        }
        *abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                         smem_u32(tmem_slot))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ---------------- producer: bulk copies of A (per query block) and B tiles ----------
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0, a_phase = 0;
            // parity of the last fill of each stage (bit 1 set = a fill was issued)
            uint32_t issued[4] = {0, 0, 0, 0};
            uint32_t a_issued = 0;
            for (uint32_t li = 0; !*abort; ++li) {  // li: this CTA's query step
                int64_t qi = blockIdx.x + (int64_t)li * gridDim.x;
                int32_t rot = 0;
                if (CLAIM) {
                    // kNN sweeps: blocks come from a global counter, so that CTAs that run faster
                    // take more of them. The block and its rotation of the shared order (the
                    // CTAs' average position: tiles issued so far over the grid) go to the MMA
                    // and epilogue warps through the ring; n_qblocks there ends their loops.
                    // The last blocks come first: rows far from every cell are ordered last, and
                    // their blocks, whose thresholds tighten slowly, would make a long tail
                    // (6.8 against 4.3 ms for the two sweeps of an anisotropic 100,000 x 64 fit).
                    qi = (int64_t)atomicAdd(P.cursor + 1, 1ull);
                    qi = qi < P.n_qblocks ? P.n_qblocks - 1 - qi : P.n_qblocks;
                    if (ROT && P.n_tiles > WARM && qi < P.n_qblocks) {
                        const unsigned long long all = *(volatile unsigned long long *)P.cursor;
                        rot = (int32_t)((all / gridDim.x) % (unsigned long long)(P.n_tiles - WARM));
                    }
                    const uint32_t rs = li & 3;
                    if (!mbar_wait(&rot_empty[rs], ((li >> 2) & 1) ^ 1, abort, P.error)) break;
                    rot_blk[rs] = qi;
                    rot_val[rs] = rot;
                    mbar_arrive(&rot_full[rs]);
                }
                if (qi >= P.n_qblocks * P.splits) break;
                const int64_t qb = qi / P.splits;
                const int64_t part = qi % P.splits;
                if (!mbar_wait(a_empty, a_phase ^ 1, abort, P.error)) break;
                a_issued = 2u | a_phase;
                a_phase ^= 1;
                mbar_expect_tx(a_full, a_bytes);
                const uint8_t *asrc = P.xq + (uint64_t)(qb >> 1) * (uint64_t)b_bytes +
                                      (uint64_t)(qb & 1) * KBLOCK_A;
                for (int kb = 0; kb < P.nbk; ++kb)
                    bulk_g2s(sA + kb * KBLOCK_A, asrc + (uint64_t)kb * KBLOCK_B, KBLOCK_A, a_full);
                int32_t qlo = 0, qhi = 0;
                if (BORUVKA) qblock_range(P, qb, qlo, qhi);
                const int64_t wa = LIST ? qb * P.n_tiles : window_start(P, qb);
                const int64_t nvis = LIST ? P.vis_count[qb] : vis_count<SYM>(P, qb);
                const int64_t i_hi = (part + 1) * nvis / P.splits;
                for (int64_t i = part * nvis / P.splits; i < i_hi; ++i) {
                    const int64_t t = LIST ? (int64_t)P.vis[wa + i]
                                      : ROT ? (int64_t)knn_tile((int32_t)P.n_tiles, (int32_t)wa, rot, (int32_t)i)
                                          : vis_tile<SYM>(P, qb, wa, i);
                    if (tile_skipped<BORUVKA>(P, t, qlo, qhi)) continue;
                    const uint8_t *bsrc = P.xt + (uint64_t)t * (uint64_t)b_bytes;
                    bool ok = true;
                    for (int k0 = 0; k0 < P.nbk; k0 += P.stage_blocks) {
                        if (!mbar_wait(&empty[stage], phase ^ 1, abort, P.error)) {
                            ok = false;
                            break;
                        }
                        issued[stage] = 2u | phase;
                        mbar_expect_tx(&full[stage], stage_bytes);
                        uint8_t *bdst = sB + (size_t)stage * stage_bytes;
                        for (int kb = 0; kb < P.stage_blocks; ++kb)
                            bulk_g2s(bdst + kb * KBLOCK_B, bsrc + (uint64_t)(k0 + kb) * KBLOCK_B,
                                     KBLOCK_B, &full[stage]);
                        if (++stage == P.stages) {
                            stage = 0;
                            phase ^= 1;
                        }
                    }
                    if (!ok) break;
                    if (ROT) atomicAdd(P.cursor, 1ull);
                }
            }
            if (*abort) {
                // let every copy this thread issued land before the CTA exits
                for (int s2 = 0; s2 < P.stages; ++s2)
                    if (issued[s2]) {
                        for (uint32_t it = 0; it < WAIT_POLLS; ++it)
                            if (mbar_try_wait(&full[s2], issued[s2] & 1u)) break;
                    }
                if (a_issued)
                    for (uint32_t it = 0; it < WAIT_POLLS; ++it)
                        if (mbar_try_wait(a_full, a_issued & 1u)) break;
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer: one thread -------------------------------------------
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0, a_phase = 0;
            uint32_t tcount = 0, a_commits = 0;
            // Descriptors of the first K step of A and of ring stage 0; a K step is 32 bytes, a
            // block of A KBLOCK_A, so each further descriptor is one addition (in 16-byte units).
            const uint64_t a_desc = desc_sw128(smem_u32(sA)), b_desc = desc_sw128(smem_u32(sB));
            // One tile's MMAs for KB K blocks (SB of them per ring stage), fully unrolled: they are
            // issued when the tile's TMEM buffer frees, so every instruction between that and the
            // last MMA adds to the chain MMA -> epilogue -> MMA. Split copies: a hi block of B
            // meets the hi and the lo block of A, a lo block of B (j >= KB) the hi block.
            auto issue = [&](auto kb_c, auto sb_c, auto split_c, uint32_t b, uint32_t tp) -> bool {
                constexpr int KB = decltype(kb_c)::value, SB = decltype(sb_c)::value;
                constexpr bool SPLIT = decltype(split_c)::value;
                constexpr int NB = SPLIT ? 2 * KB : KB;
                const uint32_t d_tmem = tmem_base + b * BN;
#pragma unroll
                for (int k0 = 0; k0 < NB; k0 += SB) {
                    if (!mbar_wait(&full[stage], phase, abort, P.error)) return false;
                    if (k0 == 0 && !mbar_wait(&t_empty[b], tp ^ 1, abort, P.error)) return false;
                    fence_after();
                    const uint64_t bd = b_desc + (uint32_t)stage * (SB * KBLOCK_B >> 4);
#pragma unroll
                    for (int j = k0; j < k0 + SB; ++j) {
                        const int ja = j < KB ? j : j - KB;  // the hi block of A
#pragma unroll
                        for (int ks = 0; ks < 4; ++ks)
                            mma_16bit(d_tmem, a_desc + ((ja * KBLOCK_A + ks * 32) >> 4),
                                      bd + (((j - k0) * KBLOCK_B + ks * 32) >> 4), P.idesc,
                                      (j | ks) != 0);
                        if (SPLIT && j < KB) {
#pragma unroll
                            for (int ks = 0; ks < 4; ++ks)
                                mma_16bit(d_tmem, a_desc + (((KB + j) * KBLOCK_A + ks * 32) >> 4),
                                          bd + (((j - k0) * KBLOCK_B + ks * 32) >> 4), P.idesc,
                                          1u);
                        }
                    }
                    mma_commit(&empty[stage]);
                    if (++stage == P.stages) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
                mma_commit(&t_full[b]);
                return true;
            };
            auto blocks = [&](auto kb_c, auto sb_c, auto split_c) {
                for (uint32_t li = 0; !*abort; ++li) {
                    int64_t qi = blockIdx.x + (int64_t)li * gridDim.x;
                    if (CLAIM) {  // the block the producer took
                        const uint32_t rs = li & 3;
                        if (!mbar_wait(&rot_full[rs], (li >> 2) & 1, abort, P.error)) break;
                        qi = *(volatile int64_t *)&rot_blk[rs];
                        mbar_arrive(&rot_empty[rs]);
                    }
                    if (qi >= P.n_qblocks * P.splits) break;
                    const int64_t qb = qi / P.splits;
                    const int64_t part = qi % P.splits;
                    if (!mbar_wait(a_full, a_phase, abort, P.error)) break;
                    a_phase ^= 1;
                    fence_after();
                    int32_t qlo = 0, qhi = 0;
                    if (BORUVKA) qblock_range(P, qb, qlo, qhi);
                    const int64_t wa = LIST ? 0 : window_start(P, qb);
                    const int64_t nvis = LIST ? P.vis_count[qb] : vis_count<SYM>(P, qb);
                    const int64_t i_hi = (part + 1) * nvis / P.splits;
                    bool ok = true;
                    for (int64_t i = part * nvis / P.splits; i < i_hi; ++i) {
                        if (BORUVKA &&
                            tile_skipped<BORUVKA>(P, vis_tile<SYM>(P, qb, wa, i), qlo, qhi))
                            continue;
                        if (!issue(kb_c, sb_c, split_c, tcount & 1, (tcount >> 1) & 1)) {
                            ok = false;
                            break;
                        }
                        ++tcount;
                    }
                    mma_commit(a_empty);
                    ++a_commits;
                    if (!ok) break;
                }
            };
            using std::integral_constant;
            constexpr integral_constant<int, 1> c1{};
            constexpr integral_constant<int, 2> c2{};
            if (P.split)  // d <= 64
                blocks(c1, c2, std::true_type{});
            else if (P.kblocks == 1)
                blocks(c1, c1, std::false_type{});
            else if (P.kblocks == 2)
                blocks(c2, c2, std::false_type{});
            else if (P.kblocks == 3)
                blocks(integral_constant<int, 3>{}, c1, std::false_type{});
            else
                blocks(integral_constant<int, 4>{}, c1, std::false_type{});
            atomicAdd(reinterpret_cast<unsigned long long *>(P.error + 2),
                      (unsigned long long)tcount);
            // wait until every issued MMA has completed before TMEM can be released
            mma_commit(done);
            for (uint32_t it = 0; it < WAIT_POLLS; ++it)
                if (mbar_try_wait(done, 0)) break;
            if (a_commits)
                for (uint32_t it = 0; it < WAIT_POLLS; ++it)
                    if (mbar_try_wait(a_empty, (a_commits - 1) & 1u)) break;
        }
    } else {
        // ---------------- epilogue: two threads per query row ---------------------------------
        // Warps 2..9: warp w reads TMEM lane quadrant w % 4 (hardware rule) and handles one half
        // of every 256-column tile; the two threads of a row keep separate top-M lists.
        const int ew = warp - 2;              // 0..7
        const int quad = warp & 3;            // TMEM lane quadrant of this warp
        const int half = ew >> 2;             // column half of each tile
        const int row_local = quad * 32 + lane;
        float *my_v = vstage + (ew * 32 + lane) * VSTRIDE;
        float *my_pb = pbuf + ew * PB_STRIDE;
        uint32_t tcount = 0;
        for (uint32_t li = 0; !*abort; ++li) {
            int64_t qi = blockIdx.x + (int64_t)li * gridDim.x;
            int32_t rot = 0;
            if (CLAIM) {  // the block the producer took and its rotation
                const uint32_t rs = li & 3;
                if (!mbar_wait(&rot_full[rs], (li >> 2) & 1, abort, P.error)) break;
                qi = *(volatile int64_t *)&rot_blk[rs];
                rot = *(volatile int32_t *)&rot_val[rs];
                __syncwarp();
                if (lane == 0) mbar_arrive(&rot_empty[rs]);
            }
            if (qi >= P.n_qblocks * P.splits) break;
            const int64_t qb = qi / P.splits;
            const int64_t part = qi % P.splits;
            // the debug entry point dumps query block 0 against tile 0 (its first tile)
            const bool debug = P.debug_tile != nullptr && qb == 0;
            const int64_t row = qb * BM + row_local;  // query row
            const bool valid = row < P.nq;
            const int64_t self = valid && P.qpos ? (int64_t)P.qpos[row] : row;
            const float p_i = valid ? P.pq[row] : 0.0f;
            const float m_i = valid ? P.mq[row] : 0.0f;
            const float ps_i = P.one_minus_cb * p_i - P.abs_c;
            const float cm_i = P.c_a * m_i;
            float core_i = 0.0f;
            int32_t lab_i = -1;
            if (BORUVKA && valid) {
                core_i = P.core[self] * P.s2;
                lab_i = P.label[self];
            }
            // kNN threshold mode: a fixed upper bound of the row's k-th distance (scaled); a row
            // without one overflows its buffer at once and is resolved exactly
            const float tau = THRESH && valid ? P.qthr[row] * P.s2 : CUSCAN_INF;
            const bool tau_ok = !THRESH || tau < CUSCAN_INF;
            // kNN: the row's M smallest lower bounds. Borůvka: an upper bound U on the row's
            // cheapest cross-component edge plus the shared bound of its component; pairs whose
            // lower bound does not exceed min(U, component bound) are appended for re-ranking.
            // kNN threshold: every pair whose lower bound does not exceed tau is appended.
            constexpr int LM = APPEND ? 1 : M;
            float L[LM];
            int J[LM];
#pragma unroll
            for (int s2 = 0; s2 < LM; ++s2) {
                L[s2] = CUSCAN_INF;
                J[s2] = -1;
            }
            float U = CUSCAN_INF, published = CUSCAN_INF;
            float lb_all = CUSCAN_INF;  // one-sided Borůvka: min chunk bound over cross chunks
            int cnt = 0;
            int32_t qlo = 0, qhi = 0;
            if (BORUVKA) qblock_range(P, qb, qlo, qhi);
            const int64_t wa = LIST ? qb * P.n_tiles : window_start(P, qb);
            const int64_t nvis = LIST ? P.vis_count[qb] : vis_count<SYM>(P, qb);
            // this work item's part [i_lo, i_hi) of the block's tile order
            const int64_t i_lo = part * nvis / P.splits, i_hi = (part + 1) * nvis / P.splits;
            // symmetric mode: the warp's 32 rows summarised for the column-side block test
            float psmin_w = CUSCAN_INF, cmmax_w = 0.0f, coremin_w = CUSCAN_INF;
            if (SYM) {
                psmin_w = warp_min_f(valid ? ps_i : CUSCAN_INF);
                cmmax_w = warp_max_f(valid ? cm_i : 0.0f);
                coremin_w = warp_min_f(valid ? core_i : CUSCAN_INF);
            }
            auto tile_at = [&](int64_t i) -> int64_t {
                return LIST  ? (int64_t)P.vis[wa + i]
                       : ROT ? (int64_t)knn_tile((int32_t)P.n_tiles, (int32_t)wa, rot, (int32_t)i)
                             : vis_tile<SYM>(P, qb, wa, i);
            };
            // next visited position i (>= i0) in this block's tile order, and its tile t_at
            int64_t t_at = 0;
            auto next_index = [&](int64_t i) -> int64_t {
                for (; i < i_hi; ++i) {
                    t_at = tile_at(i);
                    if (!tile_skipped<BORUVKA>(P, t_at, qlo, qhi)) break;
                }
                return i;
            };
            // per-tile column data, fetched one tile ahead: the chunk minima of this warp's four
            // chunks (the per-column terms are read where a chunk is tested pair by pair)
            float4 pre_k01 = make_float4(0, 0, 0, 0), pre_k23 = make_float4(0, 0, 0, 0);
            int32_t pre_ch = -2;
            float pre_mt = 0.0f, pre_cb = CUSCAN_INF;
            float4 pre_t = make_float4(0, 0, 0, 0);  // symmetric mode: column row bounds (raw)
            auto prefetch = [&](int64_t t, uint32_t slot) {
                const int64_t col = t * BN + half * HALF + lane * 4;
                pre_k01 = P.cmin[t * 4 + half * 2];
                pre_k23 = P.cmin[t * 4 + half * 2 + 1];
                pre_mt = P.tile_mmax[t];
                if (STAGE) {  // straight into the tile's shared slots (no registers)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                                     smem_u32(my_pb + slot * HALF + lane * 4)),
                                 "l"(P.colp + col)
                                 : "memory");
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                                     smem_u32(my_pb + (2 + slot) * HALF + lane * 4)),
                                 "l"(P.mnorm + col)
                                 : "memory");
                }
                if (BORUVKA) {
                    const int64_t ch = t * 8 + half * 4 + (lane & 3);
                    pre_ch = -2;
                    if (lane < 8 && ch < P.n_chunks) pre_ch = lane < 4 ? P.chunk_lo[ch] : P.chunk_hi[ch];
                    pre_cb = valid ? __uint_as_float(*(volatile uint32_t *)&P.cbound[lab_i])
                                   : CUSCAN_INF;
                    if (SYM) {
                        const volatile uint32_t *ur = P.urow;
                        pre_t.x = col + 0 < P.n ? __uint_as_float(ur[col + 0]) : -CUSCAN_INF;
                        pre_t.y = col + 1 < P.n ? __uint_as_float(ur[col + 1]) : -CUSCAN_INF;
                        pre_t.z = col + 2 < P.n ? __uint_as_float(ur[col + 2]) : -CUSCAN_INF;
                        pre_t.w = col + 3 < P.n ? __uint_as_float(ur[col + 3]) : -CUSCAN_INF;
                    }
                }
            };
            int64_t ti = next_index(i_lo);
            if (ti < i_hi) prefetch(t_at, tcount & 1);
            bool ok = true;
            while (ti < i_hi) {
                const int64_t t = t_at;
                const int64_t ti_next = next_index(ti + 1);
                const uint32_t b = tcount & 1, tp = (tcount >> 1) & 1;
                // this warp's columns: scaled norms pb, norms mb and (Borůvka) scaled cores cb,
                // and (min pb, min cb) of each 32-column chunk
                const int64_t col0 = t * BN + half * HALF;
                const float *pb = STAGE ? my_pb + b * HALF : P.colp + col0;
                const float *mb = STAGE ? my_pb + (2 + b) * HALF : P.mnorm + col0;
                const float *cb = BORUVKA ? P.colc + col0 : nullptr;
                if (STAGE) {  // this tile's column terms, copied one tile ahead
                    asm volatile("cp.async.wait_all;" ::: "memory");
                    __syncwarp();
                }
                const float2 chunk_min[4] = {make_float2(pre_k01.x, pre_k01.y),
                                             make_float2(pre_k01.z, pre_k01.w),
                                             make_float2(pre_k23.x, pre_k23.y),
                                             make_float2(pre_k23.z, pre_k23.w)};
                // symmetric mode: the largest column row bound of each chunk (scaled)
                float chunk_tmax[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                if (SYM) {
                    float tm = fmaxf(fmaxf(pre_t.x, pre_t.y), fmaxf(pre_t.z, pre_t.w)) * P.s2;
#pragma unroll
                    for (int o = 1; o < 8; o <<= 1)
                        tm = fmaxf(tm, __shfl_xor_sync(0xffffffffu, tm, o));
#pragma unroll
                    for (int c = 0; c < 4; ++c) chunk_tmax[c] = __shfl_sync(0xffffffffu, tm, 8 * c);
                }
                const float mt = pre_mt;
                const int32_t ch_word = pre_ch;
                const float comp_bound = pre_cb * P.s2;
                __syncwarp();
                if (ti_next < i_hi) prefetch(t_at, b ^ 1);
                if (!mbar_wait(&t_full[b], tp, abort, P.error)) { ok = false; break; }
                fence_after();
                const uint32_t taddr =
                    tmem_base + ((uint32_t)(quad * 32) << 16) + b * BN + half * HALF;
                // Phase 1: the largest dot product of each 32-column chunk, from the TMEM loads
                // themselves (tcgen05.ld.red); two chunks per wait, as the kNN lists leave room
                // for two 32-column loads in flight.
                // Phase 2: one coarse test per chunk against this tile's thresholds and one warp
                // vote per tile; the chunks that pass are read again from TMEM (the buffer is
                // released only after this tile) and tested element by element.
                float vmax[HALF / 32];
#pragma unroll
                for (int c = 0; c < HALF / 32; c += 2) {
                    uint32_t rA[32], rB[32];
                    tmem_ld32_max_issue(taddr + c * 32, rA, vmax[c]);
                    tmem_ld32_max_issue(taddr + (c + 1) * 32, rB, vmax[c + 1]);
                    tmem_ld_wait(rA);
                    tmem_ld_wait(rB);
                    asm volatile("" : "+f"(vmax[c]), "+f"(vmax[c + 1]));
                    if (debug && t == 0) {
#pragma unroll
                        for (int e = 0; e < 32; ++e) {
                            P.debug_tile[row_local * BN + half * HALF + c * 32 + e] = __uint_as_float(rA[e]);
                            P.debug_tile[row_local * BN + half * HALF + (c + 1) * 32 + e] = __uint_as_float(rB[e]);
                        }
                        if (P.debug_chunk) {
                            P.debug_chunk[row_local * 8 + half * 4 + c] = vmax[c];
                            P.debug_chunk[row_local * 8 + half * 4 + c + 1] = vmax[c + 1];
                        }
                    }
                }
                // Thresholds moved to the scale of F = (1 - C_B) p_j - 2 dot with the tile's
                // largest norm, then widened by a few ulps so that no pair whose exact-path
                // bound would pass is filtered out. For Borůvka the core condition
                // core_j < T rides along as max(F, core_j + (thr2 - T)). The element path
                // recomputes them after it lowers U or the list bound; a stale (larger)
                // threshold only admits more pairs to the exact test.
                float T = 0.0f, dlt = 0.0f, thr_fast = 0.0f;
                auto thresholds = [&]() {
                    T = BORUVKA ? fminf(U, comp_bound) : THRESH ? tau : L[LM - 1];
                    const float base = T - ps_i + cm_i * mt;
                    const float thr2 = base + 0x1p-21f * (fabsf(T) + ps_i + cm_i * mt);
                    dlt = thr2 - T;
                    thr_fast = thr2 + 0x1p-20f * (fabsf(thr2) + fabsf(T));
                };
                thresholds();
                // Coarse test of each chunk: with the chunk's smallest scaled norm and core,
                // fmaf(-2, max v, min pb) is below (or equal to) every element's
                // fmaf(-2, v_j, pb_j) and min core + dlt bounds the core term, because rounding
                // is monotonic.
                unsigned hitbits = 0, mixbits = 0;
                {
                    const bool row_on = valid && tau_ok && (!BORUVKA || core_i <= T);
#pragma unroll
                    for (int c = 0; c < HALF / 32; ++c) {
                        int32_t clo = 0, chi = 0;
                        if (BORUVKA) {
                            clo = __shfl_sync(0xffffffffu, ch_word, c);
                            chi = __shfl_sync(0xffffffffu, ch_word, 4 + c);
                        }
                        const bool cross = !BORUVKA || (clo != -2 && !(clo == lab_i && chi == lab_i));
                        const bool on = row_on && cross;
                        const float2 cmin = chunk_min[c];
                        float flb = fmaf(-2.0f, vmax[c], cmin.x);
                        if (MODE == MODE_BORUVKA && cross) {
                            if (clo <= lab_i && lab_i <= chi) {
                                // the chunk also holds rows of the row's own component: its
                                // bound may come from those, so it is taken pair by pair below
                                mixbits |= 1u << c;
                            } else {
                                // below every pair of the chunk: mb <= mt, dot <= vmax,
                                // pb >= min pb, core_j >= min core, and fmaf/add rounding is
                                // monotonic
                                const float lbc = fmaf(-cm_i, mt, flb + ps_i);
                                lb_all = fminf(lb_all, fmaxf(fmaxf(lbc, core_i), cmin.y));
                            }
                        }
                        if (BORUVKA) flb = fmaxf(flb, cmin.y + dlt);
                        if (on && flb < thr_fast) hitbits |= 1u << c;
                    }
                }
                const unsigned warp_bits = __reduce_or_sync(0xffffffffu, hitbits);
                // Symmetric mode, tiles after the block's own: the pairs of this block are also
                // the pairs of the tile's rows. Block test: with the warp's smallest scaled norm
                // and core and largest C_A m, the chunk's smallest scaled norm and core and the
                // block's largest dot product, fmaf/add rounding being monotonic, wl is below
                // every pair's exact-path bound max(lb, core_i, core_j); only blocks where it
                // reaches a column's row bound are tested pair by pair.
                unsigned colbits = 0;
                if (SYM && t > (qb >> 1)) {
#pragma unroll
                    for (int c = 0; c < HALF / 32; ++c) {
                        const float vb = warp_max_f(vmax[c]);
                        const float2 cmn = chunk_min[c];
                        const float lbb = fmaf(-cmmax_w, mt, fmaf(-2.0f, vb, cmn.x) + psmin_w);
                        const float wl = fmaxf(fmaxf(lbb, coremin_w), cmn.y);
                        if (wl <= chunk_tmax[c]) colbits |= 1u << c;
                    }
                }
                for (int c = 0; colbits != 0 && c < HALF / 32; ++c) {
                    if (!((colbits >> c) & 1u)) continue;
                    uint32_t rc2[32];
                    tmem_ld32_issue(taddr + c * 32, rc2);
                    // lane e refreshes column e's row bound with its component's current bound
                    // (rows of components that found edges elsewhere get tight at once)
                    const int64_t j0 = t * BN + half * HALF + c * 32;
                    int32_t lab_l = -1;
                    float t_l = -CUSCAN_INF;
                    if (j0 + lane < P.n) {
                        lab_l = P.label[j0 + lane];
                        const uint32_t cbv = *(volatile uint32_t *)&P.cbound[lab_l];
                        const uint32_t old = atomicMin(&P.urow[j0 + lane], cbv);
                        t_l = __uint_as_float(old < cbv ? old : cbv) * P.s2;
                    }
                    tmem_ld_wait(rc2);
#pragma unroll
                    for (int e = 0; e < 32; ++e) {
                        const float tj = __shfl_sync(0xffffffffu, t_l, e);
                        const int32_t lab_j = __shfl_sync(0xffffffffu, lab_l, e);
                        const int col = c * 32 + e;
                        const int64_t j = j0 + e;
                        if (j >= P.n) break;  // the same for every lane
                        const float lb = fmaf(-cm_i, mb[col],
                                              fmaf(-2.0f, __uint_as_float(rc2[e]), pb[col]) + ps_i);
                        const float cj = cb[col];
                        const float lbw = fmaxf(fmaxf(lb, core_i), cj);
                        const bool pv = valid && lab_j != lab_i && lbw <= tj;
                        const float eps2 =
                            2.0f * fmaf(cm_i, mb[col], P.c_b * (ps_i + pb[col]) * 1.001f) +
                            4.0f * P.abs_c;
                        const float ubr = lb + eps2;
                        const float ub =
                            fmaxf(fmaxf(ubr + 0x1p-20f * (fabsf(ubr) + eps2), core_i), cj);
                        // the block's best upper bound for this column's row: a pair above
                        // it cannot be the row's cheapest edge
                        const float tmin = warp_min_f(pv ? ub : CUSCAN_INF);
                        if (pv && lbw <= tmin) {
                            const int slot = atomicAdd(&P.colcnt[j], 1);
                            if (slot < P.capc) P.colbuf[j * P.capc + slot] = (int32_t)row;
                        }
                        if (lane == 0 && tmin < CUSCAN_INF) {
                            const uint32_t ub_raw = __float_as_uint(__fmul_ru(tmin, P.inv_s2));
                            atomicMin(&P.urow[j], ub_raw);
                            atomicMin(&P.cbound[lab_j], ub_raw);
                        }
                    }
                    __syncwarp();
                }
                for (int c = 0; warp_bits != 0 && c < HALF / 32; ++c) {
                    if (!((warp_bits >> c) & 1u)) continue;
                    uint32_t rc_[32];
                    tmem_ld32_issue(taddr + c * 32, rc_);
                    tmem_ld_wait(rc_);
                    float v[32];
#pragma unroll
                    for (int e = 0; e < 32; ++e) v[e] = __uint_as_float(rc_[e]);
                    const bool any_hit = (hitbits >> c) & 1u;
                    {

                        unsigned hits = 0;
                        if (any_hit) {
                            const float4 *pc = reinterpret_cast<const float4 *>(pb + c * 32);
                            const float4 *cc = reinterpret_cast<const float4 *>(cb + c * 32);
#pragma unroll
                            for (int q = 0; q < 8; ++q) {
                                const float4 pq = pc[q];
                                float f0 = fmaf(-2.0f, v[4 * q + 0], pq.x);
                                float f1 = fmaf(-2.0f, v[4 * q + 1], pq.y);
                                float f2 = fmaf(-2.0f, v[4 * q + 2], pq.z);
                                float f3 = fmaf(-2.0f, v[4 * q + 3], pq.w);
                                if (BORUVKA) {
                                    // core_j <= T is necessary for an append
                                    const float4 cq = cc[q];
                                    f0 = fmaxf(f0, cq.x + dlt);
                                    f1 = fmaxf(f1, cq.y + dlt);
                                    f2 = fmaxf(f2, cq.z + dlt);
                                    f3 = fmaxf(f3, cq.w + dlt);
                                }
                                hits |= (f0 < thr_fast ? 1u : 0u) << (4 * q + 0);
                                hits |= (f1 < thr_fast ? 1u : 0u) << (4 * q + 1);
                                hits |= (f2 < thr_fast ? 1u : 0u) << (4 * q + 2);
                                hits |= (f3 < thr_fast ? 1u : 0u) << (4 * q + 3);
                            }
#pragma unroll
                            for (int q = 0; q < 8; ++q)
                                reinterpret_cast<float4 *>(my_v)[q] =
                                    make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                        }
                        int32_t clo = 0, chi = 0;
                        if (BORUVKA) {
                            clo = __shfl_sync(0xffffffffu, ch_word, c);
                            chi = __shfl_sync(0xffffffffu, ch_word, 4 + c);
                        }
                        const bool uniform_other = BORUVKA && clo == chi && clo != lab_i;
                        while (hits) {
                            const int e = __ffs(hits) - 1;
                            hits &= hits - 1;
                            const int col = c * 32 + e;
                            const int64_t j = t * BN + half * HALF + col;
                            if (j >= P.n) continue;
                            if (!BORUVKA && j == self) continue;
                            const float dot = my_v[e];
                            // exact lower bound for this pair (per-column norm instead of the
                            // tile maximum); pb holds (1 - C_B) p_j
                            float lb = fmaf(-cm_i, mb[col], fmaf(-2.0f, dot, pb[col]) + ps_i);
                            if constexpr (BORUVKA) {
                                if (!uniform_other && P.label[j] == lab_i) continue;
                                const float cj = cb[col];
                                const float lbw = fmaxf(fmaxf(lb, core_i), cj);
                                const float Tn = fminf(U, comp_bound);
                                if (lbw <= Tn) {
                                    // split work items share the row's slots
                                    const int slot = P.splits > 1
                                        ? atomicAdd(&P.rowcnt[row * 2 + half], 1) : cnt;
                                    if (slot < P.cap) P.cand_ids[(row * 2 + half) * P.cap + slot] = (int32_t)j;
                                    ++cnt;
                                    // upper bound of this pair's weight: D + eps = L + 2 eps
                                    const float eps2 =
                                        2.0f * fmaf(cm_i, mb[col], P.c_b * (ps_i + pb[col]) * 1.001f) +
                                        4.0f * P.abs_c;
                                    const float ubr = lb + eps2;
                                    const float ub = fmaxf(fmaxf(ubr + 0x1p-20f * (fabsf(ubr) + eps2), core_i), cj);
                                    U = fminf(U, ub);
                                }
                            } else if constexpr (THRESH) {
                                if (lb <= tau) {
                                    if (cnt < P.cap) P.cand_ids[(row * 2 + half) * P.cap + cnt] = (int32_t)j;
                                    ++cnt;
                                }
                            } else {
                                if (lb < L[LM - 1]) list_insert<LM>(L, J, lb, (int)j);
                            }
                        }
                        __syncwarp();
                        thresholds();
                    }
                }
                // one-sided Borůvka: row bounds over the chunks shared with the own component,
                // other components' pairs only (at most a couple of chunks per component)
                if (MODE == MODE_BORUVKA) {
                    const unsigned wmix = __reduce_or_sync(0xffffffffu, mixbits);
                    for (int c = 0; wmix != 0 && c < HALF / 32; ++c) {
                        if (!((wmix >> c) & 1u)) continue;
                        uint32_t rm[32];
                        tmem_ld32_issue(taddr + c * 32, rm);
                        tmem_ld_wait(rm);
                        if ((mixbits >> c) & 1u) {
                            const int64_t j0 = t * BN + half * HALF + c * 32;
                            // fully unrolled: rm stays in registers
#pragma unroll
                            for (int e = 0; e < 32; ++e) {
                                const int col = c * 32 + e;
                                if (j0 + e >= P.n || P.label[j0 + e] == lab_i) continue;
                                const float lb = fmaf(-cm_i, mb[col],
                                                      fmaf(-2.0f, __uint_as_float(rm[e]), pb[col]) + ps_i);
                                lb_all = fminf(lb_all, fmaxf(fmaxf(lb, core_i), cb[col]));
                            }
                        }
                        __syncwarp();
                    }
                }
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&t_empty[b]);
                if (BORUVKA && valid && U < published) {
                    // raw units, rounded up so that the bound stays an upper bound
                    const uint32_t u_raw = __float_as_uint(__fmul_ru(U, P.inv_s2));
                    atomicMin(&P.cbound[lab_i], u_raw);
                    if (SYM) atomicMin(&P.urow[row], u_raw);
                    published = U;
                }
                ++tcount;
                ti = ti_next;
            }
            if (!ok) break;
            if (APPEND) {
                // each half of a row appends into its own slot range [(2 row + half) * cap, +cap)
                if (valid && P.splits == 1) P.rowcnt[row * 2 + half] = tau_ok ? cnt : P.cap + 1;
                if (MODE == MODE_BORUVKA && valid && P.rowlb) {
                    const float lbr = __fmul_rd(lb_all, P.inv_s2);
                    if (P.splits == 1) {
                        P.rowlb[row * 2 + half] = lbr;
                    } else {
                        // the least over the block's parts; pair weights are >= 0, so a bound
                        // below 0 is worth 0 and the bounds compare as unsigned bit patterns
                        atomicMin(reinterpret_cast<unsigned int *>(P.rowlb) + row * 2 + half,
                                  __float_as_uint(lbr > 0.0f ? lbr : 0.0f));
                    }
                }
            } else if (valid) {
                const int64_t base_at = row * (2 * M) + half * M;
#pragma unroll
                for (int s2 = 0; s2 < LM; ++s2) {
                    P.cand_ids[base_at + s2] = J[s2];
                    // raw units, rounded down so that the bound stays a lower bound
                    P.cand_lb[base_at + s2] = __fmul_rd(L[s2], P.inv_s2);
                }
            }
        }
        // copies of column terms still in flight (a loop left early) land before the CTA exits
        if (STAGE) asm volatile("cp.async.wait_all;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    if (warp == 1) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base)
                     : "memory");
    }
}

// Exact squared distance (the reference's order) from the warp's query row q_s (shared) to the
// candidate row j held by this lane (j < 0: none, returns +inf). The warp first copies the 32
// candidate rows into its shared staging area, then every lane sums its own row sequentially.
// What bounds it is the copies (32 rows of L2 per 32 candidates). VEC: rows of d % 4 == 0 features
// on 16-byte boundaries move in 16-byte pieces, 32 / (d / 4) rows per instruction, and are read
// back as float4 (row stride d + 4: eight lanes cover the 32 banks); other rows move in 4-byte
// pieces with row stride d + 1. 500,000 x 128 rows, 32 candidates each: 3.1 ms against 4.0 ms
// in 4-byte pieces.
template <bool VEC>
__device__ __forceinline__ float staged_d2(const float *__restrict__ x, int d,
                                           const float *q_s, int32_t j, float *rows_s,
                                           int lane) {
    float acc = CUSCAN_INF;
    if (VEC) {
        const int pieces = d >> 2, total = 32 * pieces, stride = d + 4;
        for (int p0 = 0; p0 < total; p0 += 32) {
            const int p = p0 + lane;  // total is a multiple of 32
            const int r = p / pieces, c = p - r * pieces;
            const int32_t jr = __shfl_sync(0xffffffffu, j, r);
            if (jr >= 0)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                                 smem_u32(rows_s + r * stride + 4 * c)),
                             "l"(x + (int64_t)jr * d + 4 * c)
                             : "memory");
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
        if (j >= 0) {
            const float4 *row = reinterpret_cast<const float4 *>(rows_s + lane * stride);
            const float4 *q = reinterpret_cast<const float4 *>(q_s);
            acc = 0.0f;
#pragma unroll 4
            for (int c = 0; c < pieces; ++c) {
                const float4 a = q[c], b = row[c];
                const float t0 = a.x - b.x, t1 = a.y - b.y, t2 = a.z - b.z, t3 = a.w - b.w;
                acc = __fmaf_rn(t0, t0, acc);
                acc = __fmaf_rn(t1, t1, acc);
                acc = __fmaf_rn(t2, t2, acc);
                acc = __fmaf_rn(t3, t3, acc);
            }
        }
    } else {
        for (int r = 0; r < 32; ++r) {
            const int32_t jr = __shfl_sync(0xffffffffu, j, r);
            if (jr < 0) continue;
            const float *src = x + (int64_t)jr * d;
            float *dst = rows_s + r * (d + 1);
            for (int f = lane; f < d; f += 32)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst + f)),
                             "l"(src + f)
                             : "memory");
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
        if (j >= 0) {
            const float *row = rows_s + lane * (d + 1);
            acc = 0.0f;
            for (int f = 0; f < d; ++f) {
                const float t = q_s[f] - row[f];
                acc = __fmaf_rn(t, t, acc);
            }
        }
    }
    __syncwarp();
    return acc;
}

// Shared floats one warp of a re-rank kernel stages: 32 candidate rows and the query row (a multiple
// of four with VEC, so that every warp's rows stay on 16-byte boundaries).
__host__ __device__ constexpr int64_t rerank_warp_floats(int d, bool vec) {
    return vec ? 32 * (d + 4) + d : 32 * (d + 1) + d;
}
static bool rerank_vec(const float *x, int d) {
    return d % 4 == 0 && reinterpret_cast<uintptr_t>(x) % 16 == 0;
}
constexpr int RERANK_WARPS = 4;

__device__ __forceinline__ unsigned long long warp_min_u64(unsigned long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        unsigned long long u = __shfl_xor_sync(0xffffffffu, v, o);
        v = u < v ? u : v;
    }
    return v;
}

// Lower bound of every pair a row's two lists left out: a full list rejected or evicted only
// pairs whose bound is >= its M-th entry; a list that is not full kept every pair it saw.
template <int M>
__device__ __forceinline__ float unseen_bound(const int32_t *ids, const float *lb) {
    float b = CUSCAN_INF;
#pragma unroll
    for (int h = 0; h < 2; ++h)
        if (ids[h * M + M - 1] >= 0) b = fminf(b, lb[h * M + M - 1]);
    return b;
}

// kNN re-rank: one warp per row, exact distances of the 2M candidates, top-k by (d, id).
// x and the candidates are in sorted positions; perm maps a position to its original row, which
// is the id the reference orders ties by and the row the output goes to.
template <int M, bool VEC>
__global__ void rerank_knn_kernel(const float *__restrict__ x, const int32_t *__restrict__ perm,
                                  int64_t n, int d, int k, const int32_t *__restrict__ cand_ids,
                                  const float *__restrict__ cand_lb, int32_t *__restrict__ ids,
                                  float *__restrict__ dist, int32_t *__restrict__ fallback,
                                  float *__restrict__ fallback_thr,
                                  int *__restrict__ fallback_count) {
    extern __shared__ __align__(16) float rerank_smem[];
    const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (row >= n) return;
    float *q_s = rerank_smem + (threadIdx.x >> 5) * rerank_warp_floats(d, VEC);
    float *rows_s = q_s + d;
    for (int f = lane; f < d; f += 32) q_s[f] = x[row * d + f];
    __syncwarp();
    constexpr int W = 2 * M;  // two lists of M per row (one per column half)
    // Each half's list is sorted by lower bound. The first round takes the F smallest bounds of
    // both lists (lanes 0..15: half 0, lanes 16..31: half 1); the rest, R per half, run in a
    // second round only when the smaller of their two first bounds does not exceed the k-th
    // distance of the first round, an upper bound of the final k-th distance: a candidate whose
    // lower bound exceeds it cannot be among the row's k nearest.
    constexpr int F = M < 16 ? M : 16;
    constexpr int R = M - F;
    static_assert(R <= 16, "two rounds of at most 16 candidates per half");
    constexpr int PER = 2;
    unsigned long long key[PER] = {~0ull, ~0ull};
    auto round_key = [&](int first, int count) -> unsigned long long {
        const int h = lane >> 4, o = lane & 15;
        const int32_t j = o < count ? cand_ids[row * W + h * M + first + o] : -1;
        const float dd = staged_d2<VEC>(x, d, q_s, j, rows_s, lane);
        return j < 0 ? ~0ull : ((unsigned long long)__float_as_uint(dd) << 32) | (uint32_t)perm[j];
    };
    key[0] = round_key(0, F);
    if (R > 0) {
        // k-th smallest key of the first round (all keys distinct: the halves hold disjoint
        // columns)
        unsigned long long a = key[0], kth = ~0ull;
        for (int r = 0; r < k; ++r) {
            kth = warp_min_u64(a);
            if (kth == ~0ull) break;
            if (a == kth) a = ~0ull;
        }
        const float dk0 = kth == ~0ull ? CUSCAN_INF : __uint_as_float((uint32_t)(kth >> 32));
        float lb_rest = CUSCAN_INF;
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (cand_ids[row * W + h * M + F] >= 0) lb_rest = fminf(lb_rest, cand_lb[row * W + h * M + F]);
        if (!(lb_rest > dk0)) key[1] = round_key(F, R);
    }
    const int64_t orow = perm[row];
    float dk = CUSCAN_INF;
    for (int r = 0; r < k; ++r) {
        unsigned long long mine = key[0];
#pragma unroll
        for (int q = 1; q < PER; ++q) mine = key[q] < mine ? key[q] : mine;
        const unsigned long long best = warp_min_u64(mine);
#pragma unroll
        for (int q = 0; q < PER; ++q)
            if (key[q] == best) key[q] = ~0ull;
        if (best == ~0ull) {
            if (lane == 0) {
                ids[orow * k + r] = (int32_t)n;
                dist[orow * k + r] = CUSCAN_INF;
            }
            dk = CUSCAN_INF;
        } else {
            dk = __uint_as_float((uint32_t)(best >> 32));
            if (lane == 0) {
                ids[orow * k + r] = (int32_t)(uint32_t)best;
                dist[orow * k + r] = dk;
            }
        }
    }
    // every pair outside a full list has a lower bound >= that list's M-th bound; an
    // inconclusive row is listed by position with dk, an upper bound of its k-th distance
    const float bound = unseen_bound<M>(cand_ids + row * W, cand_lb + row * W);
    if (lane == 0 && !(bound > dk)) {
        const int at = atomicAdd(fallback_count, 1);
        fallback[at] = (int32_t)row;
        fallback_thr[at] = dk;
    }
}

// kNN re-rank of the threshold screen: query q (position qpos[q]) holds every pair whose lower
// bound does not exceed an upper bound of its k-th distance, so the exact top k of its appended
// candidates by (d, original id) is its exact kNN row. A buffer that overflowed (or a row with
// fewer than k candidates) sends the row's original index to the exact f32 sweep.
template <bool VEC>
__global__ void rerank_knn_threshold_kernel(const float *__restrict__ x,
                                            const int32_t *__restrict__ perm,
                                            const int32_t *__restrict__ qpos, int64_t nq, int d,
                                            int k, const int32_t *__restrict__ cand_ids,
                                            const int32_t *__restrict__ rowcnt, int cap,
                                            int32_t *__restrict__ ids, float *__restrict__ dist,
                                            int32_t *__restrict__ fallback,
                                            int *__restrict__ fallback_count) {
    const int64_t q = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (q >= nq) return;
    constexpr int PER = 2 * KNN_CAP / 32;
    const int64_t pos = qpos[q];
    const int64_t orow = perm[pos];
    const int c0 = rowcnt[q * 2], c1 = rowcnt[q * 2 + 1];
    if (c0 > cap || c1 > cap || c0 + c1 < k) {
        if (lane == 0) fallback[atomicAdd(fallback_count, 1)] = (int32_t)orow;
        return;
    }
    extern __shared__ __align__(16) float rerank_smem[];
    float *q_s = rerank_smem + (threadIdx.x >> 5) * rerank_warp_floats(d, VEC);
    float *rows_s = q_s + d;
    for (int f = lane; f < d; f += 32) q_s[f] = x[pos * d + f];
    __syncwarp();
    unsigned long long key[PER];
#pragma unroll
    for (int t = 0; t < PER; ++t) {
        const int s = lane + 32 * t;
        int32_t j = -1;
        if (s < c0 + c1)
            j = s < c0 ? cand_ids[(q * 2) * cap + s] : cand_ids[(q * 2 + 1) * cap + (s - c0)];
        // every lane joins the staging (it is warp-wide), the rounds are uniform per warp
        const float dd = t * 32 < c0 + c1 ? staged_d2<VEC>(x, d, q_s, j, rows_s, lane) : CUSCAN_INF;
        key[t] = j < 0 ? ~0ull : ((unsigned long long)__float_as_uint(dd) << 32) | (uint32_t)perm[j];
    }
    for (int r = 0; r < k; ++r) {
        unsigned long long mine = key[0];
#pragma unroll
        for (int t = 1; t < PER; ++t) mine = key[t] < mine ? key[t] : mine;
        const unsigned long long best = warp_min_u64(mine);
#pragma unroll
        for (int t = 0; t < PER; ++t)
            if (key[t] == best) key[t] = ~0ull;
        if (lane == 0) {
            ids[orow * k + r] = (int32_t)(uint32_t)best;
            dist[orow * k + r] = __uint_as_float((uint32_t)(best >> 32));
        }
    }
}

// Original row of each listed position (in place).
__global__ void positions_to_rows_kernel(int32_t *__restrict__ list, int64_t count,
                                         const int32_t *__restrict__ perm) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) list[i] = perm[list[i]];
}

// Borůvka re-rank over component-sorted positions: exact weight of every appended candidate of
// both row halves, row minimum (w, original j) into row_keys[original row]. Rows whose buffer
// overflowed are re-run exactly; rows without candidates keep an empty key (they cannot hold
// their component's cheapest edge: every pair reaching it is appended).
template <bool VEC>
__global__ void rerank_boruvka_kernel(const float *__restrict__ xp, const float *__restrict__ corep,
                                      const int32_t *__restrict__ labp,
                                      const int32_t *__restrict__ perm, int64_t nq,
                                      const int32_t *__restrict__ qpos, int d,
                                      const int32_t *__restrict__ cand_ids,
                                      const int32_t *__restrict__ rowcnt, int cap,
                                      const int32_t *__restrict__ colcnt,
                                      const int32_t *__restrict__ colbuf, int capc,
                                      const float *__restrict__ lbtmp, float *__restrict__ rowlb,
                                      unsigned long long *__restrict__ row_keys,
                                      int32_t *__restrict__ fallback,
                                      int *__restrict__ fallback_count) {
    // q indexes the screened rows (all positions, or the gathered positions qpos)
    const int64_t q = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (q >= nq) return;
    const int64_t pos = qpos ? (int64_t)qpos[q] : q;
    // Fold the one-sided screen's bounds (two column halves per query row) into the per-row lower
    // bounds, kept in original row order across rounds.
    if (lbtmp && lane == 0) {
        const int32_t orow = perm[pos];
        rowlb[orow] = fmaxf(rowlb[orow], fminf(lbtmp[2 * q], lbtmp[2 * q + 1]));
    }
    const int c0 = rowcnt[q * 2], c1 = rowcnt[q * 2 + 1];
    const int c2 = colcnt ? colcnt[pos] : 0;  // pairs other blocks appended for this row
    if (c0 > cap || c1 > cap || c2 > capc) {
        if (lane == 0) {
            const int at = atomicAdd(fallback_count, 1);
            fallback[at] = (int32_t)pos;
        }
        return;
    }
    const int total = c0 + c1 + c2;
    if (total == 0) return;  // no candidate: the row keeps an empty key
    extern __shared__ __align__(16) float rerank_smem[];
    float *q_s = rerank_smem + (threadIdx.x >> 5) * rerank_warp_floats(d, VEC);
    float *rows_s = q_s + d;
    for (int f = lane; f < d; f += 32) q_s[f] = xp[pos * d + f];
    __syncwarp();
    const float ci = corep[pos];
    const int32_t li = labp[pos];
    unsigned long long mine = ~0ull;
    for (int base = 0; base < total; base += 32) {
        const int s = base + lane;
        int32_t j = -1;
        if (s < total) {
            j = s < c0        ? cand_ids[(q * 2) * cap + s]
                : s < c0 + c1 ? cand_ids[(q * 2 + 1) * cap + (s - c0)]
                              : colbuf[pos * capc + (s - c0 - c1)];
            if (labp[j] == li) j = -1;
        }
        const float d2 = staged_d2<VEC>(xp, d, q_s, j, rows_s, lane);
        if (j < 0) continue;
        const float w = fmaxf(fmaxf(d2, ci), corep[j]);
        if (w != w) continue;
        const unsigned long long key =
            ((unsigned long long)weight_key_bits(w) << 32) | (uint32_t)perm[j];
        mine = key < mine ? key : mine;
    }
    const unsigned long long best = warp_min_u64(mine);
    if (lane == 0 && best != ~0ull) row_keys[perm[pos]] = best;
}

// Upper bounds of each component's cheapest edge from the exact kNN rows: a neighbour in another
// component is an edge of known exact weight max(d2, core_i, core_j).
__global__ void seed_bounds_kernel(const int32_t *__restrict__ knn_ids,
                                   const float *__restrict__ knn_sq, int k,
                                   const float *__restrict__ core, const int32_t *__restrict__ label,
                                   int64_t n, uint32_t *__restrict__ cbound) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int32_t li = label[i];
    const float ci = core[i];
    float best = CUSCAN_INF;
    for (int s = 0; s < k; ++s) {
        const int32_t j = knn_ids[i * k + s];
        if (j < 0 || (int64_t)j >= n || label[j] == li) continue;
        best = fminf(best, fmaxf(fmaxf(knn_sq[i * k + s], ci), core[j]));
    }
    if (best < CUSCAN_INF) atomicMin(&cbound[li], __float_as_uint(best));
}

// Per-row bounds of the symmetric screen: the bound of the row's component.
// Also counts the rows whose component has no bound yet.
// Row bounds of the symmetric screen (the component bounds), the count of rows without one, and
// the rows that can hold their component's cheapest edge. Every edge of row i weighs at least
// core_i and at least the row's lower bound from earlier rounds (its component has only grown
// since, so it has fewer cross edges); a row where either exceeds its component's upper bound
// cannot hold the cheapest edge, ties included.
__global__ void init_row_bounds_kernel(const uint32_t *__restrict__ cbound,
                                       const int32_t *__restrict__ labp,
                                       const float *__restrict__ corep,
                                       const float *__restrict__ rowlb,
                                       const int32_t *__restrict__ perm, int64_t n,
                                       uint32_t *__restrict__ urow, int *__restrict__ unbounded,
                                       int32_t *__restrict__ active) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool inf = false;
    if (i < n) {
        const uint32_t b = cbound[labp[i]];
        urow[i] = b;
        inf = b >= 0x7f800000u;
        const float ub = __uint_as_float(b);
        active[i] = !(corep[i] > ub) && !(rowlb[perm[i]] > ub) ? 1 : 0;
    }
    const unsigned m = __ballot_sync(0xffffffffu, inf);
    if ((threadIdx.x & 31) == 0 && m) atomicAdd(unbounded, __popc(m));
}

// Start of a screened round: no component bound, empty column-side buffers, zero counts and, in a
// fit's first round (rowlb given), no row bounds.
__global__ void round_clear_kernel(uint32_t *__restrict__ cbound, int32_t *__restrict__ colcnt,
                                   float *__restrict__ rowlb, int32_t *__restrict__ count,
                                   int64_t n) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < 2) count[i] = 0;
    if (i >= n) return;
    cbound[i] = 0x7f800000u;
    colcnt[i] = 0;
    if (rowlb) rowlb[i] = 0.0f;
}

// Exact rounds: the weight of each scanned row's cheapest cross-component edge (the top half of
// its candidate key) is a lower bound of its cheapest cross edge in every later round, because
// merging components only removes cross edges. A row without a candidate keeps ~0: +inf.
__global__ void row_lb_from_keys_kernel(const unsigned long long *__restrict__ row_keys,
                                        const int32_t *__restrict__ qpos,
                                        const int32_t *__restrict__ perm, int64_t nq,
                                        const int32_t *__restrict__ labp,
                                        const uint32_t *__restrict__ cbound,
                                        float *__restrict__ rowlb) {
    int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= nq) return;
    const int64_t pos = qpos ? (int64_t)qpos[q] : q;
    const int32_t orow = perm[pos];
    const unsigned long long key = row_keys[orow];  // keys are kept by original row
    float w = key == ~0ull ? CUSCAN_INF : __uint_as_float((uint32_t)(key >> 32));
    // a pruned round left out pairs above the smaller of the row's best and its component's bound
    if (cbound) w = fminf(w, __uint_as_float(cbound[labp[pos]]));
    rowlb[orow] = fmaxf(rowlb[orow], w);
}

// Positions of the flagged rows, in order (idx is the exclusive scan of the flags).
__global__ void compact_positions_kernel(const int32_t *__restrict__ flag,
                                         const int32_t *__restrict__ idx,
                                         const int32_t *__restrict__ sums, int64_t n,
                                         int32_t *__restrict__ out) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && flag[i]) out[idx[i] + sums[i / kScanTile]] = (int32_t)i;
}

__global__ void fill_u32_kernel(uint32_t *p, int64_t n, uint32_t v) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = v;
}

// Error bound coefficients of one operand format (fmt) at d features, K blocks of 64 (d_pad).
//  * Operands: unit roundoff u = 2^-8 (bf16) or 2^-11 (fp16 of the scaled values; |x * scale|
//    <= 2^15, so nothing overflows). Split bf16 represents x = hi + lo + e with |e| <= u^2 |x|,
//    so hi.hi' + hi.lo' + lo.hi' misses x.y by at most u^2 (3 + 4u) |x||y| per feature instead
//    of (2u + u^2) |x||y|.
//  * Accumulation: the K products of an entry (d_pad, or 3 d_pad for split operands) are
//    assumed to come out of the tensor core's f32 accumulation within K 2^-23 of the sum of
//    their magnitudes, two f32 units in the last place per product where f32 sequential
//    summation needs one. tests/test_gpu_accumulation.py drives the accumulator with
//    adversarial operands and requires the observed worst case to stay within a quarter of it.
//  * C_B: norms and the reference sum each carry at most (d + 2) f32 roundings; the epilogue
//    adds a few more; everything is taken three times over.
//  * abs_c: scaled fp16 values below 2^-14 round in the subnormal range with an absolute error
//    of at most 2^-25, which adds at most 2 [2^-25 (1 + u) sqrt(d) (m_i + m_j) + d 2^-50] to the
//    distance; with every scaled norm at most sqrt(d) 2^15 this is a constant. bf16 values (hi,
//    lo) in the subnormal range, or flushed to zero, err by at most 2^-126 each.
void error_coefficients(int d, int d_pad, int fmt, float absmax, float &c_a, float &c_b,
                        float &abs_c) {
    const bool fp16 = fmt == FMT_FP16;
    const double u = std::ldexp(1.0, fp16 ? -11 : -8);  // unit roundoff (round to nearest)
    const double u32 = std::ldexp(1.0, -24);            // f32 unit roundoff
    const double K = fmt == FMT_SPLIT ? 3.0 * d_pad : (double)d_pad;
    double rnd, mag;
    if (fmt == FMT_SPLIT) {
        rnd = u * u * (3.0 + 4.0 * u);
        mag = (1 + u) * (1 + u) * (1 + 2 * u * (1 + u));
    } else {
        rnd = 2.0 * u + u * u;
        mag = (1 + u) * (1 + u);
    }
    const double a1 = rnd + K * std::ldexp(1.0, -23) * mag;
    const double b = 3.5 * (double)(d + 4) * u32 + 1e-7;
    c_a = (float)(2.0 * a1 * (1.0 + 1e-4));
    c_b = (float)b;
    const double dd = (double)d;
    if (fp16) {
        const double eta = std::ldexp(1.0, -25);
        const double m_max = std::sqrt(dd) * std::ldexp(1.0, 15);
        abs_c = (float)(2.0 * (eta * (1 + u) * std::sqrt(dd) * 2.0 * m_max + dd * eta * eta) * 1.01);
    } else {
        abs_c = (float)(std::ldexp(1.0, -126) * (8.0 * dd * (double)absmax * 1.01 + 2.0 * K));
    }
}

// Power-of-two scale that brings the largest |x| into [2^14, 2^15) for fp16 operands; 0 when
// no such scale keeps scale^2 and the scaled sums inside the f32 range (bf16 is used then).
float fp16_scale(float absmax) {
    if (absmax == 0.0f) return 1.0f;
    if (!(absmax > 0.0f) || !std::isfinite(absmax)) return 0.0f;
    int e = 0;
    std::frexp((double)absmax, &e);  // absmax in [2^(e-1), 2^e)
    const int k = 15 - e;            // absmax * 2^k in [2^14, 2^15)
    if (k > 60 || k < -60) return 0.0f;
    return (float)std::ldexp(1.0, k);
}

}  // namespace

int refined_available() { return 1; }

struct Layout {
    int d_pad, kblocks, stages, stage_blocks;
    int nbk, split;  // K blocks per tile row of the copy; split bf16 copy
    int64_t n_pad, n_tiles, n_qblocks;
    size_t smem;
};

// Tiling of n rows of d features: up to four 64-column K blocks. Split copies hold hi and lo
// blocks and cost three MMAs per block pair; they are used up to d = 64 (wider rows take scaled
// fp16 operands, one MMA per block).
static bool refined_layout(int64_t n, int d, Layout &L, bool split = false) {
    L.d_pad = (int)ceil_div(d, 64) * 64;
    if (L.d_pad > (split ? 64 : 256)) return false;
    L.kblocks = L.d_pad / 64;
    L.split = split ? 1 : 0;
    L.nbk = split ? 2 * L.kblocks : L.kblocks;
    L.n_tiles = ceil_div(n, BN);
    L.n_pad = L.n_tiles * BN;
    L.n_qblocks = ceil_div(n, BM);
    L.stage_blocks = L.nbk <= 2 ? L.nbk : 1;
    const size_t a = (size_t)L.nbk * KBLOCK_A, b = (size_t)L.stage_blocks * KBLOCK_B;
    const size_t fixed = a + (size_t)EPI_WARPS * (PB_STRIDE + 32 * VSTRIDE) * 4 +
                         256 + 1024;
    int st = (int)((227 * 1024 - fixed) / b);
    if (st > 4) st = 4;
    if (st < 2) return false;
    L.stages = st;
    L.smem = fixed + (size_t)st * b;
    return true;
}

// Shapes beyond these run the exact sweeps on a lean context.
constexpr int LEAN_MAX_FEATURES = 128;
constexpr int SCREEN_MAX_K = 32;  // longer lists run the exact kNN sweep, and screened rounds
static bool lean_exact(int d, int k) { return d > LEAN_MAX_FEATURES || k > SCREEN_MAX_K; }

static bool refined_shape_ok(int64_t n, int d, int k) {
    Layout L;
    return n >= 2048 && k <= SCREEN_MAX_K && refined_layout(n, d, L);
}


size_t refined_workspace_bytes(int64_t n, int d, int k, bool lean) {
    Layout L;
    if ((lean && lean_exact(d, k)) || !refined_shape_ok(n, d, 1) || !refined_layout(n, d, L)) return 0;
    // a bf16-refined fit may switch to split copies (twice the columns) when d <= 64
    const size_t copy_cols = (size_t)L.d_pad * (L.d_pad <= 64 ? 2 : 1);
    size_t b = (size_t)L.n_pad * copy_cols * 2 + 2 * sizeof(float) * (size_t)L.n_pad;  // xt, norms
    b += 3 * sizeof(float) * (size_t)L.n_tiles + 64;          // tile stats, flags, cursor
    b += 2 * sizeof(float) * (size_t)L.n_pad + sizeof(float) * (size_t)L.n_pad / 16;  // column terms
    b += sizeof(int32_t) * (size_t)n;                                                 // fallback
    // candidates of both row halves, and with lists their bounds
    b += 4 * (size_t)n * 2 * BORUVKA_CAP + (k <= SCREEN_MAX_K ? 4 * (size_t)n * 2 * KNN_LIST : 0);
    b += sizeof(uint32_t) * (size_t)n + 2 * sizeof(int32_t) * (size_t)n;  // cbound, rowcnt
    b += cells_workspace_bytes(n, d);
    // gathered query rows (subset rounds, threshold re-screen): tiles and norms
    b += (size_t)L.n_pad * copy_cols * 2 + 2 * sizeof(float) * (size_t)L.n_pad;
    // threshold re-screen of inconclusive kNN rows (at most all n): thresholds, candidates, counts,
    // fallback list
    if (k <= SCREEN_MAX_K) b += 4 * (size_t)n + 4 * (size_t)n * 2 * KNN_CAP + 8 * (size_t)n + 4 * (size_t)n;
    // symmetric Borůvka: row bounds, column-side counts and candidates; subset rounds: flags,
    // their scan and the gathered positions
    b += 8 * (size_t)n + 4 * (size_t)n * BORUVKA_COL_CAP + 12 * (size_t)n;
    b += 12 * (size_t)n;  // row lower bounds (original order) and per-half screen bounds
    b += 8 * (size_t)(L.n_pad / 32);  // label ranges of gathered rows
    if (!lean && n >= LIST_MIN_ROWS && L.n_tiles <= kMaxVisitTiles)  // balls, thresholds, lists of tiles
        b += 2 * (size_t)L.n_qblocks * (4 * (size_t)d + 8 + (size_t)L.n_tiles + 2);
    return b;
}

// prep_rows_kernel over n_pad / 256 tiles in the fit's operand format.
static int tile_rows(cuscan_ctx *ctx, const RefinedBuffers &R, const float *x, int64_t n, int d,
                     int d_pad, int64_t n_pad, const int32_t *rowmap, uint8_t *xt, float *pnorm,
                     float *mnorm, cudaStream_t s, float *tile_mmax = nullptr,
                     const int32_t *label = nullptr, int32_t *chunk_lo = nullptr,
                     int32_t *chunk_hi = nullptr, int32_t *tile_lo = nullptr,
                     int32_t *tile_hi = nullptr) {
    const unsigned tiles = (unsigned)(n_pad / BN);
    const int vec4 = d % 4 == 0 && reinterpret_cast<uintptr_t>(x) % 16 == 0;  // aligned rows
    if (R.fp16)
        CUSCAN_KERNEL(prep_rows_kernel<FMT_FP16>, tiles, PREP_THREADS, 0, s, x, n, d, d_pad, R.scale,
                      rowmap, vec4, xt, pnorm, mnorm, tile_mmax, label, chunk_lo, chunk_hi, tile_lo,
                      tile_hi);
    else if (R.split)
        CUSCAN_KERNEL(prep_rows_kernel<FMT_SPLIT>, tiles, PREP_THREADS, 0, s, x, n, d, d_pad, 1.0f,
                      rowmap, vec4, xt, pnorm, mnorm, tile_mmax, label, chunk_lo, chunk_hi, tile_lo,
                      tile_hi);
    else
        CUSCAN_KERNEL(prep_rows_kernel<FMT_BF16>, tiles, PREP_THREADS, 0, s, x, n, d, d_pad, 1.0f,
                      rowmap, vec4, xt, pnorm, mnorm, tile_mmax, label, chunk_lo, chunk_hi, tile_lo,
                      tile_hi);
    CUSCAN_LAUNCH(ctx, "prep_rows_kernel");
    return CUSCAN_OK;
}

// Tiles, norms and statistics of the reference rows; with labels, their chunk and tile ranges.
static int prep(cuscan_ctx *ctx, RefinedBuffers &R, const Layout &L, const float *x, int64_t n,
                int d, const int32_t *label, int32_t *chunk_lo, int32_t *chunk_hi,
                cudaStream_t s) {
    int rc = ensure(ctx, R.xt, (size_t)L.n_tiles * L.nbk * KBLOCK_B, "16-bit tiles");
    if (!rc) rc = ensure(ctx, R.pnorm, sizeof(float) * L.n_pad, "norms");
    if (!rc) rc = ensure(ctx, R.mnorm, sizeof(float) * L.n_pad, "norms");
    if (!rc) rc = ensure(ctx, R.tile_mmax, sizeof(float) * L.n_tiles, "tile norms");
    if (!rc) rc = ensure(ctx, R.tile_lo, sizeof(int32_t) * L.n_tiles, "tile labels");
    if (!rc) rc = ensure(ctx, R.tile_hi, sizeof(int32_t) * L.n_tiles, "tile labels");
    if (!rc) rc = ensure(ctx, R.error, sizeof(int) * SCREEN_STATUS_WORDS, "screen status");
    if (!rc) rc = ensure(ctx, R.cursor, 16, "tile cursor");
    if (!rc) rc = ensure(ctx, R.fallback, sizeof(int32_t) * n, "fallback rows");
    if (!rc) rc = ensure(ctx, R.qthr, sizeof(float) * n, "fallback thresholds");
    if (rc) return rc;
    return tile_rows(ctx, R, x, n, d, L.d_pad, L.n_pad, nullptr, as<uint8_t>(R.xt),
                     as<float>(R.pnorm), as<float>(R.mnorm), s, as<float>(R.tile_mmax), label,
                     chunk_lo, chunk_hi, as<int32_t>(R.tile_lo), as<int32_t>(R.tile_hi));
}

// Operand format of this fit's screens: fp16 of x * scale when the caller asked for it and the
// data's range admits a power-of-two scale, else bf16. One reduction and one host read per fit.
// Largest d * max|x|^2 for which the screens stay exact: squared norms, dot products, bounds
// and every exact squared distance (at most 4 d max|x|^2) then stay below FLT_MAX / 4. Above it
// an f32 quantity may overflow: a bound may become NaN, and exact weights may tie at +inf,
// where the reference breaks the ties among ALL overflowing pairs, which bounds cannot narrow.
constexpr double kScreenRangeMax = 3.4028234663852886e38 / 16.0;

// Per fit: the largest |x| (one reduction and one host read) decides whether the screens may run
// (range_ok) and, when fp16 operands are wanted, their power-of-two scale.
static void set_operands(RefinedBuffers &R, int d, unsigned int absmax_bits) {
    R.fp16 = false;
    R.split = false;
    R.scale = 1.0f;
    float amax;
    memcpy(&amax, &absmax_bits, sizeof(amax));
    R.range_ok = std::isfinite(amax) && (double)d * (double)amax * (double)amax <= kScreenRangeMax;
    R.amax_value = std::isfinite(amax) ? amax : 0.0f;
    if (R.want_fp16) {
        const float sc = fp16_scale(amax);
        if (sc > 0.0f) {
            R.fp16 = true;
            R.scale = sc;
        }
    }
    R.have_scale = true;
}
static int choose_operands(cuscan_ctx *ctx, RefinedBuffers &R, const float *x, int64_t n, int d,
                           cudaStream_t s) {
    if (R.have_scale) return CUSCAN_OK;
    int rc = ensure(ctx, R.absmax, 16, "range reduction");
    if (rc) return rc;
    CUSCAN_CUDA(ctx, cudaMemsetAsync(R.absmax.ptr, 0, sizeof(unsigned int), s));
    const int64_t count = n * (int64_t)d;
    int64_t blocks = ceil_div(count, 256);
    if (blocks > 8 * (int64_t)ctx->sm_count) blocks = 8 * (int64_t)ctx->sm_count;
    CUSCAN_KERNEL(absmax_kernel, (unsigned)blocks, 256, 0, s, x, count,
                  as<unsigned int>(R.absmax));
    CUSCAN_LAUNCH(ctx, "absmax_kernel");
    unsigned int bits = 0;
    CUSCAN_CUDA(ctx, cudaMemcpyAsync(&bits, R.absmax.ptr, sizeof(bits), cudaMemcpyDeviceToHost, s));
    CUSCAN_CUDA(ctx, cudaStreamSynchronize(s));
    set_operands(R, d, bits);
    return CUSCAN_OK;
}

// The same from what sort_by_cells left (one host read), and whether plain bf16 bounds are so loose
// against the cells' scales that a first screen with them would only be thrown away: then `tight`
// is set and the screens start with the tightened operands. The estimate only picks the order of
// attempts; its factor of two keeps data that passes (unit vectors of 128 features: half the
// limit) on plain bf16.
static int choose_operands_by_cells(cuscan_ctx *ctx, ForestBuffers &b, int64_t n, int d, int d_pad,
                                    int k, bool &tight, float &apart, cudaStream_t s) {
    RefinedBuffers &R = b.refined;
    float ca, cb, abs_c;
    error_coefficients(d, d_pad, FMT_BF16, 0.0f, ca, cb, abs_c);
    const double entries = 2.0 * KNN_LIST;
    const float gap = (float)(2.0 * (2.0 / d) * std::log(k < entries ? entries / k : 1.0));
    if (int rc = count_tight_rows(ctx, b, n, ca, gap, s)) return rc;
    unsigned int *words = reinterpret_cast<unsigned int *>(ctx->fit->host_words());
    CUSCAN_CUDA(ctx, cudaMemcpyAsync(words, R.norm_range.ptr, 5 * sizeof(unsigned int),
                                     cudaMemcpyDeviceToHost, s));
    CUSCAN_CUDA(ctx, cudaStreamSynchronize(s));
    set_operands(R, d, words[2]);
    tight = !R.fp16 && (double)words[3] > TIGHT_START * (double)n;
    float pairs;
    memcpy(&pairs, &words[4], sizeof(pairs));
    apart = (float)((double)pairs / ((double)n * (double)n));
    return CUSCAN_OK;
}

// Operand format of the current fit's screens.
static int operand_format(const RefinedBuffers &R) {
    return R.split ? FMT_SPLIT : R.fp16 ? FMT_FP16 : FMT_BF16;
}

// Operand format a refined fit ended with: 0 bf16, 1 fp16, 2 split bf16 (-1: no screen ran).
int refined_operand_format(const ForestBuffers &b) {
    return b.refined.tile_pairs == 0 ? -1 : operand_format(b.refined);
}

// A operand of a screen and the outputs of the kNN threshold mode; the defaults mean the
// reference rows themselves.
struct QuerySet {
    const uint8_t *xq = nullptr;
    const float *pq = nullptr, *mq = nullptr;
    int64_t nq = -1;
    const int32_t *qpos = nullptr;
    const int32_t *qchunk_lo = nullptr, *qchunk_hi = nullptr;
    const float *qthr = nullptr;
    int32_t *cand_ids = nullptr;
    int32_t *rowcnt = nullptr;
    float *rowlb = nullptr;  // one-sided Borůvka: per query row and half, the pair lower bound
};

// Parts of every query block's tile order in a one-sided Borůvka screen. The blocks run in waves of one
// per SM; a last wave that is nearly empty, or a round of few blocks, leaves SMs idle. The count is the
// one whose waves take the least, a part costing its tiles and PART_START more (its A tile, the
// pipeline's start, bounds that start anew), with parts of at least PART_MIN tiles. Splitting only
// rounds of fewer blocks than SMs, a 50,000 x 128 fit took 3.96 ms and now takes 3.63 ms, 9,001 x 32
// 1.41 -> 1.27 ms, 100,000 x 64 8.90 -> 8.58 ms (parts of 16 tiles and a start of 6: 1.34 ms at 9,001
// rows, 3 and 3 no better than 6 and 4). A serving stream's p99 stays at 12.4 to 12.7 ms.
constexpr int64_t PART_MIN = 6, PART_START = 4;
static int screen_parts(int64_t blocks, int64_t tiles, int64_t sms) {
    int64_t most = tiles / PART_MIN < 16 ? tiles / PART_MIN : 16;
    if (blocks > 8 * sms) most = 1;  // the last wave is a small share
    int64_t best = 1, least = 0;
    for (int64_t s = 1; s <= most || s == 1; ++s) {
        const int64_t cost = ceil_div(blocks * s, sms) * (ceil_div(tiles, s) + PART_START);
        if (s == 1 || cost < least) {
            least = cost;
            best = s;
        }
    }
    return (int)best;
}

template <int M, int MODE, bool LIST = false>
static int run_screen(cuscan_ctx *ctx, RefinedBuffers &R, const Layout &L, int64_t n, int d,
                      const float *core, const int32_t *label, const int32_t *chunk_lo,
                      const int32_t *chunk_hi, cudaStream_t s, float *debug_tile = nullptr,
                      float *debug_chunk = nullptr,
                      const QuerySet &Q = QuerySet()) {
    constexpr bool BORUVKA = MODE == MODE_BORUVKA || MODE == MODE_BORUVKA_SYM;
    int rc = ensure(ctx, R.cand_ids, sizeof(int32_t) * n * 2 * M, "screen candidates");
    if (!rc && MODE == MODE_KNN_LIST)  // the lists; other forms append candidates without bounds
        rc = ensure(ctx, R.cand_lb, sizeof(float) * n * 2 * M, "screen bounds");
    if (rc) return rc;
    Params P{};
    P.xt = as<uint8_t>(R.xt);
    P.pnorm = as<float>(R.pnorm);
    P.mnorm = as<float>(R.mnorm);
    P.xq = Q.xq ? Q.xq : P.xt;
    P.pq = Q.pq ? Q.pq : P.pnorm;
    P.mq = Q.mq ? Q.mq : P.mnorm;
    P.nq = Q.nq >= 0 ? Q.nq : n;
    P.qpos = Q.qpos;
    P.qchunk_lo = Q.qchunk_lo;
    P.qchunk_hi = Q.qchunk_hi;
    P.qthr = Q.qthr;
    P.core = core;
    P.label = label;
    P.tile_mmax = as<float>(R.tile_mmax);
    P.chunk_lo = chunk_lo;
    P.chunk_hi = chunk_hi;
    P.tile_lo = as<int32_t>(R.tile_lo);
    P.tile_hi = as<int32_t>(R.tile_hi);
    P.n = n;
    P.n_tiles = L.n_tiles;
    P.n_qblocks = ceil_div(P.nq, (int64_t)BM);
    P.n_chunks = ceil_div(n, 32);
    P.kblocks = L.kblocks;
    P.nbk = L.nbk;
    P.split = L.split;
    P.stages = L.stages;
    P.stage_blocks = L.stage_blocks;
    P.cursor = as<unsigned long long>(R.cursor);
    P.vis = reinterpret_cast<const uint16_t *>(R.vis.ptr);
    P.vis_count = as<int32_t>(R.vis_count);
    P.splits = 1;
    if (MODE == MODE_BORUVKA && P.n_qblocks > 0 && !debug_tile)
        P.splits = screen_parts(P.n_qblocks, P.n_tiles, ctx->sm_count);
    float ca, cb, abs_c;
    error_coefficients(d, L.d_pad, operand_format(R), R.fp16 ? R.amax_value * R.scale : R.amax_value, ca, cb, abs_c);
    P.c_a = ca;
    P.one_minus_cb = 1.0f - cb;
    P.abs_c = abs_c;
    P.idesc = R.fp16 ? IDESC_F16 : IDESC_BF16;
    const float sc = R.fp16 ? R.scale : 1.0f;
    P.s2 = sc * sc;
    P.inv_s2 = 1.0f / (sc * sc);
    P.cand_ids = as<int32_t>(R.cand_ids);
    P.cand_lb = as<float>(R.cand_lb);
    P.error = as<int>(R.error);
    P.debug_tile = debug_tile;
    P.debug_chunk = debug_chunk;
    P.c_b = cb;
    P.cap = BORUVKA_CAP;
    if (BORUVKA) {
        rc = ensure(ctx, R.cbound, sizeof(uint32_t) * n, "component bounds");
        if (!rc) rc = ensure(ctx, R.rowcnt, sizeof(int32_t) * 2 * n, "row candidate counts");
        if (rc) return rc;
        P.cbound = as<uint32_t>(R.cbound);
        P.rowcnt = as<int32_t>(R.rowcnt);
    }
    if (MODE == MODE_BORUVKA_SYM) {
        P.urow = as<uint32_t>(R.urow);
        P.colcnt = as<int32_t>(R.colcnt);
        P.colbuf = as<int32_t>(R.colbuf);
        P.capc = BORUVKA_COL_CAP;
    }
    if (MODE == MODE_BORUVKA) P.rowlb = Q.rowlb;
    if (MODE == MODE_KNN_THRESHOLD) {
        P.cap = KNN_CAP;
        P.cand_ids = Q.cand_ids;
        P.rowcnt = Q.rowcnt;
    }
    if (P.n_qblocks == 0) return CUSCAN_OK;
    // the column terms of this launch (its C_B and, for Borůvka, the core scale)
    if (int rc = ensure(ctx, R.colp, sizeof(float) * L.n_pad, "screen column norms")) return rc;
    if (BORUVKA)
        if (int rc = ensure(ctx, R.colc, sizeof(float) * L.n_pad, "screen column cores")) return rc;
    if (int rc = ensure(ctx, R.cmin, sizeof(float) * L.n_pad / 16, "screen chunk minima")) return rc;
    P.colp = as<float>(R.colp);
    P.colc = BORUVKA ? as<float>(R.colc) : nullptr;
    P.cmin = as<float4>(R.cmin);
    CUSCAN_KERNEL(screen_columns_kernel, (unsigned)(L.n_pad / 256), 256, 0, s, P.pnorm,
                  BORUVKA ? core : nullptr, n, P.one_minus_cb, P.s2, as<float>(R.colp),
                  BORUVKA ? as<float>(R.colc) : nullptr, as<float2>(R.cmin), P.error, P.cursor,
                  BORUVKA ? reinterpret_cast<int2 *>(P.rowcnt) : nullptr,
                  P.splits > 1 ? reinterpret_cast<float2 *>(P.rowlb) : nullptr, P.nq);
    CUSCAN_LAUNCH(ctx, "screen_columns_kernel");
    auto kernel = screen_kernel<M, MODE, LIST>;
    if (int rc = allow_dynamic_smem(ctx, kernel, L.smem)) return rc;
    const int64_t items = P.n_qblocks * P.splits;
    int64_t grid = items < ctx->sm_count ? items : ctx->sm_count;
    CUSCAN_KERNEL(kernel, (unsigned)grid, THREADS, L.smem, s, P);
    CUSCAN_LAUNCH(ctx, "screen_kernel");
    return CUSCAN_OK;
}

static int read_screen_status(cuscan_ctx *ctx, RefinedBuffers &R, cudaStream_t s, int &fallbacks) {
    static_assert(SCREEN_STATUS_WORDS <= FitWorkspace::kHostWords, "pinned words");
    int *status = ctx->fit->host_words();
    CUSCAN_CUDA(ctx, cudaMemcpyAsync(status, R.error.ptr, sizeof(int) * SCREEN_STATUS_WORDS,
                                     cudaMemcpyDeviceToHost, s));
    CUSCAN_CUDA(ctx, cudaStreamSynchronize(s));
    if (status[0])
        return fail(ctx, CUSCAN_BACKEND_UNAVAILABLE,
                    "tensor-core screening timed out waiting on a pipeline barrier");
    unsigned long long tiles;
    memcpy(&tiles, status + 2, sizeof(tiles));
    R.tile_pairs += (int64_t)tiles;
    fallbacks = status[STATUS_FALLBACKS];
    return CUSCAN_OK;
}

// The kNN list screen over every row in sorted positions and its exact re-rank. Rows whose
// lists are inconclusive are listed by position in R.fallback, with the k-th exact distance
// among their candidates in R.qthr; returns their count.
static int knn_list_pass(cuscan_ctx *ctx, RefinedBuffers &R, const Layout &L, const float *xs,
                         const int32_t *perm, int64_t n, int d, int k, int32_t *ids, float *dist,
                         cudaStream_t s, int &fallbacks) {
    // 22 bounds per row half: enough that nearly every row's unseen bound clears its k-th
    // exact distance at k <= 32 for bf16 screens (the rest go to the threshold re-screen), and
    // each insertion shifts 22 registers; 20 and 24 entries measured slower
    constexpr int M = KNN_LIST;
    if (int rc = prep(ctx, R, L, xs, n, d, nullptr, nullptr, nullptr, s)) return rc;
    for (cudaEvent_t &e : R.screen_ev)
        if (!e) CUSCAN_CUDA(ctx, cudaEventCreate(&e));
    CUSCAN_CUDA(ctx, cudaEventRecord(R.screen_ev[0], s));
    const int rc = R.listed
                       ? run_screen<M, MODE_KNN_LIST, true>(ctx, R, L, n, d, nullptr, nullptr, nullptr,
                                                            nullptr, s)
                       : run_screen<M, MODE_KNN_LIST>(ctx, R, L, n, d, nullptr, nullptr, nullptr,
                                                      nullptr, s);
    if (rc) return rc;
    CUSCAN_CUDA(ctx, cudaEventRecord(R.screen_ev[1], s));
    R.screen_timed = true;
    const bool vec = rerank_vec(xs, d);
    const size_t rr_smem = sizeof(float) * RERANK_WARPS * (size_t)rerank_warp_floats(d, vec);
    const auto rerank = vec ? rerank_knn_kernel<M, true> : rerank_knn_kernel<M, false>;
    if (int rc = allow_dynamic_smem(ctx, rerank, rr_smem)) return rc;
    CUSCAN_KERNEL(rerank, (unsigned)ceil_div(n, (int64_t)RERANK_WARPS),
                  32 * RERANK_WARPS, rr_smem, s, xs, perm, n, d,
                  k, as<int32_t>(R.cand_ids), as<float>(R.cand_lb), ids, dist,
                  as<int32_t>(R.fallback), as<float>(R.qthr), as<int>(R.error) + STATUS_FALLBACKS);
    CUSCAN_LAUNCH(ctx, "rerank_knn_kernel");
    return read_screen_status(ctx, R, s, fallbacks);
}

// Whether there was something to release.
static bool release_lists(RefinedBuffers &R) {
    bool held = false;
    for (Buffer *b : {&R.ball_thr, &R.vis, &R.vis_count, &R.tile_centre, &R.tile_radius}) {
        held |= b->ptr != nullptr;
        release(*b);
    }
    R.listed = false;
    return held;
}

static int knn_refined(cuscan_ctx *ctx, ForestBuffers &b, const float *x, int64_t n, int d, int k,
                       int32_t *ids, float *dist, cudaStream_t s, int64_t *refined_rows,
                       int64_t *fallback_rows, int64_t *rescreened_rows) {
    if (!refined_shape_ok(n, d, k) || (b.refined.lean && lean_exact(d, k))) {
        // shapes outside the tensor-core tiling run the exact f32 sweep
        return launch_exact_knn_fp32(ctx, x, n, x, n, d, k, 1, 0, 1, ids, dist, s, b.knn_ids_tmp,
                                     b.knn_dist_tmp);
    }
    RefinedBuffers &R = b.refined;
    R.listed = false;
    Layout L;
    refined_layout(n, d, L);
    // 1, 2. rows in spatial order (b.perm, b.xp), and the screens' operands
    bool tight = false;
    float apart = 0.0f;
    int rc = sort_by_cells(ctx, b, x, n, d, s);
    if (!rc) rc = choose_operands_by_cells(ctx, b, n, d, L.d_pad, k, tight, apart, s);
    if (rc) return rc;
    if (!R.range_ok)  // values large enough to overflow f32: the exact sweep decides alone
        return launch_exact_knn_fp32(ctx, x, n, x, n, d, k, 1, 0, 1, ids, dist, s, b.knn_ids_tmp,
                                     b.knn_dist_tmp);
    R.pivots_valid = true;
    if (!R.lean && !R.no_lists && n >= LIST_MIN_ROWS && L.n_tiles <= kMaxVisitTiles && apart > LIST_MIN_APART) {
        if ((rc = visit_lists(ctx, b, n, d, k, s)) && rc != CUSCAN_MEMORY) return rc;
        R.listed = rc == CUSCAN_OK;  // without room for the lists every tile is visited
        if (rc) {
            release_lists(R);
            clear_error(ctx);
        }
    }
    // the tightened operands: split bf16, or scaled fp16 for rows too wide to split
    auto tighten = [&]() {
        Layout Ls;
        const float sc = fp16_scale(R.amax_value);
        if (refined_layout(n, d, Ls, true)) {
            R.split = true;
            L = Ls;
        } else if (sc > 0.0f) {
            R.fp16 = true;
            R.scale = sc;
        }
    };
    if (tight) tighten();
    const float *xs = as<float>(b.xp);
    const int32_t *perm = as<int32_t>(b.perm);
    // 3. screen + exact re-rank in sorted positions, outputs in original rows
    int fallbacks = 0;
    if ((rc = knn_list_pass(ctx, R, L, xs, perm, n, d, k, ids, dist, s, fallbacks))) return rc;
    if (refined_rows) *refined_rows += n;
    if (!R.fp16 && !R.split && (double)fallbacks > TIGHTEN_TRIGGER * (double)n) {
        // the bf16 bound is too loose for this data (norms large against the neighbour
        // distances): screen again, and run the Borůvka rounds, with the tightened operands
        tighten();
        if (R.split || R.fp16)
            if ((rc = knn_list_pass(ctx, R, L, xs, perm, n, d, k, ids, dist, s, fallbacks)))
                return rc;
    }
    if (fallbacks == 0) return CUSCAN_OK;
    constexpr int M = KNN_LIST;
    const bool vec = rerank_vec(xs, d);
    const size_t rr_smem = sizeof(float) * RERANK_WARPS * (size_t)rerank_warp_floats(d, vec);
    const auto rerank = vec ? rerank_knn_threshold_kernel<true> : rerank_knn_threshold_kernel<false>;
    int32_t *exact_rows = as<int32_t>(R.fallback);
    int exact = fallbacks;
    if (fallbacks >= RESCREEN_MIN_ROWS && k <= 2 * KNN_CAP) {
        // 4. inconclusive rows, screened again in threshold mode: every pair whose bound does
        // not exceed the row's k-th distance among its candidates is appended and re-ranked
        const int64_t nq = fallbacks;
        const int64_t nq_pad = ceil_div(nq, (int64_t)BN) * BN;
        rc = ensure(ctx, R.xq, (size_t)(nq_pad / BN) * L.nbk * KBLOCK_B, "re-screen tiles");
        if (!rc) rc = ensure(ctx, R.pq, sizeof(float) * nq_pad, "re-screen norms");
        if (!rc) rc = ensure(ctx, R.mq, sizeof(float) * nq_pad, "re-screen norms");
        if (!rc) rc = ensure(ctx, R.cand2, sizeof(int32_t) * nq * 2 * KNN_CAP, "re-screen candidates");
        if (!rc) rc = ensure(ctx, R.rowcnt2, sizeof(int32_t) * nq * 2, "re-screen counts");
        if (!rc) rc = ensure(ctx, R.fallback2, sizeof(int32_t) * nq, "re-screen fallbacks");
        if (!rc) rc = tile_rows(ctx, R, xs, nq, d, L.d_pad, nq_pad, as<int32_t>(R.fallback),
                                as<uint8_t>(R.xq), as<float>(R.pq), as<float>(R.mq), s);
        if (rc) return rc;
        QuerySet Q;
        Q.xq = as<uint8_t>(R.xq);
        Q.pq = as<float>(R.pq);
        Q.mq = as<float>(R.mq);
        Q.nq = nq;
        Q.qpos = as<int32_t>(R.fallback);
        Q.qthr = as<float>(R.qthr);
        Q.cand_ids = as<int32_t>(R.cand2);
        Q.rowcnt = as<int32_t>(R.rowcnt2);
        if ((rc = run_screen<M, MODE_KNN_THRESHOLD>(ctx, R, L, n, d, nullptr, nullptr, nullptr,
                                                   nullptr, s, nullptr, nullptr, Q)))
            return rc;
        if ((rc = allow_dynamic_smem(ctx, rerank, rr_smem))) return rc;
        CUSCAN_KERNEL(rerank, (unsigned)ceil_div(nq, (int64_t)RERANK_WARPS),
                      32 * RERANK_WARPS, rr_smem, s, xs,
                      perm, as<int32_t>(R.fallback), nq, d, k, as<int32_t>(R.cand2),
                      as<int32_t>(R.rowcnt2), KNN_CAP, ids, dist, as<int32_t>(R.fallback2),
                      as<int>(R.error) + STATUS_FALLBACKS);
        CUSCAN_LAUNCH(ctx, "rerank_knn_threshold_kernel");
        if ((rc = read_screen_status(ctx, R, s, exact))) return rc;
        if (rescreened_rows) *rescreened_rows += fallbacks;
        exact_rows = as<int32_t>(R.fallback2);
    } else {
        CUSCAN_KERNEL(positions_to_rows_kernel, (unsigned)ceil_div((int64_t)fallbacks, 256), 256, 0,
                      s, exact_rows, (int64_t)fallbacks, perm);
        CUSCAN_LAUNCH(ctx, "positions_to_rows_kernel");
    }
    if (fallback_rows) *fallback_rows += exact;
    // 5. rows still inconclusive (original indices): exact f32 sweep
    if (exact > 0)
        return launch_exact_knn_fp32(ctx, x, exact, x, n, d, k, 1, 0, 1, ids, dist, s,
                                     b.knn_ids_tmp, b.knn_dist_tmp, exact_rows);
    return CUSCAN_OK;
}

// Lists of tiles are given up where the screens' own buffers have no room beside them. Wide rows take
// more device memory on the screens than in the exact sweeps: without room for it the fit goes on with
// those.
int launch_knn_refined(cuscan_ctx *ctx, ForestBuffers &b, const float *x, int64_t n, int d, int k,
                       int32_t *ids, float *dist, cudaStream_t s, int64_t *refined_rows,
                       int64_t *fallback_rows, int64_t *rescreened_rows) {
    b.refined.no_room = false;
    b.refined.no_lists = false;
    auto screens = [&]() {
        for (int64_t *rows : {refined_rows, fallback_rows, rescreened_rows})
            if (rows) *rows = 0;
        return knn_refined(ctx, b, x, n, d, k, ids, dist, s, refined_rows, fallback_rows,
                           rescreened_rows);
    };
    int rc = screens();
    if (rc == CUSCAN_MEMORY && release_lists(b.refined)) {
        clear_error(ctx);
        b.refined.no_lists = true;
        rc = screens();
    }
    if (rc != CUSCAN_MEMORY || d <= LEAN_MAX_FEATURES) return rc;
    clear_error(ctx);
    b.refined.no_room = true;
    forest_release_refined(b);
    for (int64_t *rows : {refined_rows, fallback_rows, rescreened_rows})
        if (rows) *rows = 0;
    return launch_exact_knn_fp32(ctx, x, n, x, n, d, k, 1, 0, 1, ids, dist, s, b.knn_ids_tmp,
                                 b.knn_dist_tmp);
}

static int candidates_refined(cuscan_ctx *ctx, ForestBuffers &b, int64_t n, int d,
                              const int32_t *knn_ids, const float *knn_sq, int k,
                              const float *core, const int32_t *label, cudaStream_t s,
                              int64_t *fallback_rows) {
    const float *xp = as<float>(b.xp);
    const float *corep = as<float>(b.corep);
    const int32_t *labp = as<int32_t>(b.labp);
    const int32_t *perm = as<int32_t>(b.perm);
    unsigned long long *row_keys = as<unsigned long long>(b.row_keys);
    int32_t *clo = as<int32_t>(b.tile_lo), *chi = as<int32_t>(b.tile_hi);
    if (!refined_shape_ok(n, d, 1) || b.refined.no_room || (b.refined.lean && lean_exact(d, k)))
        return launch_candidates_fp32(ctx, xp, corep, labp, perm, n, d, row_keys, clo, chi, s);
    RefinedBuffers &R = b.refined;
    Layout L;
    refined_layout(n, d, L, R.split != 0);
    int rc = choose_operands(ctx, R, xp, n, d, s);
    if (rc) return rc;
    if (!R.range_ok)  // values large enough to overflow f32: the exact round decides alone
        return launch_candidates_fp32(ctx, xp, corep, labp, perm, n, d, row_keys, clo, chi, s);
    if ((rc = prep(ctx, R, L, xp, n, d, labp, clo, chi, s))) return rc;
    // component bounds: +inf, then the exact cross-component edges of the kNN rows. Symmetric
    // screen: per-row bounds start at the component bounds; empty column buffers
    if ((rc = ensure(ctx, R.cbound, sizeof(uint32_t) * n, "component bounds"))) return rc;
    if ((rc = ensure(ctx, R.urow, sizeof(uint32_t) * n, "row bounds"))) return rc;
    if ((rc = ensure(ctx, R.colcnt, sizeof(int32_t) * n, "column-side counts"))) return rc;
    if ((rc = ensure(ctx, R.colbuf, sizeof(int32_t) * n * BORUVKA_COL_CAP, "column-side candidates")))
        return rc;
    rc = ensure(ctx, R.act_flag, sizeof(int32_t) * n, "active rows");
    if (!rc) rc = ensure(ctx, R.act_idx, sizeof(int32_t) * n, "active rows");
    if (!rc) rc = ensure(ctx, R.act_pos, sizeof(int32_t) * n, "active rows");
    if (!rc) rc = ensure(ctx, R.rowlb, sizeof(float) * n, "row lower bounds");
    if (!rc) rc = ensure(ctx, R.lbtmp, sizeof(float) * 2 * n, "row lower bounds");
    if (rc) return rc;
    CUSCAN_KERNEL(round_clear_kernel, (unsigned)ceil_div(n, 256), 256, 0, s, as<uint32_t>(R.cbound),
                  as<int32_t>(R.colcnt), R.lb_valid ? nullptr : as<float>(R.rowlb),
                  b.status->row_counts, n);
    R.lb_valid = true;
    CUSCAN_KERNEL(seed_bounds_kernel, (unsigned)ceil_div(n, 256), 256, 0, s, knn_ids, knn_sq, k,
                  core, label, n, as<uint32_t>(R.cbound));
    // a late component's neighbours are all its own: the pivots bound it (without a bound every
    // row of it is screened, and every pair appended until the first blocks have found one)
    if (R.pivots_valid &&
        (rc = pivot_component_bounds(ctx, b, n, core, label, as<uint32_t>(R.cbound), s)))
        return rc;
    CUSCAN_KERNEL(init_row_bounds_kernel, (unsigned)ceil_div(n, 256), 256, 0, s,
                  as<uint32_t>(R.cbound), labp, corep, as<float>(R.rowlb), perm, n,
                  as<uint32_t>(R.urow), b.status->row_counts, as<int32_t>(R.act_flag));
    CUSCAN_LAUNCH(ctx, "init_row_bounds_kernel");
    if ((rc = scan_exclusive(ctx, b, as<int32_t>(R.act_flag), as<int32_t>(R.act_idx), n,
                             b.status->row_counts + 1, s)))
        return rc;
    const DevStatus *hs = ctx->fit->host_status;
    CUSCAN_CUDA(ctx, cudaMemcpyAsync(ctx->fit->host_status, b.status, sizeof(DevStatus),
                                     cudaMemcpyDeviceToHost, s));
    CUSCAN_CUDA(ctx, cudaStreamSynchronize(s));
    const int unbounded = hs->row_counts[0];
    const double same_pairs = hs->same_pairs;
    const int64_t active = hs->row_counts[1];
    // Gathered blocks look for tiles of their own component only where components hold a fair share
    // of the pairs: the look costs every tile two loads in each role (4 % of a round at 500,000 x 128,
    // where 1 to 2 % of the tiles could go; at 100,000 x 64 rounds 3 and 4 run 12 % and 51 % fewer
    // tiles, 6.1 -> 5.3 ms over the fit's screens).
    const bool skip_own = same_pairs > 0.06 * (double)n * (double)n;
    // Forms of the round:
    //  * one-sided over the rows that can hold their component's cheapest edge (all rows, or a
    //    gathered subset): it also leaves each screened row a lower bound of its cheapest cross
    //    edge, which lets most rows skip the later rounds. After the kNN seed most components
    //    have a bound from a neighbour in another component and few rows are that close to the
    //    boundary; later rounds skip the rows whose earlier bound already exceeds the bound.
    //  * symmetric: each unordered pair once. It halves the tensor-core and epilogue work but
    //    leaves no row bounds and tests a pair for its column's row only against that row's
    //    known bound (rows of components without a bound draw many appends there); it is used
    //    only when nearly every row is screened.
    const bool sym = n >= SYM_MIN_ROWS &&
                     (double)unbounded <= SYM_UNBOUNDED_MAX * (double)n &&
                     (double)active > SYM_ACTIVE_MIN * (double)n;
    const bool subset = !sym && active < n;
    CUSCAN_LAUNCH(ctx, "component bounds");
    constexpr int M = 32;
    const int32_t *qpos = nullptr;
    int64_t nq = n;
    if (subset) {
        nq = active;
        const int64_t nq_pad = ceil_div(nq > 0 ? nq : 1, (int64_t)BN) * BN;
        rc = ensure(ctx, R.xq, (size_t)(nq_pad / BN) * L.nbk * KBLOCK_B, "subset tiles");
        if (!rc) rc = ensure(ctx, R.pq, sizeof(float) * nq_pad, "subset norms");
        if (!rc) rc = ensure(ctx, R.mq, sizeof(float) * nq_pad, "subset norms");
        if (rc) return rc;
        CUSCAN_KERNEL(compact_positions_kernel, (unsigned)ceil_div(n, 256), 256, 0, s,
                      as<int32_t>(R.act_flag), as<int32_t>(R.act_idx),
                      as<int32_t>(b.scan_tmp), n, as<int32_t>(R.act_pos));
        CUSCAN_LAUNCH(ctx, "compact_positions_kernel");
        qpos = as<int32_t>(R.act_pos);
        rc = ensure(ctx, R.qchunk_lo, sizeof(int32_t) * (nq_pad / 32), "subset labels");
        if (!rc) rc = ensure(ctx, R.qchunk_hi, sizeof(int32_t) * (nq_pad / 32), "subset labels");
        if (!rc)
            rc = tile_rows(ctx, R, xp, nq, d, L.d_pad, nq_pad, qpos, as<uint8_t>(R.xq),
                           as<float>(R.pq), as<float>(R.mq), s, nullptr, skip_own ? labp : nullptr,
                           as<int32_t>(R.qchunk_lo), as<int32_t>(R.qchunk_hi));
        if (rc) return rc;
        QuerySet Q;
        Q.xq = as<uint8_t>(R.xq);
        Q.pq = as<float>(R.pq);
        Q.mq = as<float>(R.mq);
        Q.nq = nq;
        Q.qpos = qpos;
        Q.qchunk_lo = skip_own ? as<int32_t>(R.qchunk_lo) : nullptr;
        Q.qchunk_hi = skip_own ? as<int32_t>(R.qchunk_hi) : nullptr;
        Q.rowlb = as<float>(R.lbtmp);
        rc = run_screen<M, MODE_BORUVKA>(ctx, R, L, n, d, corep, labp, clo, chi, s, nullptr, nullptr, Q);
    } else if (sym) {
        rc = run_screen<M, MODE_BORUVKA_SYM>(ctx, R, L, n, d, corep, labp, clo, chi, s);
    } else {
        QuerySet Q;
        Q.rowlb = as<float>(R.lbtmp);
        rc = run_screen<M, MODE_BORUVKA>(ctx, R, L, n, d, corep, labp, clo, chi, s, nullptr, nullptr, Q);
    }
    if (rc) return rc;
    R.screened_rows += nq;
    if (sym) ++R.symmetric_rounds;
    const bool vec = rerank_vec(xp, d);
    const size_t rr_smem = sizeof(float) * RERANK_WARPS * (size_t)rerank_warp_floats(d, vec);
    const auto rerank = vec ? rerank_boruvka_kernel<true> : rerank_boruvka_kernel<false>;
    if ((rc = allow_dynamic_smem(ctx, rerank, rr_smem))) return rc;
    if (nq > 0) {
        CUSCAN_KERNEL(rerank, (unsigned)ceil_div(nq, (int64_t)RERANK_WARPS),
                      32 * RERANK_WARPS, rr_smem, s, xp, corep, labp, perm, nq, qpos, d,
                      as<int32_t>(R.cand_ids), as<int32_t>(R.rowcnt), BORUVKA_CAP,
                      sym ? as<int32_t>(R.colcnt) : nullptr, as<int32_t>(R.colbuf),
                      BORUVKA_COL_CAP, sym ? nullptr : as<float>(R.lbtmp), as<float>(R.rowlb),
                      row_keys, as<int32_t>(R.fallback), as<int>(R.error) + STATUS_FALLBACKS);
        CUSCAN_LAUNCH(ctx, "rerank_boruvka_kernel");
    }
    int fallbacks = 0;
    if (nq > 0 && (rc = read_screen_status(ctx, R, s, fallbacks))) return rc;
    if (fallback_rows) *fallback_rows += fallbacks;
    if (fallbacks > 0)
        return launch_candidates_fp32(ctx, xp, corep, labp, perm, n, d, row_keys, clo, chi, s,
                                      as<int32_t>(R.fallback), fallbacks, 0, true);
    return CUSCAN_OK;
}

// As launch_knn_refined: every buffer of a round is there before its first kernel writes a key.
int launch_candidates_refined(cuscan_ctx *ctx, ForestBuffers &b, int64_t n, int d,
                              const int32_t *knn_ids, const float *knn_sq, int k,
                              const float *core, const int32_t *label, cudaStream_t s,
                              int64_t *fallback_rows) {
    int rc = candidates_refined(ctx, b, n, d, knn_ids, knn_sq, k, core, label, s, fallback_rows);
    if (rc == CUSCAN_MEMORY && release_lists(b.refined)) {
        clear_error(ctx);
        rc = candidates_refined(ctx, b, n, d, knn_ids, knn_sq, k, core, label, s, fallback_rows);
    }
    if (rc == CUSCAN_MEMORY && d > LEAN_MAX_FEATURES) {
        clear_error(ctx);
        b.refined.no_room = true;
        b.refined.pivots_valid = false;
        forest_release_refined(b);
        rc = candidates_refined(ctx, b, n, d, knn_ids, knn_sq, k, core, label, s, fallback_rows);
    }
    return rc;
}

// Device memory of the exact rounds (a fit takes it before the spatial order, which it can do without).
int reserve_exact_rows(cuscan_ctx *ctx, ForestBuffers &b, int64_t n) {
    RefinedBuffers &R = b.refined;
    int rc = ensure(ctx, R.cbound, sizeof(uint32_t) * n, "component bounds");
    if (!rc) rc = ensure(ctx, R.urow, sizeof(uint32_t) * n, "row bounds");
    if (!rc) rc = ensure(ctx, R.act_flag, sizeof(int32_t) * n, "active rows");
    if (!rc) rc = ensure(ctx, R.act_idx, sizeof(int32_t) * n, "active rows");
    if (!rc) rc = ensure(ctx, R.act_pos, sizeof(int32_t) * n, "active rows");
    if (!rc) rc = ensure(ctx, R.rowlb, sizeof(float) * n, "row lower bounds");
    return rc;
}

// An exact (plain f32) Borůvka round over the rows that can hold their component's cheapest
// edge. The rows are chosen as in the screened rounds: every component gets an upper bound of
// its cheapest cross edge from the kNN pairs (seed_bounds_kernel), and a row is skipped when its
// core distance or its lower bound from earlier rounds exceeds that bound. Every cross edge of a
// skipped row then weighs strictly more than the component's cheapest, so the round's winners
// (crates/hdbscan/src/kernels/boruvka.rs:68-140 over all rows) are unchanged. The rows scanned
// leave their exact cheapest cross edge as their lower bound for the next round.
int launch_candidates_exact_rows(cuscan_ctx *ctx, ForestBuffers &b, int64_t n, int d,
                                 const int32_t *knn_ids, const float *knn_sq, int k,
                                 const float *core, const int32_t *label, cudaStream_t s,
                                 int64_t *screened_rows, const TileBounds *bounds) {
    const float *xp = as<float>(b.xp);
    const float *corep = as<float>(b.corep);
    const int32_t *labp = as<int32_t>(b.labp);
    const int32_t *perm = as<int32_t>(b.perm);
    unsigned long long *row_keys = as<unsigned long long>(b.row_keys);
    int32_t *clo = as<int32_t>(b.tile_lo), *chi = as<int32_t>(b.tile_hi);
    RefinedBuffers &R = b.refined;
    int rc = reserve_exact_rows(ctx, b, n);
    if (rc) return rc;
    if (!R.lb_valid) {  // first round of the fit: no bounds yet
        CUSCAN_CUDA(ctx, cudaMemsetAsync(R.rowlb.ptr, 0, sizeof(float) * n, s));
        R.lb_valid = true;
    }
    CUSCAN_KERNEL(fill_u32_kernel, (unsigned)ceil_div(n, 256), 256, 0, s, as<uint32_t>(R.cbound), n,
                  0x7f800000u);
    CUSCAN_KERNEL(seed_bounds_kernel, (unsigned)ceil_div(n, 256), 256, 0, s, knn_ids, knn_sq, k,
                  core, label, n, as<uint32_t>(R.cbound));
    // a component whose neighbours are all its own has no bound from them; in spatial order the
    // pivots give it one, and the walk something to beat
    if (bounds &&
        (rc = pivot_component_bounds(ctx, b, n, core, label, as<uint32_t>(R.cbound), s)))
        return rc;
    CUSCAN_CUDA(ctx, cudaMemsetAsync(b.status->row_counts, 0, 2 * sizeof(int), s));
    CUSCAN_KERNEL(init_row_bounds_kernel, (unsigned)ceil_div(n, 256), 256, 0, s,
                  as<uint32_t>(R.cbound), labp, corep, as<float>(R.rowlb), perm, n,
                  as<uint32_t>(R.urow), b.status->row_counts, as<int32_t>(R.act_flag));
    CUSCAN_LAUNCH(ctx, "component bounds");
    if ((rc = scan_exclusive(ctx, b, as<int32_t>(R.act_flag), as<int32_t>(R.act_idx), n,
                             b.status->row_counts + 1, s)))
        return rc;
    int *counts = ctx->fit->host_status->row_counts;
    CUSCAN_CUDA(ctx, cudaMemcpyAsync(counts, b.status->row_counts, 2 * sizeof(int),
                                     cudaMemcpyDeviceToHost, s));
    CUSCAN_CUDA(ctx, cudaStreamSynchronize(s));
    const int64_t active = counts[1];
    const int32_t *qpos = nullptr;
    const uint32_t *cbound = bounds ? as<uint32_t>(R.cbound) : nullptr;
    if (active == n) {
        rc = launch_candidates_fp32(ctx, xp, corep, labp, perm, n, d, row_keys, clo, chi, s, nullptr,
                                    0, 0, false, bounds, cbound);
    } else if (active > 0) {
        CUSCAN_KERNEL(compact_positions_kernel, (unsigned)ceil_div(n, 256), 256, 0, s,
                      as<int32_t>(R.act_flag), as<int32_t>(R.act_idx),
                      as<int32_t>(b.scan_tmp), n, as<int32_t>(R.act_pos));
        CUSCAN_LAUNCH(ctx, "compact_positions_kernel");
        qpos = as<int32_t>(R.act_pos);
        rc = launch_candidates_fp32(ctx, xp, corep, labp, perm, n, d, row_keys, clo, chi, s, qpos,
                                    active, 0, false, bounds, cbound);
    }
    if (rc) return rc;
    if (active > 0) {
        CUSCAN_KERNEL(row_lb_from_keys_kernel, (unsigned)ceil_div(active, 256), 256, 0, s, row_keys,
                      qpos, perm, active, labp, cbound, as<float>(R.rowlb));
        CUSCAN_LAUNCH(ctx, "row_lb_from_keys_kernel");
    }
    if (screened_rows) *screened_rows += active;
    return CUSCAN_OK;
}

// The per-row terms of the bound for the debug entry point: (ps, pb, cm, m) with
// ps = (1 - C_B) p - abs_c, pb = (1 - C_B) p, cm = C_A m, so that the screen's bound of entry
// (r, c) is fmaf(-cm_r, m_c, fmaf(-2, acc_rc, pb_c) + ps_r) (screen units).
__global__ void debug_rows_kernel(const float *__restrict__ pnorm, const float *__restrict__ mnorm,
                                  int64_t n, float one_minus_cb, float abs_c, float c_a,
                                  float *__restrict__ rows) {
    int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    const float p = pnorm[r], m = mnorm[r];
    rows[4 * r + 0] = one_minus_cb * p - abs_c;
    rows[4 * r + 1] = one_minus_cb * p;
    rows[4 * r + 2] = c_a * m;
    rows[4 * r + 3] = m;
}

int debug_screen_tile(cuscan_ctx *ctx, ForestBuffers &b, const float *x, int64_t n, int d,
                      int operands, float *out, float *rows_out, float *chunk_out,
                      float *scale_out, cudaStream_t s) {
    RefinedBuffers &R = b.refined;
    R.have_scale = false;
    R.want_fp16 = operands == FMT_FP16;
    int rc = choose_operands(ctx, R, x, n, d, s);
    if (rc) return rc;
    if (operands == FMT_FP16 && !R.fp16)
        return fail(ctx, CUSCAN_INVALID_INPUT, "no fp16 scale for this data");
    R.split = operands == FMT_SPLIT;
    Layout L;
    if (!refined_layout(n, d, L, R.split))
        return fail(ctx, CUSCAN_CAPACITY, "shape outside the tensor-core tiling%s",
                    R.split ? " (split copies need d <= 64)" : "");
    if (scale_out) *scale_out = R.fp16 ? R.scale : 1.0f;
    rc = prep(ctx, R, L, x, n, d, nullptr, nullptr, nullptr, s);
    if (!rc)
        rc = run_screen<32, MODE_KNN_LIST>(ctx, R, L, n, d, nullptr, nullptr, nullptr, nullptr, s,
                                           out, chunk_out);
    if (!rc && rows_out) {
        float ca, cb, abs_c;
        error_coefficients(d, L.d_pad, operand_format(R), R.fp16 ? R.amax_value * R.scale : R.amax_value, ca, cb, abs_c);
        CUSCAN_KERNEL(debug_rows_kernel, (unsigned)ceil_div(n, 256), 256, 0, s, as<float>(R.pnorm),
                      as<float>(R.mnorm), n, 1.0f - cb, abs_c, ca, rows_out);
        CUSCAN_LAUNCH(ctx, "debug_rows_kernel");
    }
    if (!rc) {
        int fallbacks = 0;
        rc = read_screen_status(ctx, R, s, fallbacks);
    }
    R.have_scale = false;
    R.split = false;
    R.fp16 = false;
    return rc;
}

}  // namespace cuscan
