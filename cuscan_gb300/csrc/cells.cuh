// Spatial order of a point set and tile bounds for pruning (cells.cu), and their use in the
// register-tiled sweeps.
#pragma once

#include "common.cuh"
#include "forest.cuh"
#include "simt.cuh"

namespace cuscan {

// Rows in spatial order: b.perm (position -> row) and b.xp (the rows in that order). The rows of
// a cell (nearest of at most 256 evenly spaced pivot rows) are contiguous, cells follow one another
// along a tour of their pivots, and rows far outside their cell's scale come last, so that the
// 128- and 256-row tiles of clustered data are compact. The toured pivots stay in
// b.refined.pivots. n >= 2048.
constexpr int kMaxPivots = 256;
inline int cell_pivots(int64_t n) {
    return (int)(n / 256 < kMaxPivots ? (n / 256 < 1 ? 1 : n / 256) : kMaxPivots);
}
int sort_by_cells(cuscan_ctx *ctx, ForestBuffers &b, const float *x, int64_t n, int d,
                  cudaStream_t s);
// Device bytes of sort_by_cells beyond the forest's own buffers.
inline size_t cells_workspace_bytes(int64_t n, int d) {
    const size_t npiv = (size_t)cell_pivots(n);
    return sizeof(float) * (2 * npiv * d + (npiv + 1) * npiv + 3 * kMaxPivots) + 32 +
           16 * (size_t)n;  // cells, distances, norms, keys
}
// Query orders for the pruned sweeps: the rows grouped by cell, every cell padded to whole balls of
// kBallRows entries with -1, so that no ball straddles two cells. A straddling ball is as wide as
// the gap between two clusters and visits every tile: at 40 clusters and 4,096 queries half of the
// 64-query tiles held one. order has padded_queries(m) entries.
constexpr int kBallRows = 16;
constexpr int64_t kMaxCells = 2 * kMaxPivots;
inline int64_t padded_queries(int64_t m) { return m + kMaxCells * (kBallRows - 1); }
// Of m rows outside the set, by their nearest of the npiv toured pivots.
int order_queries(cuscan_ctx *ctx, ForestBuffers &b, const float *pivots, int npiv, const float *q,
                  int64_t m, int d, int32_t *order, cudaStream_t s);
// Of the n positions of the set itself, right after sort_by_cells.
int order_positions(cuscan_ctx *ctx, ForestBuffers &b, int64_t n, int32_t *order, cudaStream_t s);
// Rows of cells whose scale times gap is below shift times the squared norm of their pivot, counted
// in word 3 of b.refined.norm_range, and in word 4 (f32) the pairs of rows in cells too far apart to be
// neighbours. Right after sort_by_cells.
int count_tight_rows(cuscan_ctx *ctx, ForestBuffers &b, int64_t n, float shift, float gap,
                     cudaStream_t s);
// The share of the n x n row pairs that lie in cells too far apart to be neighbours, read on the host.
// Right after sort_by_cells.
int read_apart(cuscan_ctx *ctx, ForestBuffers &b, int64_t n, float &apart, cudaStream_t s);
// cbound[label] (f32 bits, labels by original row) lowered to the weights of edges between pivots
// of different components. Needs sort_by_cells of the same fit.
int pivot_component_bounds(cuscan_ctx *ctx, ForestBuffers &b, int64_t n, const float *core,
                           const int32_t *label, uint32_t *cbound, cudaStream_t s);

// Bounds of the reference tiles (simt::RT rows) of a row-major set, a ball per half tile: centres
// feature-major, first halves then second halves ([d][PARTS][tiles], so that lanes read
// neighbouring tiles), and radii rounded up (-inf for a half without rows).
struct TileBounds {
    static constexpr int PARTS = 2;
    const float *centre = nullptr;  // null: every tile is visited
    const float *radius = nullptr;  // [PARTS][tiles]
    int64_t tiles = 0, stride = 0;  // stride = PARTS * tiles
};
int tile_bounds(cuscan_ctx *ctx, const float *x, int64_t n, int d, Buffer &centre, Buffer &radius,
                TileBounds &out, cudaStream_t s, int k = 0, float *thr = nullptr);

// Lists of the 256-row tiles that the 128-row blocks of a kNN screen visit (refined.cu): b.refined.vis
// and vis_count. Right after sort_by_cells; tiles up to kMaxVisitTiles.
constexpr int64_t kMaxVisitTiles = 8192;  // 2,097,152 rows: 268 MB of lists
int visit_lists(cuscan_ctx *ctx, ForestBuffers &b, int64_t n, int d, int k, cudaStream_t s);

// Masks of the tiles that the pruned candidate sweeps may visit: a bit per 128-row tile for every 64
// query rows, up to kMaxMaskTiles tiles.
constexpr int64_t kMaxMaskTiles = 16384;  // 2,097,152 rows: 67 MB of masks
inline int64_t mask_words(int64_t n) { return ceil_div(ceil_div(n, (int64_t)simt::RT), (int64_t)32); }
inline size_t mask_bytes(int64_t n) {
    return ceil_div(n, (int64_t)simt::RT) > kMaxMaskTiles
               ? 0
               : sizeof(uint32_t) * (size_t)(ceil_div(n, (int64_t)simt::QT) * mask_words(n));
}

// Exact kNN of query rows against a spatially ordered set (knn.cu): squared distances, the rows
// and order of launch_exact_knn_fp32, every tile that cannot hold a neighbour left out. ref_ids
// maps reference positions to the ids that order ties and leave in `ids` (null: positions). Entry i
// of the nq entries of qmap (a padded order) is row qmap[i] of `query`, none when -1, and its
// results go to row qmap[i], or with out_rows to row out_rows[qmap[i]]. self: query and reference are the same positions, which exclude
// themselves.
bool knn_pruned_shape(int d, int k);
constexpr int64_t kPrunedPartials = 256ll << 20;  // most bytes of partial lists
// Parts of the reference tiles: a query tile among far rows visits every reference tile, one in a
// cluster a few per cent of them, so the longest CTA sets the end of the launch. Parts of at least 32
// tiles, 16 at most, within kPrunedPartials of partial lists (100,000 x 64: 16.3 ms in one part,
// 11.1 ms in 16).
inline int64_t pruned_parts(int64_t nq, int64_t nr, int k) {
    const int64_t tiles = ceil_div(nr, (int64_t)simt::RT);
    int64_t parts = tiles / 32 < 16 ? tiles / 32 : 16;
    const int64_t room = kPrunedPartials / (8 * nq * k);
    if (parts > room) parts = room;
    return parts < 1 ? 1 : parts;
}
// Bytes of the partial lists: one part writes its results in place.
inline int64_t pruned_partial_bytes(int64_t nq, int64_t nr, int k) {
    const int64_t parts = pruned_parts(nq, nr, k);
    return parts > 1 ? 8 * parts * nq * k : 0;
}
int launch_knn_pruned(cuscan_ctx *ctx, const float *query, int64_t nq, const float *ref, int64_t nr,
                      int d, int k, int self, int32_t *ids, float *dist, cudaStream_t s,
                      Buffer &scratch_ids, Buffer &scratch_dist, Buffer &thr0,
                      const TileBounds &bounds, const int32_t *ref_ids, const int32_t *qmap,
                      const int32_t *out_rows);
// Rows and work from which ordering the rows pays: the cells, their order and the bounds take about
// 0.15 ms, a sweep of nq x nr pairs at d features about nq nr d / 13e12 s.
inline bool worth_pruning(int64_t nq, int64_t nr, int d) {
    return nr >= 2048 && (double)nq * (double)nr * (double)d >= 1e10;
}

#ifdef __CUDACC__
// A lower bound of the reference's f32 squared distance between any row within radius_sum's two
// radii of two centres whose computed squared distance is centre_sq. The triangle inequality
// holds for the exact distances of the stored rows to the stored centres; the computed centre
// distance is within (d + 4) 2^-24 of the exact one and the computed row distance within
// (d + 3) 2^-24 (d <= 256: both below 2e-5), and the radii carry their own rounding. The factors
// of 1e-4 cover all of it. Overflowing values bound nothing.
__device__ __forceinline__ float pruned_bound(float centre_sq, float radius_sum) {
    if (!(centre_sq < 3.0e38f)) return 0.0f;
    const float gap = sqrtf(centre_sq) * (1.0f - 1e-4f) - radius_sum;
    return gap > 0.0f ? gap * gap * (1.0f - 1e-4f) : 0.0f;
}
// Radius from a computed squared distance, rounded up past its rounding and underflow.
__device__ __forceinline__ float bound_radius(float sq) {
    return sqrtf(sq) * (1.0f + 1e-4f) + 1e-17f;
}

namespace simt {

// Balls around the CTA's query rows, one per 16 (shared memory): a tile that straddles two clusters
// still has compact quarters.
constexpr int BALLS = 4;
constexpr int BALL_ROWS = QT / BALLS;
static_assert(BALL_ROWS == kBallRows, "query orders are padded to whole balls");
struct QueryBalls {
    float centre[CUSCAN_PACK_MAX_FEATURES][BALLS];
    float radius[BALLS];
};

// Balls of the 64 rows rows_s[] of x: one warp per ball. Every thread takes part; ends with a
// barrier.
__device__ __forceinline__ void query_balls(QueryBalls &balls, const float *__restrict__ x,
                                            const int32_t *rows_s, int d) {
    static_assert(BALLS == THREADS / 32, "a warp per ball");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int32_t *rows = rows_s + warp * BALL_ROWS;
    for (int f = lane; f < d; f += 32) {
        float sum = 0.0f;
#pragma unroll
        for (int r = 0; r < BALL_ROWS; ++r) sum += x[(int64_t)rows[r] * d + f];
        balls.centre[f][warp] = sum * (1.0f / BALL_ROWS);
    }
    __syncwarp();
    float worst = 0.0f;
    for (int r = 0; r < BALL_ROWS; ++r) {
        const float *row = x + (int64_t)rows[r] * d;
        float sq = 0.0f;
        for (int f = lane; f < d; f += 32) {
            const float t = row[f] - balls.centre[f][warp];
            sq = __fmaf_rn(t, t, sq);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        // a NaN (inf - inf) must not look small
        worst = fmaxf(worst, sq == sq ? sq : CUSCAN_INF);
    }
    if (lane == 0) balls.radius[warp] = bound_radius(worst);
    __syncthreads();
}

// Squared distances of one reference ball's centre to the query balls' centres.
__device__ __forceinline__ void centre_distances(float (&sq)[BALLS], const QueryBalls &balls,
                                                 const TileBounds &B, int d, int64_t ball) {
#pragma unroll
    for (int q = 0; q < BALLS; ++q) sq[q] = 0.0f;
#pragma unroll 4
    for (int f = 0; f < d; ++f) {
        const float c = B.centre[(int64_t)f * B.stride + ball];
        const float4 qc = *reinterpret_cast<const float4 *>(balls.centre[f]);
        const float t0 = c - qc.x, t1 = c - qc.y, t2 = c - qc.z, t3 = c - qc.w;
        sq[0] = __fmaf_rn(t0, t0, sq[0]);
        sq[1] = __fmaf_rn(t1, t1, sq[1]);
        sq[2] = __fmaf_rn(t2, t2, sq[2]);
        sq[3] = __fmaf_rn(t3, t3, sq[3]);
    }
}

// Walk over the tiles [t, t_end) that the query rows must visit: tiles of which some ball's lower
// bound does not exceed the largest threshold of that ball's rows. Each warp bounds 32 tiles at a
// time, one per lane: 8 d multiply-adds per tile against the 8,192 d of the tile itself. The
// thresholds only fall, so a tile left out once stays out. Called at the same points by every
// warp, between barriers that keep the thresholds still, so that all warps walk alike.
// mask: tiles to leave out in any case (a clear bit per tile), null for none.
struct PrunedWalk {
    const QueryBalls *balls;
    int64_t window = -1;  // first tile of the bounds in lb
    float lb[BALLS];      // this lane's tile, by query ball
    const uint32_t *mask = nullptr;
    uint32_t word = ~0u;  // the mask of the window

    __device__ __forceinline__ int64_t next(const TileBounds &B, int d, int64_t t, int64_t t_end,
                                            const float *thr) {
        const int lane = threadIdx.x & 31;
        // the rows of balls 0 and 1, 2 and 3 sit in the lower and upper half warp
        float a = thr[lane], b = thr[lane + 32];
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
            a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, o));
            b = fmaxf(b, __shfl_xor_sync(0xffffffffu, b, o));
        }
        const float worst[BALLS] = {__shfl_sync(0xffffffffu, a, 0), __shfl_sync(0xffffffffu, a, 16),
                                    __shfl_sync(0xffffffffu, b, 0), __shfl_sync(0xffffffffu, b, 16)};
        while (t < t_end) {
            const int64_t base = t & ~(int64_t)31;
            if (base != window) {
                if (mask && !(word = mask[base >> 5])) {
                    window = -1;
                    t = base + 32;
                    continue;
                }
                window = base;
                const int64_t mine = base + lane < B.tiles ? base + lane : B.tiles - 1;
#pragma unroll
                for (int h = 0; h < TileBounds::PARTS; ++h) {
                    float sq[BALLS];
                    const int64_t part = h * B.tiles + mine;
                    centre_distances(sq, *balls, B, d, part);
#pragma unroll
                    for (int q = 0; q < BALLS; ++q) {
                        const float v = pruned_bound(sq[q], balls->radius[q] + B.radius[part]);
                        lb[q] = h == 0 ? v : fminf(lb[q], v);
                    }
                }
            }
            bool near = false;
#pragma unroll
            for (int q = 0; q < BALLS; ++q) near |= !(lb[q] > worst[q]);
            const unsigned visit =
                __ballot_sync(0xffffffffu, near) & word & (0xffffffffu << (int)(t - base));
            if (visit) {
                const int64_t to = base + __ffs(visit) - 1;
                return to < t_end ? to : t_end;
            }
            t = base + 32;
        }
        return t_end;
    }
};

}  // namespace simt
#endif

}  // namespace cuscan
