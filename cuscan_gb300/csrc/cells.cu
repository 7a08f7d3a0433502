// Spatial order of a point set: cells of pivot rows along a tour of the pivots, rows far outside
// their cell's scale last; and the bounds of its tiles.
//
// The sweeps of this library compare tiles of rows with tiles of rows. In this order a tile of
// clustered data is a small ball, so a tile's nearest rows sit in a few other tiles: the screens
// see them first, and the sweeps with bounds (cells.cuh) leave most of the others out. Nothing
// but the order of work depends on it; every result is decided by exact distances.
#include "cells.cuh"

#include "workspace.cuh"

namespace cuscan {
namespace {

// Evenly spaced rows as cell pivots.
__global__ void pick_pivots_kernel(const float *__restrict__ x, int64_t n, int d, int npiv,
                                   float *__restrict__ piv) {
    int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (int64_t)npiv * d) return;
    const int64_t p = e / d;
    const int f = (int)(e - p * d);
    const int64_t r = (p * n) / npiv;
    piv[e] = x[r * d + f];
}

// Squared distances of pivot blockIdx.x to every pivot, one warp per pair.
__global__ void pivot_distances_kernel(const float *__restrict__ piv, int npiv, int d,
                                       float *__restrict__ out) {
    const float *a = piv + (int64_t)blockIdx.x * d;
    const int lane = threadIdx.x & 31;
    for (int j = threadIdx.x >> 5; j < npiv; j += blockDim.x >> 5) {
        float sq = 0.0f;
        for (int f = lane; f < d; f += 32) {
            const float t = a[f] - piv[(int64_t)j * d + f];
            sq = fmaf(t, t, sq);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        if (lane == 0) out[blockIdx.x * npiv + j] = sq;
    }
}

// Greedy tour of the pivots: from each to the nearest one not visited yet, so that the cells of
// a cluster follow one another and few tiles straddle two clusters. Also writes the pivots in tour
// order, and the order. One CTA, a thread per pivot: a step is a serial chain, so the distances sit
// in shared memory (the lower triangle, 130 KB) and a block minimum is two warp reductions around
// one barrier: 32-bit keys of a distance's upper bits over the pivot's number. 256 pivots of 64
// features take 69 us; with a row of the matrix read from L2 and a 64-bit shuffle minimum per
// step they took 172 us.
constexpr size_t tour_smem(int npiv) { return sizeof(float) * (size_t)npiv * (npiv - 1) / 2; }
__global__ void __launch_bounds__(kMaxPivots)
    pivot_tour_kernel(const float *__restrict__ piv, const float *__restrict__ dist, int npiv, int d,
                      float *__restrict__ out, int32_t *__restrict__ tour) {
    static_assert(kMaxPivots == 256, "a pivot's number takes the low byte of a key");
    constexpr int WARPS = kMaxPivots / 32;
    extern __shared__ float tri[];  // [i (i - 1) / 2 + j], j < i
    __shared__ unsigned best[2][WARPS];
    __shared__ int order[kMaxPivots];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
#pragma unroll 8
    for (int i = 1; i < npiv; ++i)
        if (t < i) tri[i * (i - 1) / 2 + t] = dist[i * npiv + t];
    bool open = t < npiv && t != 0;
    if (t == 0) order[0] = 0;
    __syncthreads();
    int at = 0;
    for (int s = 1; s < npiv; ++s) {
        unsigned key = ~0u;
        if (open) {
            const int i = max(at, t), j = min(at, t);
            const float v = tri[i * (i - 1) / 2 + j];
            // NaN and infinite distances come last, in index order
            key = (__float_as_uint(v >= 0.0f ? v : CUSCAN_INF) & ~255u) | (unsigned)t;
        }
        key = __reduce_min_sync(0xffffffffu, key);
        if (lane == 0) best[s & 1][warp] = key;
        __syncthreads();  // the other buffer's readers are past it too
        at = (int)(__reduce_min_sync(0xffffffffu, best[s & 1][lane % WARPS]) & 255u);
        if (t == at) open = false;
        if (t == 0) order[s] = at;
    }
    __syncthreads();
    if (t < npiv) tour[t] = order[t];
    for (int64_t e = t; e < (int64_t)npiv * d; e += blockDim.x) {
        const int64_t p = e / d;
        out[e] = piv[(int64_t)order[p] * d + (e - p * d)];
    }
}

// Per cell: rows with a positive distance and the sum of its inverse (their ratio is the cell's
// scale, which a few far rows hardly move).
__global__ void cell_scale_kernel(const int32_t *__restrict__ cell, const float *__restrict__ dist,
                                  int64_t n, float *__restrict__ count, float *__restrict__ inv) {
    __shared__ float c[kMaxPivots], v[kMaxPivots];
    for (int i = threadIdx.x; i < kMaxPivots; i += blockDim.x) c[i] = v[i] = 0.0f;
    __syncthreads();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const float sq = dist[i];
        if (sq > 1e-30f && sq < 1e30f) {
            atomicAdd(&c[cell[i]], 1.0f);
            atomicAdd(&v[cell[i]], 1.0f / sq);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kMaxPivots; i += blockDim.x)
        if (c[i] != 0.0f) {
            atomicAdd(&count[i], c[i]);
            atomicAdd(&inv[i], v[i]);
        }
}

// Rows whose squared distance to the pivot is over three times the cell's scale (harmonic mean) go
// to a second run of cells after all others: a few noise rows would widen every tile they sit in.
constexpr float FAR_ROWS = 3.0f;
// Norm levels per cell: 2 * npiv cells of 64 levels are at most n / 2 keys.
constexpr int CELL_LEVELS = 64;
__global__ void far_rows_kernel(int32_t *__restrict__ cell, const float *__restrict__ dist,
                                int64_t n, int npiv, const float *__restrict__ count,
                                const float *__restrict__ inv) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    // A row without a distance to any pivot (not a number somewhere) got the number past the last
    // cell, where the order has no entry; the last cell takes it.
    const int32_t c = min(cell[i], npiv - 1);
    cell[i] = dist[i] * inv[c] > FAR_ROWS * count[c] ? c + npiv : c;
}

// Start of every cell in a padded order (kMaxCells threads), from its row count.
__device__ __forceinline__ int padded_start(int count, int *warp_sums) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int mine = (count + kBallRows - 1) / kBallRows * kBallRows;
    int x = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    int before = 0;
    for (int w = 0; w < warp; ++w) before += warp_sums[w];
    return before + x - mine;
}

// Padded order of m query rows by cell, one CTA; the order within a cell is free.
__global__ void __launch_bounds__(kMaxCells)
    order_queries_kernel(const int32_t *__restrict__ cell, int64_t m, int npiv, int64_t padded,
                         int32_t *__restrict__ order) {
    __shared__ int start[kMaxCells];
    __shared__ int warp_sums[kMaxCells / 32];
    const int t = threadIdx.x;
    start[t] = 0;
    for (int64_t i = t; i < padded; i += kMaxCells) order[i] = -1;
    __syncthreads();
    for (int64_t i = t; i < m; i += kMaxCells) atomicAdd(&start[min(cell[i], npiv - 1)], 1);
    __syncthreads();
    const int at = padded_start(start[t], warp_sums);
    start[t] = at;
    __syncthreads();
    for (int64_t i = t; i < m; i += kMaxCells)
        order[atomicAdd(&start[min(cell[i], npiv - 1)], 1)] = (int32_t)i;
}

// The same of a sorted set's positions: shift[c] is what a position of cell c moves by. The cells
// were sorted by keys of `levels` levels each; key k starts at start[k] + sums[k / kScanTile].
__global__ void __launch_bounds__(kMaxCells)
    cell_shift_kernel(const int32_t *__restrict__ start, const int32_t *__restrict__ sums, int64_t n,
                      int levels, int32_t *__restrict__ shift) {
    __shared__ int warp_sums[kMaxCells / 32];
    const int t = threadIdx.x;
    auto begin = [&](int64_t key) { return key < n ? start[key] + sums[key / kScanTile] : (int)n; };
    const int64_t key = (int64_t)t * levels;
    const int from = begin(key), to = t + 1 < (int)kMaxCells ? begin(key + levels) : (int)n;
    const int at = padded_start(to - from, warp_sums);
    shift[t] = at - from;
}
__global__ void order_positions_kernel(const int32_t *__restrict__ cell,
                                       const int32_t *__restrict__ shift, int64_t n,
                                       int32_t *__restrict__ order) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p < n) order[p + shift[cell[p]]] = (int32_t)p;
}

// Upper bounds of the components' cheapest edges from the pivot rows: a pair of pivots in two
// components is an edge of known weight, up to the rounding of the pivot distances (their sums
// run in another order than the reference's; both are within 2e-5 of exact). Block p: pivot p.
__global__ void pivot_bounds_kernel(const float *__restrict__ dist, int npiv, int64_t n,
                                    const float *__restrict__ core,
                                    const int32_t *__restrict__ label,
                                    uint32_t *__restrict__ cbound) {
    const int64_t row = ((int64_t)blockIdx.x * n) / npiv;
    const int32_t l = label[row];
    float best = CUSCAN_INF;
    for (int j = threadIdx.x; j < npiv; j += 32) {
        const int64_t other = ((int64_t)j * n) / npiv;
        if (label[other] == l) continue;
        const float v = dist[blockIdx.x * npiv + j] * (1.0f + 1e-4f) + 1e-30f;
        best = fminf(best, fmaxf(fmaxf(v, core[row]), core[other]));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) best = fminf(best, __shfl_xor_sync(0xffffffffu, best, o));
    if (threadIdx.x == 0 && best < CUSCAN_INF) atomicMin(&cbound[l], __float_as_uint(best));
}

// Squared norms of the rows, their range and the largest |x| (f32 bits in range[0..2]; range[0] starts
// at the largest pattern). Eight lanes per row.
__global__ void row_norms_kernel(const float *__restrict__ x, int64_t n, int d,
                                 float *__restrict__ out, unsigned int *__restrict__ range) {
    const int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3;
    const int sub = threadIdx.x & 7;
    float sq = 0.0f, most = 0.0f;
    if (r < n)
        for (int f = sub; f < d; f += 8) {
            const float v = x[r * d + f];
            sq = fmaf(v, v, sq);
            most = fmaxf(most, fabsf(v));
        }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    if (r < n && sub == 0) out[r] = sq;
    const unsigned bits = __float_as_uint(sq);
    const unsigned lo = __reduce_min_sync(0xffffffffu, r < n ? bits : 0xffffffffu);
    const unsigned hi = __reduce_max_sync(0xffffffffu, r < n ? bits : 0u);
    const unsigned mx = __reduce_max_sync(0xffffffffu, __float_as_uint(most));
    if ((threadIdx.x & 31) == 0) {
        if (lo < *(volatile unsigned int *)&range[0]) atomicMin(&range[0], lo);
        if (hi > *(volatile unsigned int *)&range[1]) atomicMax(&range[1], hi);
        if (mx > *(volatile unsigned int *)&range[2]) atomicMax(&range[2], mx);
    }
}
// Squared norm of pivot blockIdx.x (one warp); block 0 also clears the range and the cell sums.
__global__ void pivot_norms_kernel(const float *__restrict__ piv, int d,
                                   unsigned int *__restrict__ range, float *__restrict__ scale,
                                   float *__restrict__ norm) {
    const int t = threadIdx.x;
    if (blockIdx.x == 0) {
        if (t < 8) range[t] = t == 0 ? 0xffffffffu : 0u;
        for (int i = t; i < 2 * kMaxPivots; i += 32) scale[i] = 0.0f;
    }
    float sq = 0.0f;
    for (int f = t; f < d; f += 32) {
        const float v = piv[(int64_t)blockIdx.x * d + f];
        sq = fmaf(v, v, sq);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    if (t == 0) norm[blockIdx.x] = sq;
}

// Rows whose cell is too tight for a screen whose bounds sit `shift` |x|^2 below the distances: the
// gap that such a row's lists must show between its k-th and their last entry is about
// H (2 / d) ln(entries / k) where the cell's scale is H and the rows fill d dimensions (fewer
// make the gap wider). Counted in range[3] by block 0.
// Block p also adds to range[4] (f32) the pairs of rows between cell p and the cells that lie too
// far off to hold a neighbour of its rows or of theirs: beyond the two cells' scales and one more.
__global__ void __launch_bounds__(kMaxPivots)
    tight_rows_kernel(const float *__restrict__ count, const float *__restrict__ inv,
                      const float *__restrict__ norm, const float *__restrict__ dist,
                      const int32_t *__restrict__ tour, int npiv, float shift, float gap,
                      unsigned int *__restrict__ range) {
    const int c = threadIdx.x, p = blockIdx.x;
    const bool used = c < npiv && inv[c] > 0.0f;
    if (p == 0) {
        unsigned rows = 0;
        if (used && shift * norm[c] > gap * (count[c] / inv[c])) rows = (unsigned)count[c];
        rows = __reduce_add_sync(0xffffffffu, rows);
        if ((c & 31) == 0 && rows) atomicAdd(&range[3], rows);
    }
    if (!(inv[p] > 0.0f)) return;
    float pairs = 0.0f;
    if (used) {
        const float a = sqrtf(count[p] / inv[p]), b = sqrtf(count[c] / inv[c]);
        if (sqrtf(dist[tour[p] * npiv + tour[c]]) > a + b + fmaxf(a, b)) pairs = count[p] * count[c];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) pairs += __shfl_xor_sync(0xffffffffu, pairs, o);
    if ((c & 31) == 0 && pairs > 0.0f) atomicAdd(reinterpret_cast<float *>(range) + 4, pairs);
}

// Centre and radius of half blockIdx.y of tile blockIdx.x (simt::RT rows). With thr also an upper
// bound of the rows' k-th nearest squared distances, excluding themselves: twice the radius, where
// the half has more than k rows.
__global__ void __launch_bounds__(simt::RT)
    tile_bounds_kernel(const float *__restrict__ x, int64_t n, int d, int64_t tiles,
                       float *__restrict__ centre, float *__restrict__ radius,
                       int k, float *__restrict__ thr) {
    __shared__ float c[CUSCAN_PACK_MAX_FEATURES];
    __shared__ float worst[simt::RT / 32];
    constexpr int ROWS = simt::RT / TileBounds::PARTS;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t row0 = (int64_t)blockIdx.x * simt::RT + blockIdx.y * ROWS;
    const int64_t at = (int64_t)blockIdx.y * tiles + blockIdx.x, stride = TileBounds::PARTS * tiles;
    const int rows = (int)(n - row0 < ROWS ? n - row0 : ROWS);
    if (rows <= 0) {  // the last tile's second half may be empty: beyond every threshold
        for (int f = tid; f < d; f += simt::RT) centre[(int64_t)f * stride + at] = 0.0f;
        if (tid == 0) radius[at] = -CUSCAN_INF;
        if (tid == 0 && thr) thr[at] = -CUSCAN_INF;
        return;
    }
    for (int f = tid; f < d; f += simt::RT) {
        float sum = 0.0f;
#pragma unroll 8
        for (int r = 0; r < rows; ++r) sum += x[(row0 + r) * d + f];
        c[f] = sum / (float)rows;
        centre[(int64_t)f * stride + at] = c[f];
    }
    __syncthreads();
    float m = 0.0f;
    for (int r = warp; r < rows; r += simt::RT / 32) {
        float sq = 0.0f;
        for (int f = lane; f < d; f += 32) {
            const float t = x[(row0 + r) * d + f] - c[f];
            sq = fmaf(t, t, sq);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        m = fmaxf(m, sq == sq ? sq : CUSCAN_INF);
    }
    if (lane == 0) worst[warp] = m;
    __syncthreads();
    if (tid == 0) {
        for (int w = 1; w < simt::RT / 32; ++w) m = fmaxf(m, worst[w]);
        m = bound_radius(m);
        radius[at] = m;
        if (thr) thr[at] = rows > k ? 4.0f * m * m * (1.0f + 1e-3f) : CUSCAN_INF;
    }
}

// The tiles (256 rows) that query block blockIdx.x (128 rows) of a kNN screen visits, without those
// whose every row is farther from the block's rows than their thresholds, by the balls around the
// block's halves and the tile's quarters (pruned_bound). The list starts with the tiles around the
// block's own rows, where its thresholds tighten, and goes on cyclically. The lookups are d L2
// reads per 128 reference rows and block: 0.06 ms at 100,000 x 64.
constexpr int VISIT_THREADS = 256;
__global__ void __launch_bounds__(VISIT_THREADS)
    visit_lists_kernel(const TileBounds balls, const float *__restrict__ ball_thr, int d, int n_tiles,
                       uint16_t *__restrict__ list, int32_t *__restrict__ counts) {
    __shared__ alignas(8) float centre[CUSCAN_PACK_MAX_FEATURES][2];  // read as float2
    __shared__ uint32_t bits[kMaxVisitTiles / 32];
    __shared__ int warp_sums[VISIT_THREADS / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t qb = blockIdx.x;
    for (int f = tid; f < d; f += VISIT_THREADS)
        for (int p = 0; p < 2; ++p)
            centre[f][p] = balls.centre[(int64_t)f * balls.stride + p * balls.tiles + qb];
    const int words = (n_tiles + 31) / 32;
    for (int w = tid; w < words; w += VISIT_THREADS) bits[w] = 0;
    float qr[2], thr[2];
    for (int p = 0; p < 2; ++p) {
        qr[p] = balls.radius[p * balls.tiles + qb];
        thr[p] = ball_thr[p * balls.tiles + qb];
    }
    int first = (int)(qb / 2) - 2;  // two tiles before the block's own
    if (first < 0) first = 0;
    __syncthreads();
    for (int u0 = 0; u0 < 2 * n_tiles; u0 += VISIT_THREADS) {
        const int u = u0 + tid, t = u >> 1;  // 128 rows of tile t: two balls
        bool visit = false;
        if (u < balls.tiles) {
            float sq[2][2] = {{0.0f, 0.0f}, {0.0f, 0.0f}};  // [ball][half]
            const float *src = balls.centre + u;
            for (int f = 0; f < d; ++f) {
                const float2 q = *reinterpret_cast<const float2 *>(centre[f]);
                const float a = src[0], b = src[balls.tiles];
                src += balls.stride;
                sq[0][0] = fmaf(a - q.x, a - q.x, sq[0][0]);
                sq[0][1] = fmaf(a - q.y, a - q.y, sq[0][1]);
                sq[1][0] = fmaf(b - q.x, b - q.x, sq[1][0]);
                sq[1][1] = fmaf(b - q.y, b - q.y, sq[1][1]);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float r = balls.radius[h * balls.tiles + u];
#pragma unroll
                for (int p = 0; p < 2; ++p)
                    if (r >= 0.0f && qr[p] >= 0.0f)  // both hold rows
                        visit |= !(pruned_bound(sq[h][p], qr[p] + r) > thr[p]);
            }
        }
        if (visit) {
            const int i = t >= first ? t - first : t - first + n_tiles;
            atomicOr(&bits[i >> 5], 1u << (i & 31));
        }
    }
    __syncthreads();
    // the set bits in order: a contiguous run of words per thread
    const int per = (words + VISIT_THREADS - 1) / VISIT_THREADS;
    const int w0 = min(tid * per, words), w1 = min(w0 + per, words);
    int mine = 0;
    for (int w = w0; w < w1; ++w) mine += __popc(bits[w]);
    int x = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    int at = x - mine;
    for (int w = 0; w < warp; ++w) at += warp_sums[w];
    uint16_t *out = list + qb * n_tiles;
    for (int w = w0; w < w1; ++w)
        for (uint32_t m = bits[w]; m; m &= m - 1) {
            const int t = w * 32 + __ffs(m) - 1 + first;
            out[at++] = (uint16_t)(t < n_tiles ? t : t - n_tiles);
        }
    if (tid == VISIT_THREADS - 1) counts[qb] = at;
}

}  // namespace

// The tour, behind the pivots' distances: pivots in tour order by their picked number.
static int32_t *pivot_tour(RefinedBuffers &R, int npiv) {
    return reinterpret_cast<int32_t *>(as<float>(R.pivot_d) + npiv * npiv);
}

int sort_by_cells(cuscan_ctx *ctx, ForestBuffers &b, const float *x, int64_t n, int d,
                  cudaStream_t s) {
    RefinedBuffers &R = b.refined;
    const int npiv = cell_pivots(n);
    int rc = ensure(ctx, R.pivots, sizeof(float) * 2 * npiv * d, "cell pivots");
    if (!rc) rc = ensure(ctx, R.pivot_d, sizeof(float) * (npiv + 1) * npiv, "pivot distances");
    if (!rc) rc = ensure(ctx, R.cells, sizeof(int32_t) * n, "cells");
    if (!rc) rc = ensure(ctx, R.cell_d, sizeof(float) * n, "cell distances");
    if (!rc) rc = ensure(ctx, R.cell_scale, sizeof(float) * 3 * kMaxPivots, "cell scales");
    if (rc) return rc;
    float *toured = as<float>(R.pivots), *picked = toured + (size_t)npiv * d;
    CUSCAN_KERNEL(pick_pivots_kernel, (unsigned)ceil_div((int64_t)npiv * d, 256), 256, 0, s, x, n, d,
                  npiv, picked);
    CUSCAN_KERNEL(pivot_distances_kernel, npiv, 256, 0, s, picked, npiv, d, as<float>(R.pivot_d));
    if ((rc = allow_dynamic_smem(ctx, pivot_tour_kernel, tour_smem(kMaxPivots)))) return rc;
    CUSCAN_KERNEL(pivot_tour_kernel, 1, kMaxPivots, tour_smem(npiv), s, picked, as<float>(R.pivot_d), npiv, d,
                  toured, pivot_tour(R, npiv));
    CUSCAN_LAUNCH(ctx, "cell pivots");
    if ((rc = launch_exact_knn_fp32(ctx, x, n, toured, npiv, d, 1, 0, 0, 1, as<int32_t>(R.cells),
                                    as<float>(R.cell_d), s, b.knn_ids_tmp, b.knn_dist_tmp)))
        return rc;
    float *count = as<float>(R.cell_scale), *inv = count + kMaxPivots;
    if ((rc = ensure(ctx, R.rnorm, sizeof(float) * n, "row norms"))) return rc;
    if ((rc = ensure(ctx, R.norm_range, 32, "norm range"))) return rc;
    unsigned int *range = as<unsigned int>(R.norm_range);
    CUSCAN_KERNEL(pivot_norms_kernel, npiv, 32, 0, s, toured, d, range, count, inv + kMaxPivots);
    CUSCAN_KERNEL(row_norms_kernel, (unsigned)ceil_div(8 * n, 256), 256, 0, s, x, n, d,
                  as<float>(R.rnorm), range);
    int64_t grid = ceil_div(n, 1024);
    if (grid > 2 * (int64_t)ctx->sm_count) grid = 2 * (int64_t)ctx->sm_count;
    CUSCAN_KERNEL(cell_scale_kernel, (unsigned)grid, 256, 0, s, as<int32_t>(R.cells),
                  as<float>(R.cell_d), n, count, inv);
    CUSCAN_KERNEL(far_rows_kernel, (unsigned)ceil_div(n, 256), 256, 0, s, as<int32_t>(R.cells),
                  as<float>(R.cell_d), n, npiv, count, inv);
    CUSCAN_LAUNCH(ctx, "cell scales");
    // within a cell by norm: a 32-column chunk of the screens is bounded by its largest dot product
    // and its smallest norm, which is tight only when its norms are alike
    R.cell_levels = CELL_LEVELS;
    if ((rc = forest_cell_keys(ctx, b, n, R.cell_levels, s))) return rc;
    return forest_sort_by_component(ctx, b, x, nullptr, as<int32_t>(R.cells), n, d, s,
                                    as<int32_t>(R.key));
}

int count_tight_rows(cuscan_ctx *ctx, ForestBuffers &b, int64_t n, float shift, float gap,
                     cudaStream_t s) {
    RefinedBuffers &R = b.refined;
    const float *count = as<float>(R.cell_scale);
    const int npiv = cell_pivots(n);
    CUSCAN_KERNEL(tight_rows_kernel, npiv, kMaxPivots, 0, s, count, count + kMaxPivots,
                  count + 2 * kMaxPivots, as<float>(R.pivot_d), pivot_tour(R, npiv), npiv, shift,
                  gap, as<unsigned int>(R.norm_range));
    CUSCAN_LAUNCH(ctx, "tight_rows_kernel");
    return CUSCAN_OK;
}

int read_apart(cuscan_ctx *ctx, ForestBuffers &b, int64_t n, float &apart, cudaStream_t s) {
    if (int rc = count_tight_rows(ctx, b, n, 0.0f, 1.0f, s)) return rc;
    float *pairs = reinterpret_cast<float *>(ctx->fit->host_words());
    CUSCAN_CUDA(ctx, cudaMemcpyAsync(pairs, as<float>(b.refined.norm_range) + 4, sizeof(float),
                                     cudaMemcpyDeviceToHost, s));
    CUSCAN_CUDA(ctx, cudaStreamSynchronize(s));
    apart = (float)((double)*pairs / ((double)n * (double)n));
    return CUSCAN_OK;
}

int order_queries(cuscan_ctx *ctx, ForestBuffers &b, const float *pivots, int npiv, const float *q,
                  int64_t m, int d, int32_t *order, cudaStream_t s) {
    RefinedBuffers &R = b.refined;
    int rc = ensure(ctx, R.cells, sizeof(int32_t) * m, "cells");
    if (!rc) rc = ensure(ctx, R.cell_d, sizeof(float) * m, "cell distances");
    if (rc) return rc;
    if ((rc = launch_exact_knn_fp32(ctx, q, m, pivots, npiv, d, 1, 0, 0, 1, as<int32_t>(R.cells),
                                    as<float>(R.cell_d), s, b.knn_ids_tmp, b.knn_dist_tmp)))
        return rc;
    CUSCAN_KERNEL(order_queries_kernel, 1, (unsigned)kMaxCells, 0, s, as<int32_t>(R.cells), m,
                  npiv, padded_queries(m), order);
    CUSCAN_LAUNCH(ctx, "order_queries_kernel");
    return CUSCAN_OK;
}

int order_positions(cuscan_ctx *ctx, ForestBuffers &b, int64_t n, int32_t *order, cudaStream_t s) {
    // the sort left the scan of its keys and the cell of every position
    int32_t *shift = as<int32_t>(b.fill);  // the sort's cursors, idle now
    CUSCAN_CUDA(ctx, cudaMemsetAsync(order, 0xff, sizeof(int32_t) * padded_queries(n), s));
    CUSCAN_KERNEL(cell_shift_kernel, 1, (unsigned)kMaxCells, 0, s, as<int32_t>(b.start),
                  as<int32_t>(b.scan_tmp), n, b.refined.cell_levels, shift);
    CUSCAN_KERNEL(order_positions_kernel, (unsigned)ceil_div(n, 256), 256, 0, s, as<int32_t>(b.labp),
                  shift, n, order);
    CUSCAN_LAUNCH(ctx, "order_positions_kernel");
    return CUSCAN_OK;
}

int pivot_component_bounds(cuscan_ctx *ctx, ForestBuffers &b, int64_t n, const float *core,
                           const int32_t *label, uint32_t *cbound, cudaStream_t s) {
    const int npiv = cell_pivots(n);
    CUSCAN_KERNEL(pivot_bounds_kernel, npiv, 32, 0, s, as<float>(b.refined.pivot_d), npiv, n, core,
                  label, cbound);
    CUSCAN_LAUNCH(ctx, "pivot_bounds_kernel");
    return CUSCAN_OK;
}

int visit_lists(cuscan_ctx *ctx, ForestBuffers &b, int64_t n, int d, int k, cudaStream_t s) {
    RefinedBuffers &R = b.refined;
    const int64_t blocks = ceil_div(n, 128), tiles = ceil_div(n, 256);
    int rc = ensure(ctx, R.ball_thr, sizeof(float) * TileBounds::PARTS * blocks, "ball thresholds");
    if (!rc) rc = ensure(ctx, R.vis, sizeof(uint16_t) * blocks * tiles, "tile lists");
    if (!rc) rc = ensure(ctx, R.vis_count, sizeof(int32_t) * blocks, "tile list lengths");
    TileBounds balls;
    if (!rc) rc = tile_bounds(ctx, as<float>(b.xp), n, d, R.tile_centre, R.tile_radius, balls, s, k,
                              as<float>(R.ball_thr));
    if (rc) return rc;
    CUSCAN_KERNEL(visit_lists_kernel, (unsigned)blocks, VISIT_THREADS, 0, s, balls,
                  as<float>(R.ball_thr), d, (int)tiles, reinterpret_cast<uint16_t *>(R.vis.ptr),
                  as<int32_t>(R.vis_count));
    CUSCAN_LAUNCH(ctx, "visit_lists_kernel");
    return CUSCAN_OK;
}

int tile_bounds(cuscan_ctx *ctx, const float *x, int64_t n, int d, Buffer &centre, Buffer &radius,
                TileBounds &out, cudaStream_t s, int k, float *thr) {
    const int64_t tiles = ceil_div(n, (int64_t)simt::RT);
    constexpr int PARTS = TileBounds::PARTS;
    int rc = ensure(ctx, centre, sizeof(float) * PARTS * tiles * d, "tile centres");
    if (!rc) rc = ensure(ctx, radius, sizeof(float) * PARTS * tiles, "tile radii");
    if (rc) return rc;
    const dim3 grid((unsigned)tiles, PARTS);
    CUSCAN_KERNEL(tile_bounds_kernel, grid, simt::RT, 0, s, x, n, d, tiles,
                  as<float>(centre), as<float>(radius), k, thr);
    CUSCAN_LAUNCH(ctx, "tile_bounds_kernel");
    out.centre = as<float>(centre);
    out.radius = as<float>(radius);
    out.tiles = tiles;
    out.stride = PARTS * tiles;
    return CUSCAN_OK;
}

}  // namespace cuscan
