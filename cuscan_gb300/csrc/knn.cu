// Exact k-nearest-neighbour sweep with f32 direct differences (the "plain" arithmetic).
//
// Semantics follow exact_kernel (crates/cuscan-common/src/kernels/neighbors.rs:17-76): every
// squared distance is acc = fmaf(q_f - r_f, q_f - r_f, acc) over features in order, rows are
// ordered by (distance, id), self is excluded by global id, empty slots hold (pad, nr).
//
// The distances come from the register-tiled sweep of simt.cuh. A thread tests its 64 pairs of a
// tile against its queries' thresholds (the k-th entry of each query's list) with one minimum per
// query; the few pairs that pass go to the query's bucket in shared memory, and after the tile
// each warp merges the buckets of its 16 queries into their sorted lists, all pairs of a bucket at
// once and a lane per list slot. A list costs 8 k bytes of shared memory and no registers, so k
// up to 256 takes the same kernel. The order of arrival does not matter: a list holds the k least
// (distance, id) pairs seen.
//
// Measured on a GB300: 100,000 x 64 rows, k = 10: 48.1 ms against 128.0 ms for one query per
// thread with register lists; 20,011 x 32, k = 50: 3.5 ms against 23.0 ms for per-thread lists
// in global memory.
//
// When there are too few query tiles to fill the SMs the reference range is split across CTAs
// and the partial lists are merged by a second kernel.
#include <limits>

#include "cells.cuh"
#include "forest.cuh"
#include "simt.cuh"

namespace cuscan {
namespace {

using simt::Packed;
using simt::QT;
using simt::RT;
constexpr int BUCKET = 26;        // pairs a query's bucket holds between two merges
constexpr int GROUPED_K = 32;     // largest k of the packed fits' kernels
constexpr int TILED_K = 256;      // largest k of the tiled kernel
constexpr int SEEDED_K = 32;      // largest k whose first thresholds come from group minima

// Shared memory of one CTA after the sweep's stages (k entries per list). Up to k = 57 three
// CTAs fit the 228 KB of an SM (49 with the balls of a pruned sweep).
struct KnnShared {
    float *thr;        // [QT] upper bound of the row's k-th distance
    int32_t *row;      // [QT] query row in the query array
    int *held;         // [QT] pairs pushed to the row's bucket (may exceed BUCKET)
    float *bucket_d;   // [QT][BUCKET] (the first tile's group minima before)
    uint8_t *bucket_r; // [QT][BUCKET] reference within the tile
    float *list_d;     // [QT][k]
    int32_t *list_i;   // [QT][k]
};
__host__ __device__ constexpr size_t knn_smem_bytes(int k, bool pruned = false) {
    return sizeof(float) * (simt::STAGES * simt::STAGE_FLOATS + 3 * QT) + 5 * QT * BUCKET +
           8 * (size_t)QT * k + (pruned ? sizeof(simt::QueryBalls) + 16 : 0);
}
__device__ __forceinline__ KnnShared knn_shared(float *smem, int k);
__device__ __forceinline__ simt::QueryBalls *knn_balls(const KnnShared &s, int k) {
    const uintptr_t end = reinterpret_cast<uintptr_t>(s.list_i + (size_t)QT * k);
    return reinterpret_cast<simt::QueryBalls *>((end + 15) & ~(uintptr_t)15);
}
__device__ __forceinline__ KnnShared knn_shared(float *smem, int k) {
    KnnShared s;
    s.thr = smem + simt::STAGES * simt::STAGE_FLOATS;
    s.row = reinterpret_cast<int32_t *>(s.thr + QT);
    s.held = s.row + QT;
    s.bucket_d = reinterpret_cast<float *>(s.held + QT);
    s.bucket_r = reinterpret_cast<uint8_t *>(s.bucket_d + QT * BUCKET);
    s.list_d = reinterpret_cast<float *>(s.bucket_r + QT * BUCKET);
    s.list_i = reinterpret_cast<int32_t *>(s.list_d + (size_t)QT * k);
    return s;
}

// Merge the pairs (x, j) of the lanes in `hits` into a sorted list of k entries in shared memory;
// one warp, slot s of the list in lane s % 32. Every pair's place is its rank in the list plus its
// rank among the pairs, and a list entry moves by the pairs before it, so the pairs do not wait
// for one another (inserting them one by one took about 900 cycles each at k = 50).
template <int L>
__device__ __forceinline__ void merge_hits(float *ld, int32_t *li, int k, float x, int32_t j,
                                           unsigned hits) {
    const int lane = threadIdx.x & 31;
    float d[L];
    int32_t id[L];
    int shift[L];
#pragma unroll
    for (int e = 0; e < L; ++e) {
        const int s = lane + 32 * e;
        d[e] = s < k ? ld[s] : CUSCAN_INF;
        id[e] = s < k ? li[s] : -1;  // after every pair
        shift[e] = 0;
    }
    int at = 0;  // this lane's pair
    for (unsigned m = hits; m; m &= m - 1) {
        const int from = __ffs(m) - 1;
        const float xo = __shfl_sync(0xffffffffu, x, from);
        const int32_t jo = __shfl_sync(0xffffffffu, j, from);
        int before = 0;
#pragma unroll
        for (int e = 0; e < L; ++e) {
            const bool b = knn_better(d[e], id[e], xo, jo);
            before += __popc(__ballot_sync(0xffffffffu, b));
            shift[e] += b ? 0 : 1;
        }
        if (lane == from) at += before;
        else if (knn_better(xo, jo, x, j)) ++at;
    }
    __syncwarp();
#pragma unroll
    for (int e = 0; e < L; ++e) {
        const int s = lane + 32 * e;
        if (s < k && shift[e] && s + shift[e] < k) {
            ld[s + shift[e]] = d[e];
            li[s + shift[e]] = id[e];
        }
    }
    if (((hits >> lane) & 1u) && at < k) {
        ld[at] = x;
        li[at] = j;
    }
    __syncwarp();
}

// First thresholds of the CTA's rows, before its first tile: each of a row's reference groups
// (two per thread) has a minimum, and the k-th least of these minima bounds the row's k-th
// distance, so that the first tile queues little more than k pairs per row instead of all 128.
// minima: [QT][32] group minima (+inf for an empty group).
__device__ __forceinline__ void seed_thresholds(const KnnShared &sh, const float *minima, int k) {
    // two threads per row, 16 groups each: the group whose rank is k - 1
    const int row = threadIdx.x >> 1, half = threadIdx.x & 1;
    const float *m = minima + row * 32;
    float v[32];
#pragma unroll
    for (int g = 0; g < 32; ++g) v[g] = m[g];
#pragma unroll
    for (int g = 0; g < 16; ++g) {
        const float x = half ? v[16 + g] : v[g];
        const int at = half ? 16 + g : g;
        int rank = 0;
#pragma unroll
        for (int o = 0; o < 32; ++o) rank += (v[o] < x || (v[o] == x && o < at)) ? 1 : 0;
        if (rank == k - 1 && x < sh.thr[row]) sh.thr[row] = x;
    }
}

// A pruned sweep: bounds of the reference tiles, an upper bound of every query's k-th distance
// (from its nearest tile, may be +inf), and the ids and output rows of a spatially ordered set
// (null: positions). thr_out: write only the k-th distance of each query there, over the BALLS
// reference tiles listed in `tiles`.
struct KnnPrune {
    TileBounds bounds;
    const float *thr0;
    const int32_t *ids;
    const int32_t *out_rows;
    float *thr_out;
};

// Padded orders (PRUNE; qmap is never null there): whether a tile holds no row (padding follows a
// cell's rows and the order's end), and the row that entry `i` of a tile stands for: padding repeats
// the first row of its ball, an empty ball the first row of the tile that there is.
__device__ __forceinline__ bool padded_tile_empty(const int32_t *__restrict__ qmap, int64_t q0,
                                                  int64_t nq) {
    for (int b = 0; b < QT; b += kBallRows)
        if (q0 + b < nq && qmap[q0 + b] >= 0) return false;
    return true;
}
__device__ __forceinline__ int32_t padded_row(const int32_t *__restrict__ qmap, int64_t q0, int64_t nq,
                                              int i) {
    int32_t row = q0 + i < nq ? qmap[q0 + i] : -1;
    if (row < 0) row = q0 + i / kBallRows * kBallRows < nq ? qmap[q0 + i / kBallRows * kBallRows] : -1;
    for (int b = 0; row < 0 && b < QT; b += kBallRows)
        if (q0 + b < nq) row = qmap[q0 + b];
    return row;
}

// One CTA: query rows [q0, q0 + 64) of nq against reference rows [r_begin, r_end) (r_begin a
// multiple of the tile). Writes each query's sorted list (k entries) to out rows of width k, at
// part * part_stride when the lists are partial, else to row qmap[qi] (or qi). root: distances
// leave as their square roots.
template <int L, bool PRUNE = false>
__device__ __forceinline__ void knn_block(
    const float *__restrict__ query, int64_t nq, const float *__restrict__ ref, int64_t nr, int d,
    int k, int exclude_self, int64_t query_offset, float pad, int64_t q0, int64_t r_begin,
    int64_t r_end, int32_t *__restrict__ out_ids, float *__restrict__ out_dist,
    int64_t part_stride, int64_t part, bool root, const int32_t *__restrict__ qmap, float *smem,
    const KnnPrune &prune = KnnPrune(), const int64_t *tiles = nullptr) {
    const KnnShared sh = knn_shared(smem, k);
    const simt::Place p = simt::place();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (PRUNE && padded_tile_empty(qmap, q0, nq)) return;
    if (tid < QT) {
        const int64_t qi = q0 + tid;
        const bool valid = qi < nq && !(PRUNE && qmap[qi] < 0);
        sh.row[tid] = PRUNE  ? padded_row(qmap, q0, nq, tid)
                      : valid ? (qmap ? qmap[qi] : (int32_t)qi)
                              : (qmap ? qmap[q0] : (int32_t)q0);
        // rows past the end and padding keep no pair
        sh.thr[tid] = !valid ? -CUSCAN_INF : PRUNE && prune.thr0 ? prune.thr0[qi] : pad;
    }
    for (int e = tid; e < QT * k; e += simt::THREADS) {
        sh.list_d[e] = pad;
        sh.list_i[e] = (int32_t)nr;
    }
    if (tid < QT) sh.held[tid] = 0;
    __syncthreads();
    bool first = true, tied = false;
    // pairs of the tile that may enter their query's list, one bit each (query i, reference j)
    auto test = [&](const Packed(&acc)[8][4], int64_t r0, unsigned long long among) {
        unsigned long long hits = 0;
        const float4 ta = *reinterpret_cast<const float4 *>(sh.thr + p.tq * 4);
        const float4 tb = *reinterpret_cast<const float4 *>(sh.thr + 32 + p.tq * 4);
        const float thr[8] = {ta.x, ta.y, ta.z, ta.w, tb.x, tb.y, tb.z, tb.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float v[8];
            simt::row_of(acc[i], v);
            const float m = fminf(fminf(fminf(v[0], v[1]), fminf(v[2], v[3])),
                                  fminf(fminf(v[4], v[5]), fminf(v[6], v[7])));
            if (m <= thr[i]) {
                const int32_t row = sh.row[simt::query_of(p, i)];
                const int64_t self = exclude_self ? query_offset + row : -1;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int64_t r = r0 + simt::ref_of(p, j);
                    if (v[j] <= thr[i] && r < r_end && r != self) hits |= 1ull << (8 * i + j);
                }
            }
        }
        return hits & among;
    };
    // of those, without the pairs that tie with the list's last entry and come after it by id
    auto without_ties = [&](const Packed(&acc)[8][4], int64_t r0, unsigned long long hits) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (((hits >> (8 * i)) & 0xffull) == 0) continue;
            const int last = simt::query_of(p, i) * k + k - 1;
            const float kth = sh.list_d[last];
            const uint32_t limit = (uint32_t)sh.list_i[last];
            float v[8];
            simt::row_of(acc[i], v);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int64_t r = r0 + simt::ref_of(p, j);
                if (((hits >> (8 * i + j)) & 1ull) && v[j] == kth &&
                    (uint32_t)(PRUNE && prune.ids ? prune.ids[r] : r) >= limit)
                    hits &= ~(1ull << (8 * i + j));
            }
        }
        return hits;
    };
    auto nothing = [](int64_t, int) {};
    const int64_t t_end = ceil_div(r_end, (int64_t)RT);
    simt::PrunedWalk walk{};
    if constexpr (PRUNE) {
        simt::QueryBalls &balls = *knn_balls(sh, k);
        if (!tiles) simt::query_balls(balls, query, sh.row, d);
        walk.balls = &balls;
    }
    auto visit = [&](int64_t t) -> int64_t {
        if constexpr (PRUNE) {
            if (!tiles) return walk.next(prune.bounds, d, t, t_end, sh.thr);
            int64_t to = t_end;  // the least listed tile at or after t
#pragma unroll
            for (int b = 0; b < simt::BALLS; ++b)
                if (tiles[b] >= t && tiles[b] < to) to = tiles[b];
            return to;
        }
        return t;
    };
    auto epilogue = [&](int64_t tile, int, const Packed(&acc)[8][4]) {
        const int64_t r0 = tile * RT;
        if (first && k > 1 && k <= SEEDED_K) {
            float *minima = sh.bucket_d;  // [QT][32], the buckets are empty
            static_assert(5 * BUCKET >= 4 * 32, "group minima fit the buckets");
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int q = simt::query_of(p, i);
                const int64_t self = exclude_self ? query_offset + sh.row[q] : -1;
                float v[8];
                simt::row_of(acc[i], v);
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    float m = CUSCAN_INF;
#pragma unroll
                    for (int j = 4 * g; j < 4 * g + 4; ++j) {
                        const int64_t r = r0 + simt::ref_of(p, j);
                        if (r < r_end && r != self) m = fminf(m, v[j]);
                    }
                    minima[q * 32 + p.tr * 2 + g] = m;
                }
            }
            __syncthreads();
            seed_thresholds(sh, minima, k);
            __syncthreads();
        }
        first = false;
        unsigned long long hits = ~0ull;
        for (bool again = false;; again = true) {
            if (hits) hits = test(acc, r0, hits);
            // A bucket that was full is rare but for rows with many equal distances (duplicates,
            // overflow), whose ties would all be pushed and merged; a thread that met them there
            // looks for them at once from then on. 10,000 equal rows of 16 features, k = 8: 6,116 us
            // without, 384 us. (Looking at ties in every test costs sweeps without them 2 to 11 %;
            // this form at most 1.5 %, pruned sweeps of 50 neighbours 2.4 %.)
            if ((again || tied) && hits) {
                const unsigned long long left = without_ties(acc, r0, hits);
                tied |= left != hits;
                hits = left;
            }
            if (hits) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    if (((hits >> (8 * i)) & 0xffull) == 0) continue;
                    const int q = simt::query_of(p, i);
                    float v[8];
                    simt::row_of(acc[i], v);
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if ((hits >> (8 * i + j)) & 1ull) {
                            const int slot = atomicAdd(&sh.held[q], 1);
                            if (slot < BUCKET) {
                                sh.bucket_d[q * BUCKET + slot] = v[j];
                                sh.bucket_r[q * BUCKET + slot] = (uint8_t)simt::ref_of(p, j);
                                hits &= ~(1ull << (8 * i + j));
                            }
                        }
                }
            }
            // pairs whose bucket was full wait for the merge below
            const int more = __syncthreads_or(hits != 0);
            const int held = lane < 16 ? sh.held[warp * 16 + lane] : 0;
            for (unsigned rows = __ballot_sync(0xffffffffu, held > 0); rows; rows &= rows - 1) {
                const int q = warp * 16 + __ffs(rows) - 1;
                const int count = min(__shfl_sync(0xffffffffu, held, q & 15), BUCKET);
                float x = 0.0f;
                int32_t j = -1;
                float *ld = sh.list_d + (size_t)q * k;
                int32_t *li = sh.list_i + (size_t)q * k;
                bool pass = false;
                if (lane < count) {
                    x = sh.bucket_d[q * BUCKET + lane];
                    j = (int32_t)(r0 + sh.bucket_r[q * BUCKET + lane]);
                    if (PRUNE && prune.ids) j = prune.ids[j];
                    // (the look costs the pruned sweeps of up to 32 neighbours 1 %)
                    pass = (PRUNE && L == 1) || knn_better(x, j, ld[k - 1], li[k - 1]);
                }
                const unsigned enter = __ballot_sync(0xffffffffu, pass);
                if (enter) merge_hits<L>(ld, li, k, x, j, enter);
                if (lane == 0) {
                    const float kth = ld[k - 1];
                    if (kth < sh.thr[q]) sh.thr[q] = kth;
                    sh.held[q] = 0;
                }
            }
            if (!more) break;  // the next tile's first barrier comes before its pushes
            __syncthreads();  // (the next test is against the tightened thresholds)
        }
    };
    if (r_begin < r_end)
        simt::sweep(query, sh.row, ref, d, r_begin / RT, t_end, r_end, smem, visit, nothing,
                    epilogue);
    __syncthreads();
    if (PRUNE && prune.thr_out) {
        if (tid < QT && q0 + tid < nq) prune.thr_out[q0 + tid] = sh.list_d[(size_t)tid * k + k - 1];
        return;  // (entries of padding are not read)
    }
    for (int e = tid; e < QT * k; e += simt::THREADS) {
        const int q = e / k, s = e - q * k;
        const int64_t qi = q0 + q;
        if (qi >= nq) break;
        int64_t row = qmap ? (int64_t)qmap[qi] : qi;
        if (PRUNE && row < 0) continue;
        if (PRUNE && prune.out_rows) row = prune.out_rows[row];
        const int64_t at = part_stride ? part * part_stride + qi * k + s : row * k + s;
        const float x = sh.list_d[e];
        out_ids[at] = sh.list_i[e];
        out_dist[at] = root ? sqrtf(x) : x;
    }
}

// k = 1 (the cell assignment of the refined fits): the nearest reference of each query stays in
// the registers of its threads, without lists or queues.
__device__ __forceinline__ void nearest_block(
    const float *__restrict__ query, int64_t nq, const float *__restrict__ ref, int64_t nr, int d,
    int exclude_self, int64_t query_offset, float pad, int64_t q0, int64_t r_begin, int64_t r_end,
    int32_t *__restrict__ out_ids, float *__restrict__ out_dist, int64_t part_stride,
    int64_t part, bool root, const int32_t *__restrict__ qmap, float *smem) {
    const KnnShared sh = knn_shared(smem, 1);
    const simt::Place p = simt::place();
    const int tid = threadIdx.x;
    if (tid < QT) {
        const int64_t qi = q0 + tid;
        sh.row[tid] = qi < nq ? (qmap ? qmap[qi] : (int32_t)qi) : (qmap ? qmap[q0] : (int32_t)q0);
    }
    __syncthreads();
    float bd[8];
    int32_t bi[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        bd[i] = pad;
        bi[i] = (int32_t)nr;
    }
    auto nothing = [](int64_t, int) {};
    auto every = [](int64_t t) { return t; };
    auto epilogue = [&](int64_t tile, int, const Packed(&acc)[8][4]) {
        const int64_t r0 = tile * RT;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float v[8];
            simt::row_of(acc[i], v);
            const float m = fminf(fminf(fminf(v[0], v[1]), fminf(v[2], v[3])),
                                  fminf(fminf(v[4], v[5]), fminf(v[6], v[7])));
            if (!(m <= bd[i])) continue;
            const int64_t self =
                exclude_self ? query_offset + sh.row[simt::query_of(p, i)] : -1;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int64_t r = r0 + simt::ref_of(p, j);
                if (r < r_end && r != self && knn_better(v[j], (int)r, bd[i], bi[i])) {
                    bd[i] = v[j];
                    bi[i] = (int32_t)r;
                }
            }
        }
    };
    if (r_begin < r_end)
        simt::sweep(query, sh.row, ref, d, r_begin / RT, ceil_div(r_end, (int64_t)RT), r_end, smem,
                    every, nothing, epilogue);
    // the 16 threads of a query: eight lanes of each of two warps
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            const float od = __shfl_xor_sync(0xffffffffu, bd[i], o);
            const int32_t oi = __shfl_xor_sync(0xffffffffu, bi[i], o);
            if (knn_better(od, oi, bd[i], bi[i])) {
                bd[i] = od;
                bi[i] = oi;
            }
        }
    __syncthreads();
    if (tid >= 64 && (tid & 7) == 0)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            sh.bucket_d[simt::query_of(p, i)] = bd[i];
            sh.list_i[simt::query_of(p, i)] = bi[i];
        }
    __syncthreads();
    if (tid < 64 && (tid & 7) == 0)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int q = simt::query_of(p, i);
            const int64_t qi = q0 + q;
            if (qi >= nq) continue;
            const float od = sh.bucket_d[q];
            const int32_t oi = sh.list_i[q];
            if (knn_better(od, oi, bd[i], bi[i])) {
                bd[i] = od;
                bi[i] = oi;
            }
            const int64_t at = part_stride ? part * part_stride + qi
                                           : (qmap ? (int64_t)qmap[qi] : qi);
            out_ids[at] = bi[i];
            out_dist[at] = root ? sqrtf(bd[i]) : bd[i];
        }
}

// L: list slots per lane (ceil(k / 32)); 0: k = 1.
template <int L>
__global__ void __launch_bounds__(simt::THREADS, simt::CTAS_PER_SM) knn_fp32_kernel(
    const float *__restrict__ query, int64_t nq, const float *__restrict__ ref, int64_t nr, int d,
    int k, int exclude_self, int64_t query_offset, float pad, int64_t ref_chunk,
    int32_t *__restrict__ out_ids, float *__restrict__ out_dist, int64_t part_stride, int root,
    const int32_t *__restrict__ qmap) {
    extern __shared__ __align__(16) float smem[];
    const int64_t r_begin = (int64_t)blockIdx.y * ref_chunk;
    const int64_t r_end = r_begin + ref_chunk < nr ? r_begin + ref_chunk : nr;
    if constexpr (L == 0)
        nearest_block(query, nq, ref, nr, d, exclude_self, query_offset, pad,
                      (int64_t)blockIdx.x * QT, r_begin, r_end, out_ids, out_dist, part_stride,
                      (int64_t)blockIdx.y, root != 0, qmap, smem);
    else
        knn_block<L>(query, nq, ref, nr, d, k, exclude_self, query_offset, pad,
                     (int64_t)blockIdx.x * QT, r_begin, r_end, out_ids, out_dist, part_stride,
                     (int64_t)blockIdx.y, root != 0, qmap, smem);
}

// First thresholds of a pruned sweep: each query tile against its own position's reference tile
// (self) or against the tiles nearest to the centres of its balls.
template <int L>
__global__ void __launch_bounds__(simt::THREADS, simt::CTAS_PER_SM) knn_thresholds_kernel(
    const float *__restrict__ query, int64_t nq, const float *__restrict__ ref, int64_t nr, int d,
    int k, int self, float pad, const int32_t *__restrict__ qmap, const KnnPrune prune) {
    extern __shared__ __align__(16) float smem[];
    __shared__ unsigned long long nearest[simt::BALLS];
    __shared__ int64_t tiles[simt::BALLS];
    __shared__ int32_t rows[QT];
    const int tid = threadIdx.x;
    const int64_t q0 = (int64_t)blockIdx.x * QT;
    if (padded_tile_empty(qmap, q0, nq)) return;
    if (!self) {
        simt::QueryBalls &balls = *knn_balls(knn_shared(smem, k), k);
        if (tid < simt::BALLS) nearest[tid] = ~0ull;
        if (tid < QT) rows[tid] = padded_row(qmap, q0, nq, tid);
        __syncthreads();
        simt::query_balls(balls, query, rows, d);
        unsigned long long best[simt::BALLS] = {~0ull, ~0ull, ~0ull, ~0ull};
        for (int64_t part = tid; part < prune.bounds.stride; part += simt::THREADS) {
            if (!(prune.bounds.radius[part] >= 0.0f)) continue;  // an empty half
            float sq[simt::BALLS];
            simt::centre_distances(sq, balls, prune.bounds, d, part);
            const uint32_t t = (uint32_t)(part % prune.bounds.tiles);
#pragma unroll
            for (int b = 0; b < simt::BALLS; ++b) {
                const float v = sq[b] == sq[b] ? sq[b] : CUSCAN_INF;
                const unsigned long long key = ((unsigned long long)__float_as_uint(v) << 32) | t;
                best[b] = key < best[b] ? key : best[b];
            }
        }
#pragma unroll
        for (int b = 0; b < simt::BALLS; ++b) atomicMin(&nearest[b], best[b]);
        __syncthreads();
    }
    // self: the tile of each ball's first position
    if (tid < simt::BALLS)
        tiles[tid] = self ? padded_row(qmap, q0, nq, tid * kBallRows) / RT
                          : (int64_t)(uint32_t)nearest[tid];
    __syncthreads();
    knn_block<L, true>(query, nq, ref, nr, d, k, self, 0, pad, q0, 0, nr, nullptr, nullptr, 0, 0,
                       false, qmap, smem, prune, tiles);
}

template <int L>
__global__ void __launch_bounds__(simt::THREADS, simt::CTAS_PER_SM) knn_pruned_kernel(
    const float *__restrict__ query, int64_t nq, const float *__restrict__ ref, int64_t nr, int d,
    int k, int self, float pad, int64_t ref_chunk, int32_t *__restrict__ out_ids,
    float *__restrict__ out_dist, int64_t part_stride, const int32_t *__restrict__ qmap,
    const KnnPrune prune) {
    extern __shared__ __align__(16) float smem[];
    const int64_t r_begin = (int64_t)blockIdx.y * ref_chunk;
    const int64_t r_end = r_begin + ref_chunk < nr ? r_begin + ref_chunk : nr;
    // the last query tiles first: far rows are ordered last and visit the most tiles
    const int64_t q0 = (int64_t)(gridDim.x - 1 - blockIdx.x) * QT;
    knn_block<L, true>(query, nq, ref, nr, d, k, self, 0, pad, q0, r_begin, r_end, out_ids, out_dist,
                       part_stride, (int64_t)blockIdx.y, false, qmap, smem, prune);
}

// Packed fits: fit blockIdx.z, query tile blockIdx.x, reference chunk blockIdx.y of `splits`
// (the self-kNN of launch_exact_knn_fp32: squared distances, self excluded, +inf padding).
// Fits with k > 32 take the per-fit launch instead.
__global__ void __launch_bounds__(simt::THREADS, simt::CTAS_PER_SM)
    pack_knn_kernel(const PackFit *__restrict__ fits, int splits) {
    extern __shared__ __align__(16) float smem[];
    const PackFit &f = fits[blockIdx.z];
    const int64_t n = f.n, q0 = (int64_t)blockIdx.x * QT;
    const int k = f.k;
    if (k > GROUPED_K || q0 >= n) return;
    const int64_t chunk = ceil_div(ceil_div(n, (int64_t)splits), (int64_t)RT) * RT;
    const int64_t r_begin = (int64_t)blockIdx.y * chunk;
    const int64_t r_end = r_begin + chunk < n ? r_begin + chunk : n;
    if (splits > 1)
        knn_block<1>(f.x, n, f.x, n, f.d, k, 1, 0, CUSCAN_INF, q0, r_begin, r_end, f.part_ids,
                     f.part_dist, n * k, (int64_t)blockIdx.y, false, nullptr, smem);
    else
        knn_block<1>(f.x, n, f.x, n, f.d, k, 1, 0, CUSCAN_INF, q0, r_begin, r_end, f.ids, f.dsq,
                     0, 0, false, nullptr, smem);
}

// Merge `splits` sorted partial lists of query q into its final row (orow): one warp, the list in
// shared memory. The entries are taken rank by rank, 32 lists at a time; a rank at which no list
// can contribute ends the merge, so few of the splits * k entries are read.
template <int L>
__device__ __forceinline__ void knn_merge_row(const int32_t *__restrict__ part_ids,
                                              const float *__restrict__ part_dist, int64_t q,
                                              int64_t orow, int k, int splits,
                                              int64_t part_stride, float pad, int64_t nr,
                                              bool root, int32_t *__restrict__ ids,
                                              float *__restrict__ dist, float *ld, int32_t *li) {
    const int lane = threadIdx.x & 31;
    for (int s = lane; s < k; s += 32) {
        ld[s] = pad;
        li[s] = (int32_t)nr;
    }
    __syncwarp();
    for (int s = 0; s < k; ++s) {
        bool any = false;
        for (int b = 0; b < splits; b += 32) {
            const int sp = b + lane;
            float x = pad;
            int32_t j = (int32_t)nr;
            if (sp < splits) {
                x = part_dist[sp * part_stride + q * k + s];
                j = part_ids[sp * part_stride + q * k + s];
            }
            const unsigned hits =
                __ballot_sync(0xffffffffu, knn_better(x, j, ld[k - 1], li[k - 1]));
            if (hits) {
                any = true;
                merge_hits<L>(ld, li, k, x, j, hits);
            }
        }
        if (!any) break;
    }
    __syncwarp();
    for (int s = lane; s < k; s += 32) {
        ids[orow * k + s] = li[s];
        dist[orow * k + s] = root ? sqrtf(ld[s]) : ld[s];
    }
}

constexpr int MERGE_WARPS = 4;

template <int L>
__global__ void __launch_bounds__(32 * MERGE_WARPS)
    knn_merge_kernel(const int32_t *__restrict__ part_ids, const float *__restrict__ part_dist,
                     int64_t nq, int k, int splits, int64_t part_stride, float pad, int64_t nr,
                     int root, int32_t *__restrict__ ids, float *__restrict__ dist,
                     const int32_t *__restrict__ qmap, const int32_t *__restrict__ out_rows) {
    __shared__ float ld[MERGE_WARPS][32 * L];
    __shared__ int32_t li[MERGE_WARPS][32 * L];
    const int warp = threadIdx.x >> 5;
    const int64_t q = (int64_t)blockIdx.x * MERGE_WARPS + warp;
    if (q >= nq) return;
    int64_t row = qmap ? (int64_t)qmap[q] : q;
    if (row < 0) return;  // padding of a query order
    if (out_rows) row = out_rows[row];
    knn_merge_row<L>(part_ids, part_dist, q, row, k, splits, part_stride, pad, nr, root != 0, ids,
                     dist, ld[warp], li[warp]);
}

// Packed fits: the partial lists of fit blockIdx.y merged into its kNN lists.
__global__ void __launch_bounds__(32 * MERGE_WARPS)
    pack_knn_merge_kernel(const PackFit *__restrict__ fits, int splits) {
    __shared__ float ld[MERGE_WARPS][32];
    __shared__ int32_t li[MERGE_WARPS][32];
    const PackFit &f = fits[blockIdx.y];
    const int warp = threadIdx.x >> 5;
    const int64_t q = (int64_t)blockIdx.x * MERGE_WARPS + warp;
    if (f.k > GROUPED_K || q >= f.n) return;
    knn_merge_row<1>(f.part_ids, f.part_dist, q, q, f.k, splits, f.n * f.k, CUSCAN_INF, f.n, false,
                     f.ids, f.dsq, ld[warp], li[warp]);
}

__global__ void sqrt_rows_kernel(float *dist, int64_t count) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) dist[i] = sqrtf(dist[i]);
}

constexpr int WIDE_Q = 128, WIDE_T = 32, WIDE_TP = 36;

__device__ __forceinline__ void cp_async4_zfill(void *smem, const void *gmem, bool valid) {
    unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    int src_size = valid ? 4 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(s), "l"(gmem),
                 "r"(src_size));
}
// Copy reference rows [r0, r0+WIDE_T) into tile[f*WIDE_TP + r] (zero fill past nr).
__device__ __forceinline__ void load_ref_tile(float *tile, const float *ref, int64_t nr, int d,
                                              int64_t r0) {
    const int total = WIDE_T * d;
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
        int r = e / d;
        int f = e - r * d;
        int64_t row = r0 + r;
        bool valid = row < nr;
        const float *src = valid ? ref + row * (int64_t)d + f : ref;
        cp_async4_zfill(&tile[f * WIDE_TP + r], src, valid);
    }
}

// Any k: one thread per query keeps its list in the output row in global memory, like the
// reference's serial kernel. Only k > 256 takes it, whose lists do not fit shared memory beside
// the sweep's stages.
__global__ void __launch_bounds__(WIDE_Q) knn_fp32_wide_kernel(
    const float *__restrict__ query, int64_t nq, const float *__restrict__ ref, int64_t nr, int d,
    int k, int exclude_self, int64_t query_offset, float pad, int32_t *__restrict__ ids,
    float *__restrict__ dist) {
    extern __shared__ __align__(16) float smem[];
    float *qs = smem;
    float *tile = smem + (size_t)d * WIDE_Q;
    const int tid = threadIdx.x;
    const int64_t q0 = (int64_t)blockIdx.x * WIDE_Q;
    const int64_t qi = q0 + tid;
    for (int e = tid; e < WIDE_Q * d; e += WIDE_Q) {
        int q = e / d;
        int f = e - q * d;
        int64_t row = q0 + q;
        qs[f * WIDE_Q + q] = row < nq ? query[row * (int64_t)d + f] : 0.0f;
    }
    int32_t *li = ids + (qi < nq ? qi : 0) * (int64_t)k;
    float *ld = dist + (qi < nq ? qi : 0) * (int64_t)k;
    if (qi < nq)
        for (int s = 0; s < k; ++s) {
            li[s] = (int32_t)nr;
            ld[s] = pad;
        }
    float worst_d = pad;
    int worst_i = (int)nr;
    const int64_t self = exclude_self ? query_offset + qi : -1;
    for (int64_t r0 = 0; r0 < nr; r0 += WIDE_T) {
        __syncthreads();
        load_ref_tile(tile, ref, nr, d, r0);
        simt::cp_async_commit();
        simt::cp_async_wait<0>();
        __syncthreads();
        float acc[WIDE_T];
#pragma unroll
        for (int r = 0; r < WIDE_T; ++r) acc[r] = 0.0f;
        for (int f = 0; f < d; ++f) {
            const float qv = qs[f * WIDE_Q + tid];
            const float4 *row4 = reinterpret_cast<const float4 *>(tile + f * WIDE_TP);
#pragma unroll
            for (int r4 = 0; r4 < WIDE_T / 4; ++r4) {
                const float4 v = row4[r4];
                float t0 = qv - v.x, t1 = qv - v.y, t2 = qv - v.z, t3 = qv - v.w;
                acc[4 * r4 + 0] = __fmaf_rn(t0, t0, acc[4 * r4 + 0]);
                acc[4 * r4 + 1] = __fmaf_rn(t1, t1, acc[4 * r4 + 1]);
                acc[4 * r4 + 2] = __fmaf_rn(t2, t2, acc[4 * r4 + 2]);
                acc[4 * r4 + 3] = __fmaf_rn(t3, t3, acc[4 * r4 + 3]);
            }
        }
        if (qi < nq) {
            for (int r = 0; r < WIDE_T; ++r) {
                const int64_t j = r0 + r;
                const float x = acc[r];
                if (j >= nr || j == self || !knn_better(x, (int)j, worst_d, worst_i)) continue;
                int slot = k - 1;
                while (slot > 0 && knn_better(x, (int)j, ld[slot - 1], li[slot - 1])) {
                    li[slot] = li[slot - 1];
                    ld[slot] = ld[slot - 1];
                    --slot;
                }
                li[slot] = (int32_t)j;
                ld[slot] = x;
                worst_d = ld[k - 1];
                worst_i = li[k - 1];
            }
        }
    }
}

// Split the reference range when the query tiles alone cannot fill the GPU: `splits` CTAs per
// query tile, each over `chunk` references.
void knn_split_plan(const cuscan_ctx *ctx, int64_t nq, int64_t nr, int64_t &splits,
                    int64_t &chunk, int d, int k) {
    // every part fills lists of its own: about 4 k merged pairs per row, against 384 d cycles per
    // tile (both per resident CTA)
    simt::split_plan(ctx->sm_count, ceil_div(nq, (int64_t)QT), nr, 2,
                     1.0 + 2.0 * (double)k / (double)d, splits, chunk, simt::split_most(nq));
}

template <int L>
int run_knn(cuscan_ctx *ctx, const float *query, int64_t nq, const float *ref, int64_t nr, int d,
            int k, int exclude_self, int64_t query_offset, int squared, int32_t *ids, float *dist,
            cudaStream_t s, Buffer &scratch_ids, Buffer &scratch_dist, const int32_t *qmap,
            int64_t *launches, bool one_part) {
    const float pad = squared ? std::numeric_limits<float>::infinity() : 3.40282346638528859812e+38f;
    int64_t splits = 1, chunk = 0;
    knn_split_plan(ctx, nq, nr, splits, chunk, d, k);
    const int64_t stride = nq * k;
    const size_t list_bytes = (size_t)(stride * splits) * sizeof(float);
    // A captured sweep allocates nothing, and one of more than 32 neighbours leaves no pointer to the
    // workspace in the graph, which a later call could free.
    if (splits > 1 && capturing(s) &&
        (L > 1 || scratch_ids.bytes < list_bytes || scratch_dist.bytes < list_bytes))
        one_part = true;
    if (one_part) splits = 1;
    if (splits > 1) {
        int rc = ensure(ctx, scratch_ids, list_bytes, "kNN partial ids");
        if (!rc) rc = ensure(ctx, scratch_dist, list_bytes, "kNN partial distances");
        if (rc && rc != CUSCAN_MEMORY) return rc;
        if (rc) {  // no room for the partial lists: the references in one part
            clear_error(ctx);
            release(scratch_ids);
            release(scratch_dist);
            splits = 1;
        }
    }
    const size_t smem = knn_smem_bytes(k);
    if (int rc = allow_dynamic_smem(ctx, knn_fp32_kernel<L>, smem)) return rc;
    const dim3 grid((unsigned)ceil_div(nq, (int64_t)QT), (unsigned)splits);
    if (splits == 1) {
        if (!squared && qmap)
            return fail(ctx, CUSCAN_INVALID_INPUT, "row-subset kNN is squared only");
        CUSCAN_KERNEL(knn_fp32_kernel<L>, grid, simt::THREADS, smem, s, query, nq, ref, nr, d, k,
                      exclude_self, query_offset, pad, nr, ids, dist, 0, squared ? 0 : 1, qmap);
        CUSCAN_LAUNCH(ctx, "knn_fp32_kernel");
        if (launches) *launches += 1;
        return CUSCAN_OK;
    }
    CUSCAN_KERNEL(knn_fp32_kernel<L>, grid, simt::THREADS, smem, s, query, nq, ref, nr, d, k,
                  exclude_self, query_offset, pad, chunk, as<int32_t>(scratch_ids),
                  as<float>(scratch_dist), stride, 0, qmap);
    CUSCAN_LAUNCH(ctx, "knn_fp32_kernel");
    constexpr int M = L == 0 ? 1 : L;
    CUSCAN_KERNEL(knn_merge_kernel<M>, (unsigned)ceil_div(nq, (int64_t)MERGE_WARPS),
                  32 * MERGE_WARPS, 0, s, as<int32_t>(scratch_ids), as<float>(scratch_dist), nq, k,
                  (int)splits, stride, pad, nr, squared ? 0 : 1, ids, dist, qmap, nullptr);
    CUSCAN_LAUNCH(ctx, "knn_merge_kernel");
    if (launches) *launches += 2;
    return CUSCAN_OK;
}

template <int L>
int run_knn_pruned(cuscan_ctx *ctx, const float *query, int64_t nq, const float *ref, int64_t nr,
                   int d, int k, int self, int32_t *ids, float *dist, cudaStream_t s,
                   Buffer &scratch_ids, Buffer &scratch_dist, Buffer &thr0,
                   const TileBounds &bounds, const int32_t *ref_ids, const int32_t *qmap,
                   const int32_t *out_rows) {
    const float pad = std::numeric_limits<float>::infinity();
    if (int rc = ensure(ctx, thr0, sizeof(float) * nq, "first thresholds")) return rc;
    const size_t smem = knn_smem_bytes(k, true);
    if (int rc = allow_dynamic_smem(ctx, knn_thresholds_kernel<L>, smem)) return rc;
    if (int rc = allow_dynamic_smem(ctx, knn_pruned_kernel<L>, smem)) return rc;
    const unsigned qtiles = (unsigned)ceil_div(nq, (int64_t)QT);
    KnnPrune prune{bounds, nullptr, ref_ids, out_rows, as<float>(thr0)};
    CUSCAN_KERNEL(knn_thresholds_kernel<L>, qtiles, simt::THREADS, smem, s, query, nq, ref, nr, d, k,
                  self, pad, qmap, prune);
    CUSCAN_LAUNCH(ctx, "knn_thresholds_kernel");
    prune.thr0 = as<float>(thr0);
    prune.thr_out = nullptr;
    int64_t splits = pruned_parts(nq, nr, k);
    const int64_t chunk = ceil_div(ceil_div(nr, (int64_t)RT), splits) * RT;
    splits = ceil_div(nr, chunk);
    const dim3 grid(qtiles, (unsigned)splits);
    if (splits == 1) {
        CUSCAN_KERNEL(knn_pruned_kernel<L>, grid, simt::THREADS, smem, s, query, nq, ref, nr, d, k,
                      self, pad, chunk, ids, dist, 0, qmap, prune);
        CUSCAN_LAUNCH(ctx, "knn_pruned_kernel");
        return CUSCAN_OK;
    }
    const int64_t stride = nq * k;
    int rc = ensure(ctx, scratch_ids, (size_t)(stride * splits) * sizeof(int32_t), "kNN partial ids");
    if (!rc) rc = ensure(ctx, scratch_dist, (size_t)(stride * splits) * sizeof(float),
                         "kNN partial distances");
    if (rc) return rc;
    CUSCAN_KERNEL(knn_pruned_kernel<L>, grid, simt::THREADS, smem, s, query, nq, ref, nr, d, k, self,
                  pad, chunk, as<int32_t>(scratch_ids), as<float>(scratch_dist), stride, qmap, prune);
    CUSCAN_LAUNCH(ctx, "knn_pruned_kernel");
    CUSCAN_KERNEL(knn_merge_kernel<L>, (unsigned)ceil_div(nq, (int64_t)MERGE_WARPS),
                  32 * MERGE_WARPS, 0, s, as<int32_t>(scratch_ids), as<float>(scratch_dist), nq, k,
                  (int)splits, stride, pad, nr, 0, ids, dist, qmap, out_rows);
    CUSCAN_LAUNCH(ctx, "knn_merge_kernel");
    return CUSCAN_OK;
}

}  // namespace

int launch_exact_knn_fp32(cuscan_ctx *ctx, const float *query, int64_t nq, const float *ref,
                          int64_t nr, int d, int k, int exclude_self, int64_t query_offset,
                          int squared, int32_t *ids, float *dist, cudaStream_t s,
                          Buffer &scratch_ids, Buffer &scratch_dist, const int32_t *qmap,
                          int64_t *launches, bool one_part) {
    if (nq == 0) return CUSCAN_OK;
    if (d > CUSCAN_PACK_MAX_FEATURES)
        return fail(ctx, CUSCAN_CAPACITY,
                    "feature count %d exceeds the shared-memory staging limit of the kNN kernel "
                    "(at most 256 features)", d);
    if (k > TILED_K) {
        if (qmap) return fail(ctx, CUSCAN_CAPACITY, "row-subset kNN supports k <= 256");
        const float pad = squared ? std::numeric_limits<float>::infinity() : 3.40282346638528859812e+38f;
        const size_t smem = ((size_t)d * WIDE_Q + (size_t)d * WIDE_TP) * sizeof(float);
        if (int rc = allow_dynamic_smem(ctx, knn_fp32_wide_kernel, smem)) return rc;
        CUSCAN_KERNEL(knn_fp32_wide_kernel, (unsigned)ceil_div(nq, WIDE_Q), WIDE_Q, smem, s,
            query, nq, ref, nr, d, k, exclude_self, query_offset, pad, ids, dist);
        CUSCAN_LAUNCH(ctx, "knn_fp32_wide_kernel");
        if (launches) *launches += squared ? 1 : 2;
        if (!squared) {
            CUSCAN_KERNEL(sqrt_rows_kernel, (unsigned)ceil_div(nq * k, 256), 256, 0, s, dist, nq * k);
            CUSCAN_LAUNCH(ctx, "sqrt_rows_kernel");
        }
        return CUSCAN_OK;
    }
#define CUSCAN_RUN_KNN(L)                                                                        \
    run_knn<L>(ctx, query, nq, ref, nr, d, k, exclude_self, query_offset, squared, ids, dist, s, \
               scratch_ids, scratch_dist, qmap, launches, one_part)
    if (k == 1) return CUSCAN_RUN_KNN(0);
    if (k <= 32) return CUSCAN_RUN_KNN(1);
    if (k <= 64) return CUSCAN_RUN_KNN(2);
    if (k <= 128) return CUSCAN_RUN_KNN(4);
    return CUSCAN_RUN_KNN(8);
#undef CUSCAN_RUN_KNN
}

bool knn_pruned_shape(int d, int k) { return d <= CUSCAN_PACK_MAX_FEATURES && k <= TILED_K; }

int launch_knn_pruned(cuscan_ctx *ctx, const float *query, int64_t nq, const float *ref, int64_t nr,
                      int d, int k, int self, int32_t *ids, float *dist, cudaStream_t s,
                      Buffer &scratch_ids, Buffer &scratch_dist, Buffer &thr0,
                      const TileBounds &bounds, const int32_t *ref_ids, const int32_t *qmap,
                      const int32_t *out_rows) {
#define CUSCAN_RUN_KNN(L)                                                                       \
    run_knn_pruned<L>(ctx, query, nq, ref, nr, d, k, self, ids, dist, s, scratch_ids,           \
                      scratch_dist, thr0, bounds, ref_ids, qmap, out_rows)
    if (nq == 0) return CUSCAN_OK;
    if (k <= 32) return CUSCAN_RUN_KNN(1);
    if (k <= 64) return CUSCAN_RUN_KNN(2);
    if (k <= 128) return CUSCAN_RUN_KNN(4);
    return CUSCAN_RUN_KNN(8);
#undef CUSCAN_RUN_KNN
}

int launch_pack_knn(cuscan_ctx *ctx, const PackFit *fits, int count, int64_t n_max, int d_max,
                    int k_max, int splits, cudaStream_t s, int64_t &launches) {
    if (d_max > CUSCAN_PACK_MAX_FEATURES)
        return fail(ctx, CUSCAN_CAPACITY, "feature count %d exceeds the kNN staging limit", d_max);
    const size_t smem = knn_smem_bytes(k_max);
    if (int rc = allow_dynamic_smem(ctx, pack_knn_kernel, smem)) return rc;
    const dim3 grid((unsigned)ceil_div(n_max, (int64_t)QT), (unsigned)splits, (unsigned)count);
    CUSCAN_KERNEL(pack_knn_kernel, grid, simt::THREADS, smem, s, fits, splits);
    ++launches;
    if (splits > 1) {
        const dim3 mg((unsigned)ceil_div(n_max, (int64_t)MERGE_WARPS), (unsigned)count);
        CUSCAN_KERNEL(pack_knn_merge_kernel, mg, 32 * MERGE_WARPS, 0, s, fits, splits);
        ++launches;
    }
    CUSCAN_LAUNCH(ctx, "pack_knn_kernel");
    return CUSCAN_OK;
}

}  // namespace cuscan
