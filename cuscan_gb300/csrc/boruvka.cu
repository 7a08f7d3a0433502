// Borůvka round kernels with f32 direct differences (the "plain" arithmetic), and the CSR
// component reduction of the reference's HdbscanOps::component_reduce.
//
// Candidate rule (crates/hdbscan/src/kernels/boruvka.rs:68-140): for row i, the
// lexicographically smallest (w_ij, j) with w_ij = max(max(d2_ij, core_i), core_j) over rows j
// of another component. Here a (w, j) pair is packed into one 64-bit key
// (canonical weight bits << 32 | j): for non-negative weights the unsigned key order is exactly
// that lexicographic order, so partial results from any split of the reference range combine
// with a single atomicMin.
//
// The fused fit path calls the kernel on component-sorted rows. A (query block, reference
// tile) pair whose rows all carry one label holds only same-component pairs and is skipped
// before any distance is computed; tile label ranges are precomputed per 32-row tile.
#include <mutex>

#include "cells.cuh"
#include "forest.cuh"
#include "simt.cuh"
#include "workspace.cuh"

namespace cuscan {
namespace {

using simt::Packed;
using simt::QT;
constexpr int RT = 32;                        // rows per label range
constexpr int RANGES = simt::RT / RT;         // label ranges per reference tile
constexpr int META_SLOTS = 4;

// Label range of each RT-row tile.
__global__ void tile_range_kernel(const int32_t *__restrict__ labels, int64_t n,
                                  int32_t *__restrict__ lo, int32_t *__restrict__ hi) {
    int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int64_t tiles = ceil_div(n, RT);
    if (t >= tiles) return;
    int64_t a = t * RT, b = a + RT < n ? a + RT : n;
    int32_t mn = labels[a], mx = labels[a];
    for (int64_t i = a + 1; i < b; ++i) {
        int32_t l = labels[i];
        mn = l < mn ? l : mn;
        mx = l > mx ? l : mx;
    }
    lo[t] = mn;
    hi[t] = mx;
}

// Shared memory of the candidate sweep after its stages: the reference rows' cores, labels and
// ids (a slot per tile in flight) and the query rows.
struct CandShared {
    float core[META_SLOTS][simt::RT];
    int32_t label[META_SLOTS][simt::RT];
    int32_t id[META_SLOTS][simt::RT];
    int32_t row[QT];        // position of each query row
    float q_core[QT];
    int32_t q_label[QT];
    int32_t q_range[2];
    // pruned sweeps: what each query's cheapest edge has to beat, and the queries' ball
    float thr[QT];
    alignas(16) simt::QueryBalls balls;
};
constexpr size_t kCandSmem =
    sizeof(float) * simt::STAGES * simt::STAGE_FLOATS + sizeof(CandShared);

// A pruned sweep: bounds of the reference tiles and the components' upper bounds (f32 bits, by
// label). A pair is left out only when its weight exceeds the smaller of its query's best so far and
// the bound of the query's component. A pair above the best is not the query's cheapest edge, and a
// query whose cheapest edge lies above the component's bound cannot win the component: its key is
// then some larger weight, or none. So every query's cheapest weight is at least the smaller of its
// key's and the bound, and its key is exact where that is at most the bound.
// The component bounds stay as the round starts with them: lowering them as the sweep finds
// edges prunes more of a round (31.2 -> 26.3 ms in the second round at 100,000 x 64), but then fewer
// rows leave a lower bound above their component's next bound, and the rounds after it scan more
// rows (18,539 -> 75,251 in the fourth): 66.6 ms became 74.7 ms over the fit's rounds.
struct CandPrune {
    TileBounds bounds;
    const uint32_t *cbound;
    const uint32_t *masks;  // candidate_masks_kernel, or null
    int words;              // of a query tile's mask
};

// Masks of the tiles that 64 query rows (tile blockIdx.x) have to visit: some row's distance to some
// half of the tile, by the ball around it, does not exceed the bound of the row's component. The
// rows themselves bound far better than the balls around them that the sweep walks with: in d
// features a row's offset in its cluster is nearly at right angles to the other cluster, so its
// centre distance is about sqrt(D^2 + r^2) where the balls leave D - r. At 100,000 x 64 (50
// clusters, noise) the rounds between clusters visit 41 % of the tiles instead of 78 %.
// A thread per half tile, the rows transposed in shared memory; 37 us per round at 20,011 x 32, where
// the sweeps fell from 2.26 to 1.66 ms over three rounds.
constexpr int MASK_THREADS = 256;
constexpr size_t mask_smem(int d, int64_t words) {
    return sizeof(float) * QT * (size_t)(d + 1) + sizeof(uint32_t) * (size_t)words;
}
__global__ void __launch_bounds__(MASK_THREADS, 2)
    candidate_masks_kernel(const float *__restrict__ data, const int32_t *__restrict__ labels, int d,
                           const int32_t *__restrict__ qmap, int64_t nq, const TileBounds B,
                           const uint32_t *__restrict__ cbound, int words,
                           uint32_t *__restrict__ masks) {
    extern __shared__ __align__(16) float rows_t[];  // [d][QT], the rows' bounds, the mask
    float *thr = rows_t + (size_t)QT * d;
    uint32_t *bits = reinterpret_cast<uint32_t *>(thr + QT);
    const int tid = threadIdx.x;
    const int64_t q0 = (int64_t)blockIdx.x * QT;
    // rows past the end repeat the first, with a bound that nothing meets
    for (int e = tid; e < QT * d; e += MASK_THREADS) {
        const int r = e / d, f = e - r * d;
        const int64_t qi = q0 + r < nq ? q0 + r : q0;
        rows_t[f * QT + r] = data[(qmap ? (int64_t)qmap[qi] : qi) * d + f];
    }
    if (tid < QT) {
        const int64_t qi = q0 + tid;
        thr[tid] = qi < nq ? __uint_as_float(cbound[labels[qmap ? (int64_t)qmap[qi] : qi]])
                           : -CUSCAN_INF;
    }
    for (int w = tid; w < words; w += MASK_THREADS) bits[w] = 0;
    __syncthreads();
    for (int64_t ball = tid; ball < B.stride; ball += MASK_THREADS) {
        const float radius = B.radius[ball];
        if (!(radius >= 0.0f)) continue;  // an empty half
        bool visit = false;
#pragma unroll 1
        for (int g = 0; g < QT && !visit; g += 32) {
            float sq[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) sq[i] = 0.0f;
            const float *centre = B.centre + ball;
            for (int f = 0; f < d; ++f) {
                const float c = *centre;
                centre += B.stride;
#pragma unroll
                for (int i = 0; i < 32; i += 4) {
                    const float4 q = *reinterpret_cast<const float4 *>(rows_t + f * QT + g + i);
                    const float t0 = q.x - c, t1 = q.y - c, t2 = q.z - c, t3 = q.w - c;
                    sq[i] = __fmaf_rn(t0, t0, sq[i]);
                    sq[i + 1] = __fmaf_rn(t1, t1, sq[i + 1]);
                    sq[i + 2] = __fmaf_rn(t2, t2, sq[i + 2]);
                    sq[i + 3] = __fmaf_rn(t3, t3, sq[i + 3]);
                }
            }
#pragma unroll
            for (int i = 0; i < 32; ++i) visit |= !(pruned_bound(sq[i], radius) > thr[g + i]);
        }
        const int64_t t = ball % B.tiles;
        if (visit) atomicOr(&bits[t >> 5], 1u << (int)(t & 31));
    }
    __syncthreads();
    for (int w = tid; w < words; w += MASK_THREADS) masks[(int64_t)blockIdx.x * words + w] = bits[w];
}

// One CTA: 64 query rows [q0, q0 + 64) against rows [r_begin, r_end) (r_begin a multiple of the
// reference tile); each query's cheapest cross-component key is folded into row_keys with
// atomicMin. The distances come from the register-tiled sweep of simt.cuh. Per pair the epilogue
// costs a three-way maximum, a label test, a select and a minimum; the exact (w, id) order is only
// looked at where a query's minimum over its eight references reaches its best so far.
// Measured on a GB300, the four rounds of the anisotropic 100,000 x 64 fit in plain f32:
// 86.7 ms against 143.1 ms for one query per thread.
template <bool PRUNE = false>
__device__ __forceinline__ void candidates_block(
    const float *__restrict__ data, const float *__restrict__ core,
    const int32_t *__restrict__ labels, const int32_t *__restrict__ ids, int64_t n, int d,
    const int32_t *__restrict__ tile_lo, const int32_t *__restrict__ tile_hi, int64_t q0,
    int64_t r_begin, int64_t r_end, unsigned long long *__restrict__ row_keys,
    const int32_t *__restrict__ qmap, int64_t nq, int64_t qoff, float *smem,
    const CandPrune &prune = CandPrune()) {
    CandShared &sh = *reinterpret_cast<CandShared *>(smem + simt::STAGES * simt::STAGE_FLOATS);
    const simt::Place p = simt::place();
    const int tid = threadIdx.x, lane = tid & 31;
    if (tid == 0) {
        sh.q_range[0] = INT32_MAX;
        sh.q_range[1] = INT32_MIN;
    }
    __syncthreads();
    // query rows are positions qmap[qi] (or qoff + qi) of the same arrays; rows past the end
    // repeat the first and are not written
    if (tid < QT) {
        const int64_t qi = q0 + tid < nq ? q0 + tid : q0;
        const int32_t pos = qmap ? qmap[qi] : (int32_t)(qoff + qi);
        const int32_t l = labels[pos];
        sh.row[tid] = pos;
        sh.q_core[tid] = core[pos];
        sh.q_label[tid] = l;
        atomicMin(&sh.q_range[0], l);
        atomicMax(&sh.q_range[1], l);
        if (PRUNE)
            sh.thr[tid] = q0 + tid < nq ? __uint_as_float(prune.cbound[l]) : -CUSCAN_INF;
    }
    __syncthreads();
    simt::PrunedWalk walk{};
    if constexpr (PRUNE) {
        simt::query_balls(sh.balls, data, sh.row, d);
        walk.balls = &sh.balls;
        walk.mask = prune.masks ? prune.masks + (q0 / QT) * prune.words : nullptr;
    }
    const int32_t qlo = sh.q_range[0];
    const bool q_uniform = qlo == sh.q_range[1];
    float qc[8], bw[8];
    int32_t ql[8], bi[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int q = simt::query_of(p, i);
        qc[i] = sh.q_core[q];
        ql[i] = sh.q_label[q];
        bw[i] = CUSCAN_INF;
        bi[i] = -1;  // none (the largest id as unsigned)
    }

    const int64_t t_end = ceil_div(r_end, (int64_t)simt::RT), ranges = ceil_div(n, (int64_t)RT);
    // A tile whose rows all carry the one label of the CTA's queries holds no cross pair. The
    // lanes of every warp look at 32 tiles at a time.
    auto other_component = [&](int64_t t) -> int64_t {
        if (!q_uniform) return t;
        while (t < t_end) {
            const int64_t mine = t + lane;
            bool skip = mine < t_end;
            for (int c = 0; c < RANGES; ++c) {
                const int64_t at = mine * RANGES + c;
                if (skip && at < ranges) skip = tile_lo[at] == qlo && tile_hi[at] == qlo;
            }
            const unsigned visit = __ballot_sync(0xffffffffu, !skip);
            if (visit) {
                const int64_t to = t + __ffs(visit) - 1;
                return to < t_end ? to : t_end;
            }
            t += 32;
        }
        return t_end;
    };
    auto next = [&](int64_t t) -> int64_t {
        if constexpr (PRUNE) {
            for (;;) {
                const int64_t a = other_component(t);
                if (a >= t_end) return t_end;
                t = walk.next(prune.bounds, d, a, t_end, sh.thr);
                if (t == a || t >= t_end) return t;
            }
        }
        return other_component(t);
    };
    auto meta = [&](int64_t t, int slot) {
        int64_t row = t * simt::RT + tid;
        if (row >= r_end) row = r_end - 1;
        simt::cp_async4(&sh.core[slot][tid], core + row);
        simt::cp_async4(reinterpret_cast<float *>(&sh.label[slot][tid]),
                        reinterpret_cast<const float *>(labels + row));
        if (ids)
            simt::cp_async4(reinterpret_cast<float *>(&sh.id[slot][tid]),
                            reinterpret_cast<const float *>(ids + row));
    };
    auto epilogue = [&](int64_t tile, int slot, const Packed(&acc)[8][4]) {
        const int64_t r0 = tile * simt::RT;
        if (PRUNE) __syncthreads();  // every warp has walked before the thresholds move
        float rc[8];
        int32_t rl[8];
        bool ok[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int r = simt::ref_of(p, j);
            rc[j] = sh.core[slot][r];
            rl[j] = sh.label[slot][r];
            ok[j] = rl[j] >= 0 && r0 + r < r_end;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float w[8];
            simt::row_of(acc[i], w);
            float m = CUSCAN_INF;
            bool any = false;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                w[j] = fmaxf(fmaxf(w[j], qc[i]), rc[j]);
                const bool cross = ok[j] && rl[j] != ql[i];
                any |= cross;
                m = fminf(m, cross ? w[j] : CUSCAN_INF);
            }
            if (!any || !(m <= bw[i])) continue;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (!ok[j] || rl[j] == ql[i] || !(w[j] <= bw[i])) continue;
                const int r = simt::ref_of(p, j);
                const int32_t id = ids ? sh.id[slot][r] : (int32_t)(r0 + r);
                if (w[j] < bw[i] || (uint32_t)id < (uint32_t)bi[i]) {
                    bw[i] = w[j];
                    bi[i] = id;
                }
            }
            // weights are >= 0, so their bit patterns order like the values; rows past the end
            // (-inf, above every weight as unsigned bits) take none
            if (PRUNE) {
                const int q = simt::query_of(p, i);
                if (q0 + q < nq)
                    atomicMin(reinterpret_cast<unsigned int *>(&sh.thr[q]),
                              weight_key_bits(bw[i]));
            }
        }
    };
    if (r_begin < r_end)
        simt::sweep(data, sh.row, data, d, r_begin / simt::RT, t_end, r_end, smem, next, meta,
                    epilogue);
    // the 16 threads of a query: eight lanes of each of two warps
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        unsigned long long key =
            bi[i] == -1 ? ~0ull
                        : ((unsigned long long)weight_key_bits(bw[i]) << 32) | (uint32_t)bi[i];
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            const unsigned long long u = __shfl_xor_sync(0xffffffffu, key, o);
            key = u < key ? u : key;
        }
        const int q = simt::query_of(p, i);
        if ((lane & 7) == 0 && key != ~0ull && q0 + q < nq) {
            const int32_t pos = sh.row[q];
            atomicMin(&row_keys[ids ? ids[pos] : pos], key);
        }
    }
}

__global__ void __launch_bounds__(simt::THREADS, simt::CTAS_PER_SM) candidates_fp32_kernel(
    const float *__restrict__ data, const float *__restrict__ core,
    const int32_t *__restrict__ labels, const int32_t *__restrict__ ids, int64_t n, int d,
    const int32_t *__restrict__ tile_lo, const int32_t *__restrict__ tile_hi, int64_t ref_chunk,
    unsigned long long *__restrict__ row_keys, const int32_t *__restrict__ qmap, int64_t nq,
    int64_t qoff) {
    extern __shared__ __align__(16) float smem[];
    const int64_t r_begin = (int64_t)blockIdx.y * ref_chunk;
    const int64_t r_end = r_begin + ref_chunk < n ? r_begin + ref_chunk : n;
    candidates_block(data, core, labels, ids, n, d, tile_lo, tile_hi, (int64_t)blockIdx.x * QT,
                     r_begin, r_end, row_keys, qmap, nq, qoff, smem);
}

__global__ void __launch_bounds__(simt::THREADS, simt::CTAS_PER_SM) candidates_pruned_kernel(
    const float *__restrict__ data, const float *__restrict__ core,
    const int32_t *__restrict__ labels, const int32_t *__restrict__ ids, int64_t n, int d,
    const int32_t *__restrict__ tile_lo, const int32_t *__restrict__ tile_hi, int64_t ref_chunk,
    unsigned long long *__restrict__ row_keys, const int32_t *__restrict__ qmap, int64_t nq,
    const CandPrune prune) {
    extern __shared__ __align__(16) float smem[];
    const int64_t r_begin = (int64_t)blockIdx.y * ref_chunk;
    const int64_t r_end = r_begin + ref_chunk < n ? r_begin + ref_chunk : n;
    candidates_block<true>(data, core, labels, ids, n, d, tile_lo, tile_hi, (int64_t)blockIdx.x * QT,
                           r_begin, r_end, row_keys, qmap, nq, 0, smem, prune);
}

// Packed fits: fit blockIdx.z (skipped unless its round runs), query tile blockIdx.x,
// reference chunk blockIdx.y of `splits`, over the fit's component-sorted copies (the launch
// launch_candidates_fp32 makes for a fit alone).
__global__ void __launch_bounds__(simt::THREADS, simt::CTAS_PER_SM)
    pack_candidates_kernel(const PackFit *__restrict__ fits, int splits) {
    extern __shared__ __align__(16) float smem[];
    const PackFit &f = fits[blockIdx.z];
    const int64_t n = f.n, q0 = (int64_t)blockIdx.x * QT;
    if (q0 >= n || !*(volatile int32_t *)&f.kept_total[1]) return;
    const int64_t chunk =
        ceil_div(ceil_div(n, (int64_t)splits), (int64_t)simt::RT) * simt::RT;
    const int64_t r_begin = (int64_t)blockIdx.y * chunk;
    if (r_begin >= n) return;
    const int64_t r_end = r_begin + chunk < n ? r_begin + chunk : n;
    candidates_block(f.xp, f.corep, f.labp, f.perm, n, f.d, f.tile_lo, f.tile_hi, q0, r_begin,
                     r_end, f.row_keys, nullptr, n, 0, smem);
}

__global__ void fill_u64_kernel(unsigned long long *p, int64_t n, unsigned long long v) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = v;
}

__global__ void keys_to_candidates_kernel(const unsigned long long *__restrict__ keys, int64_t n,
                                          float *__restrict__ w, int32_t *__restrict__ dst) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    unsigned long long k = keys[i];
    if (k == ~0ull) {
        w[i] = CUSCAN_INF;
        dst[i] = (int32_t)n;
    } else {
        w[i] = __uint_as_float((uint32_t)(k >> 32));
        dst[i] = (int32_t)(uint32_t)k;
    }
}

// ---- CSR component reduction (component_reduce.rs semantics) ----

struct Fold {
    uint32_t key, bits, source, bad;
};

__device__ __forceinline__ void fold_take(Fold &a, const Fold &b) {
    if (b.key < a.key || (b.key == a.key && b.source < a.source)) {
        a.key = b.key;
        a.bits = b.bits;
        a.source = b.source;
    }
    a.bad = b.bad < a.bad ? b.bad : a.bad;
}

__device__ __forceinline__ Fold warp_fold(Fold v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        Fold u;
        u.key = __shfl_xor_sync(0xffffffffu, v.key, o);
        u.bits = __shfl_xor_sync(0xffffffffu, v.bits, o);
        u.source = __shfl_xor_sync(0xffffffffu, v.source, o);
        u.bad = __shfl_xor_sync(0xffffffffu, v.bad, o);
        fold_take(v, u);
    }
    return v;
}

// One warp per tile of CSR positions [tile_starts[t], tile_ends[t]).
__global__ void reduce_tiles_kernel(const float *__restrict__ weights,
                                    const int32_t *__restrict__ indices,
                                    const int32_t *__restrict__ members,
                                    const int32_t *__restrict__ starts,
                                    const int32_t *__restrict__ ends, int64_t p, uint32_t n,
                                    Fold *__restrict__ partial) {
    int64_t t = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32;
    int lane = threadIdx.x & 31;
    if (t >= p) return;
    Fold acc{0xffffffffu, 0x7f800000u, n, n};
    // a malformed plan is clamped to the member array [0, n) and to member ids below n, so
    // it never reads outside the caller's buffers (a valid plan is unaffected)
    const int64_t lo = starts[t] > 0 ? starts[t] : 0;
    const int64_t hi = (int64_t)ends[t] < (int64_t)n ? (int64_t)ends[t] : (int64_t)n;
    for (int64_t pos = lo + lane; pos < hi; pos += 32) {
        uint32_t member = (uint32_t)members[pos];
        if (member >= n) continue;
        uint32_t original = __float_as_uint(weights[member]);
        int32_t destination = indices[member];
        Fold v{0xffffffffu, 0x7f800000u, n, n};
        if (numerical_bits(original) || destination >= (int32_t)n) {
            v.bad = member;
        } else if (destination >= 0) {
            v.key = (original & 0x7fffffffu) == 0 ? 0u : original;
            v.bits = original;
            v.source = member;
        }
        fold_take(acc, v);
    }
    acc = warp_fold(acc);
    if (lane == 0) partial[t] = acc;
}

// One warp per component over its tile partials; writes winner weight and 5-int metadata.
__global__ void reduce_components_kernel(const float *__restrict__ weights,
                                         const int32_t *__restrict__ indices,
                                         const int32_t *__restrict__ partial_offsets,
                                         const Fold *__restrict__ partial, int64_t c, int64_t p,
                                         uint32_t n, float *__restrict__ win_w,
                                         int32_t *__restrict__ win_meta) {
    int64_t s = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32;
    int lane = threadIdx.x & 31;
    if (s >= c) return;
    Fold acc{0xffffffffu, 0x7f800000u, n, n};
    // partials of a malformed plan outside [0, p) are not read (a valid plan is unaffected)
    const int64_t lo = partial_offsets[s] > 0 ? partial_offsets[s] : 0;
    const int64_t hi = partial_offsets[s + 1] < p ? partial_offsets[s + 1] : p;
    for (int64_t t = lo + lane; t < hi; t += 32)
        fold_take(acc, partial[t]);
    acc = warp_fold(acc);
    if (lane != 0) return;
    int32_t destination = acc.source < n ? indices[acc.source] : -1;
    int32_t kind = 0, bad_destination = -1;
    if (acc.bad < n) {
        if (numerical_bits(__float_as_uint(weights[acc.bad]))) {
            kind = 1;
        } else {
            kind = 2;
            bad_destination = indices[acc.bad];
        }
    }
    win_w[s] = __uint_as_float(acc.bits);
    int32_t *m = win_meta + s * 5;
    m[0] = acc.source < n ? (int32_t)acc.source : -1;
    m[1] = destination;
    m[2] = (int32_t)acc.bad;
    m[3] = kind;
    m[4] = bad_destination;
}

}  // namespace

int launch_tile_ranges(cuscan_ctx *ctx, const int32_t *labels, int64_t n, int32_t *tile_lo,
                       int32_t *tile_hi, cudaStream_t s) {
    const int64_t tiles = ceil_div(n, RT);
    CUSCAN_KERNEL(tile_range_kernel, (unsigned)ceil_div(tiles, 256), 256, 0, s, labels, n,
                  tile_lo, tile_hi);
    CUSCAN_LAUNCH(ctx, "tile_range_kernel");
    return CUSCAN_OK;
}

int launch_candidates_fp32(cuscan_ctx *ctx, const float *data, const float *core_sq,
                           const int32_t *labels, const int32_t *ids, int64_t n, int d,
                           unsigned long long *row_keys, int32_t *tile_lo, int32_t *tile_hi,
                           cudaStream_t s, const int32_t *qmap, int64_t nq, int64_t qoff,
                           bool ranges_ready, const TileBounds *bounds, const uint32_t *cbound) {
    if (!qmap && qoff == 0 && nq == 0) nq = n;
    if (nq == 0) return CUSCAN_OK;
    if (!ranges_ready)
        if (int rc = launch_tile_ranges(ctx, labels, n, tile_lo, tile_hi, s)) return rc;
    if (d > CUSCAN_PACK_MAX_FEATURES)
        return fail(ctx, CUSCAN_CAPACITY,
                    "feature count %d exceeds the shared-memory staging limit of the Boruvka "
                    "kernel (at most 256 features)", d);
    const int64_t qtiles = ceil_div(nq, (int64_t)QT);
    int64_t splits = 1, chunk = 0;
    simt::split_plan(ctx->sm_count, qtiles, n, 2, 1.0, splits, chunk);
    if (int rc = allow_dynamic_smem(ctx, candidates_fp32_kernel, kCandSmem)) return rc;
    const dim3 grid((unsigned)qtiles, (unsigned)splits);
    if (bounds) {
        if (int rc = allow_dynamic_smem(ctx, candidates_pruned_kernel, kCandSmem)) return rc;
        CandPrune prune{*bounds, cbound, nullptr, (int)mask_words(n)};
        Buffer &masks = ctx->fit->forest.refined.masks;
        if (const size_t bytes = mask_bytes(n)) {
            const size_t smem = mask_smem(d, prune.words);
            int rc = ensure(ctx, masks, bytes, "tile masks");
            if (!rc) rc = allow_dynamic_smem(ctx, candidate_masks_kernel, smem);
            if (rc && rc != CUSCAN_MEMORY) return rc;
            if (rc) {  // no room: the balls alone
                clear_error(ctx);
            } else {
                prune.masks = as<uint32_t>(masks);
                CUSCAN_KERNEL(candidate_masks_kernel, (unsigned)qtiles, MASK_THREADS, smem, s, data,
                              labels, d, qmap, nq, *bounds, cbound, prune.words,
                              as<uint32_t>(masks));
            }
        }
        CUSCAN_KERNEL(candidates_pruned_kernel, grid, simt::THREADS, kCandSmem, s, data, core_sq,
                      labels, ids, n, d, tile_lo, tile_hi, chunk, row_keys, qmap, nq, prune);
        CUSCAN_LAUNCH(ctx, "candidates_pruned_kernel");
        return CUSCAN_OK;
    }
    CUSCAN_KERNEL(candidates_fp32_kernel, grid, simt::THREADS, kCandSmem, s, data, core_sq, labels, ids, n, d,
                  tile_lo, tile_hi, chunk, row_keys, qmap, nq, qoff);
    CUSCAN_LAUNCH(ctx, "candidates_fp32_kernel");
    return CUSCAN_OK;
}

int launch_pack_candidates(cuscan_ctx *ctx, const PackFit *fits, int count, int64_t n_max,
                           int d_max, int splits, cudaStream_t s) {
    if (d_max > CUSCAN_PACK_MAX_FEATURES)
        return fail(ctx, CUSCAN_CAPACITY, "feature count %d exceeds the Boruvka staging limit",
                    d_max);
    if (int rc = allow_dynamic_smem(ctx, pack_candidates_kernel, kCandSmem)) return rc;
    const dim3 grid((unsigned)ceil_div(n_max, (int64_t)QT), (unsigned)splits, (unsigned)count);
    CUSCAN_KERNEL(pack_candidates_kernel, grid, simt::THREADS, kCandSmem, s, fits, splits);
    CUSCAN_LAUNCH(ctx, "pack_candidates_kernel");
    return CUSCAN_OK;
}

int launch_fill_u64(cuscan_ctx *ctx, unsigned long long *p, int64_t n, unsigned long long v,
                    cudaStream_t s) {
    if (n <= 0) return CUSCAN_OK;
    CUSCAN_KERNEL(fill_u64_kernel, (unsigned)ceil_div(n, 256), 256, 0, s, p, n, v);
    CUSCAN_LAUNCH(ctx, "fill_u64_kernel");
    return CUSCAN_OK;
}

int launch_keys_to_candidates(cuscan_ctx *ctx, const unsigned long long *keys, int64_t n,
                              float *w, int32_t *dst, cudaStream_t s) {
    CUSCAN_KERNEL(keys_to_candidates_kernel, (unsigned)ceil_div(n, 256), 256, 0, s, keys, n, w, dst);
    CUSCAN_LAUNCH(ctx, "keys_to_candidates_kernel");
    return CUSCAN_OK;
}

int launch_component_reduce(cuscan_ctx *ctx, const float *weights, const int32_t *indices,
                            const int32_t *members, const int32_t *starts, const int32_t *ends,
                            const int32_t *partial_offsets, int64_t n, int64_t p, int64_t c,
                            float *win_w, int32_t *win_meta, Buffer &scratch, cudaStream_t s) {
    if (c == 0) return CUSCAN_OK;
    int rc = ensure(ctx, scratch, (size_t)(p > 0 ? p : 1) * sizeof(Fold), "component partials");
    if (rc) return rc;
    if (p > 0) {
        CUSCAN_KERNEL(reduce_tiles_kernel, (unsigned)ceil_div(p * 32, 256), 256, 0, s, 
            weights, indices, members, starts, ends, p, (uint32_t)n, as<Fold>(scratch));
        CUSCAN_LAUNCH(ctx, "reduce_tiles_kernel");
    }
    CUSCAN_KERNEL(reduce_components_kernel, (unsigned)ceil_div(c * 32, 256), 256, 0, s, 
        weights, indices, partial_offsets, as<Fold>(scratch), c, p, (uint32_t)n, win_w, win_meta);
    CUSCAN_LAUNCH(ctx, "reduce_components_kernel");
    return CUSCAN_OK;
}

// ---------------------------------------------------------------------------------------------
// Component reduction without any device allocation.
//
// Some callers cannot allocate device memory at the moment they need this reduction: a host
// whose device memory is owned by another framework's caching pool, a real-time loop that must
// not take the implicit synchronisation of cudaMalloc/cudaFree, or a plugin that is handed
// device buffers and nothing else. For them the per-tile partial results live in a fixed
// array of static device memory that the CUDA module owns: every GPU that loads this library
// keeps NOALLOC_MAX_TILES * 16 bytes (1 MiB) for it until the process exits.
// ---------------------------------------------------------------------------------------------
namespace {

constexpr int64_t NOALLOC_MAX_TILES = 65536;  // == CUSCAN_NOALLOC_MAX_TILES in the header

static __device__ __align__(256) Fold g_noalloc_partials[NOALLOC_MAX_TILES];

// The array's address on each device. In host code the symbol is only a host-side stand-in;
// the device address is fetched once per device with that device current.
std::mutex g_noalloc_mutex;
Fold *g_noalloc_ptr[64] = {};

void set_err(char *err, size_t len, const char *msg) {
    if (err && len) {
        snprintf(err, len, "%s", msg);
    }
}

}  // namespace

}  // namespace cuscan

extern "C" int cuscan_component_reduce_noalloc(
    const float *weights, const int32_t *indices, const int32_t *members,
    const int32_t *tile_starts, const int32_t *tile_ends, const int32_t *partial_offsets,
    int64_t n, int64_t p, int64_t c, float *win_weights, int32_t *win_meta, void *stream,
    char *err, size_t err_len) {
    using namespace cuscan;
    if (n < 0 || p < 0 || c < 0 || c > n || p > n) {
        set_err(err, err_len, "component_reduce_noalloc received inconsistent sizes");
        return CUSCAN_INVALID_INPUT;
    }
    if (n > INT32_MAX) {
        set_err(err, err_len, "component member index exceeds the supported integer range");
        return CUSCAN_OVERFLOW;
    }
    if (p > NOALLOC_MAX_TILES) {
        char msg[160];
        snprintf(msg, sizeof(msg),
                 "component_reduce_noalloc supports at most %lld tiles (got %lld); use "
                 "cuscan_component_reduce for larger plans",
                 (long long)NOALLOC_MAX_TILES, (long long)p);
        set_err(err, err_len, msg);
        return CUSCAN_CAPACITY;
    }
    if (c == 0) return CUSCAN_OK;
    int device = -1;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess || device < 0 || device >= 64) {
        cudaGetLastError();
        set_err(err, err_len, "no usable current CUDA device");
        return CUSCAN_BACKEND_UNAVAILABLE;
    }
    Fold *scratch = nullptr;
    {
        // first call on a device: resolve the static array's device address (done once)
        std::lock_guard<std::mutex> lock(g_noalloc_mutex);
        if (!g_noalloc_ptr[device]) {
            void *ptr = nullptr;
            e = cudaGetSymbolAddress(&ptr, g_noalloc_partials);
            if (e != cudaSuccess || !ptr) {
                cudaGetLastError();
                set_err(err, err_len, "cudaGetSymbolAddress of the static partials failed");
                return CUSCAN_BACKEND_UNAVAILABLE;
            }
            g_noalloc_ptr[device] = static_cast<Fold *>(ptr);
        }
        scratch = g_noalloc_ptr[device];
    }
    // every tile writes its own partial, so no clearing of the shared array is needed
    cudaStream_t s = (cudaStream_t)stream;
    if (p > 0) {
        CUSCAN_KERNEL(reduce_tiles_kernel, (unsigned)ceil_div(p * 32, 256), 256, 0, s, weights,
                      indices, members, tile_starts, tile_ends, p, (uint32_t)n, scratch);
    }
    CUSCAN_KERNEL(reduce_components_kernel, (unsigned)ceil_div(c * 32, 256), 256, 0, s, weights,
                  indices, partial_offsets, scratch, c, p, (uint32_t)n, win_weights, win_meta);
    e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_err(err, err_len, cudaGetErrorString(e));
        return CUSCAN_BACKEND_UNAVAILABLE;
    }
    return CUSCAN_OK;
}
