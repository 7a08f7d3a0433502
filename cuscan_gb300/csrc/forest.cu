// Exact integer work of the MST on the device: the kNN seed forest, per-round component
// winners, cycle breaking that reproduces the reference's sequential merge order, pointer
// jumping union/relabel, component sorting and an exclusive scan.
//
// Why cycle breaking is enough. In both the seed (crates/hdbscan-core/src/mst.rs:368-420) and
// a Borůvka merge (mst.rs:259-277) every node (a point, or a component slot) proposes at most
// one edge, so the proposals form a functional graph: each weakly connected part is a tree
// (one node without a proposal) or has exactly one cycle. The reference walks the proposals in
// slot order and skips an edge whose endpoints are already joined. An edge is skipped only if
// the edges processed before it already connect its endpoints, which closes the part's only
// cycle, so exactly one edge per cycle is skipped: the cycle edge with the largest slot. Slots
// are numbered by first appearance, i.e. by the smallest point of a component; components are
// therefore labelled here by their smallest point, and "largest slot" is "largest label".
// Pointer doubling with a running maximum finds, for every node, a node on its cycle and the
// cycle's largest label, without any sequential pass.
#include "common.cuh"
#include "forest.cuh"

namespace cuscan {
namespace {

constexpr int SMALL_RANGE = 32;  // rows per label range of the candidate sweep

__device__ __forceinline__ int log2_ceil_dev(int64_t c) {
    int l = 0;
    while ((1ll << l) < c) ++l;
    return l;
}

__device__ __forceinline__ bool active_node(const int32_t *label, int64_t s) {
    return label == nullptr || label[s] == (int32_t)s;
}

__device__ __forceinline__ void core_at(int64_t i, const float *__restrict__ knn_sq, int64_t n,
                                        int k, int min_samples, float *__restrict__ core) {
    float c;
    if ((int64_t)min_samples >= n)
        c = CUSCAN_INF;
    else if (min_samples == 1)
        c = 0.0f;
    else
        c = knn_sq[i * k + min_samples - 1];
    core[i] = c;
}

__global__ void core_kernel(const float *__restrict__ knn_sq, int64_t n, int k, int min_samples,
                            float *__restrict__ core) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) core_at(i, knn_sq, n, k, min_samples, core);
}

// Seed proposal of point i: the first non-padding neighbour j with core_i >= core_j
// (mst.rs:390-417); next[i] = i when there is none.
__device__ __forceinline__ void seed_at(int64_t i, const float *__restrict__ core,
                                        const int32_t *__restrict__ ids,
                                        const float *__restrict__ dsq, int64_t n, int k,
                                        int32_t *__restrict__ next, uint32_t *__restrict__ esrc,
                                        uint32_t *__restrict__ edst, float *__restrict__ ew,
                                        DevStatus *status) {
    const float ci = core[i];
    int32_t pick = (int32_t)i;
    float w = 0.0f;
    for (int s = 0; s < k; ++s) {
        int32_t j = ids[i * k + s];
        if (j < 0) continue;
        if ((int64_t)j >= n) {
            atomicCAS(&status->err_kind, 0, 2);
            break;
        }
        if (ci >= core[j]) {
            pick = j;
            w = fmaxf(ci, dsq[i * k + s]);
            break;
        }
    }
    next[i] = pick;
    esrc[i] = (uint32_t)i;
    edst[i] = (uint32_t)pick;
    ew[i] = w;
}

__global__ void seed_kernel(const float *__restrict__ core, const int32_t *__restrict__ ids,
                            const float *__restrict__ dsq, int64_t n, int k,
                            int32_t *__restrict__ next, uint32_t *__restrict__ esrc,
                            uint32_t *__restrict__ edst, float *__restrict__ ew,
                            int32_t *__restrict__ label, DevStatus *status) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    seed_at(i, core, ids, dsq, n, k, next, esrc, edst, ew, status);
    label[i] = (int32_t)i;  // every point is its own component before the merge
}

// Per-node steps of the cycle breaking and union (resolve_proposals). Each is run by one
// thread per node, either as a kernel of its own or inside the single-CTA steps of small fits;
// the step order and the barriers between them are the same in both.
__device__ __forceinline__ void dbl_init_at(int64_t s, const int32_t *__restrict__ next,
                                            const int32_t *__restrict__ label,
                                            int32_t *__restrict__ jmp, int32_t *__restrict__ mx) {
    if (!active_node(label, s)) return;
    jmp[s] = next[s];
    mx[s] = (int32_t)s;
}
__device__ __forceinline__ void dbl_step_at(int64_t s, const int32_t *__restrict__ jin,
                                            const int32_t *__restrict__ min_,
                                            const int32_t *__restrict__ label,
                                            int32_t *__restrict__ jout, int32_t *__restrict__ mout) {
    if (!active_node(label, s)) return;
    int32_t j = jin[s];
    jout[s] = jin[j];
    int32_t a = min_[s], b = min_[j];
    mout[s] = a > b ? a : b;
}
// keep[s] = s proposes an edge that is not its cycle's largest-label edge; parent[s] is the
// forest parent after the skipped edges are removed.
__device__ __forceinline__ void keep_at(int64_t s, const int32_t *__restrict__ next,
                                        const int32_t *__restrict__ jmp,
                                        const int32_t *__restrict__ mx,
                                        const int32_t *__restrict__ label,
                                        int32_t *__restrict__ keep, int32_t *__restrict__ parent) {
    if (!active_node(label, s)) {
        keep[s] = 0;
        return;
    }
    int32_t t = next[s];
    bool k = t != (int32_t)s && mx[jmp[s]] != (int32_t)s;
    keep[s] = k ? 1 : 0;
    parent[s] = k ? t : (int32_t)s;
}
__device__ __forceinline__ void emit_at(int64_t s, const int32_t *__restrict__ keep,
                                        const int32_t *__restrict__ pos,
                                        const uint32_t *__restrict__ esrc,
                                        const uint32_t *__restrict__ edst,
                                        const float *__restrict__ ew, int64_t edges,
                                        uint32_t *__restrict__ out_src,
                                        uint32_t *__restrict__ out_dst, float *__restrict__ out_w,
                                        int64_t capacity) {
    if (!keep[s]) return;
    int64_t at = edges + pos[s];
    if (at >= capacity) return;
    out_src[at] = esrc[s];
    out_dst[at] = edst[s];
    out_w[at] = ew[s];
}
// Path halving toward the root (in place).
__device__ __forceinline__ void jump_at(int64_t s, int32_t *__restrict__ parent,
                                        const int32_t *__restrict__ label) {
    if (!active_node(label, s)) return;
    int32_t p = parent[s];
    int32_t pp = parent[p];
    if (pp != p) parent[s] = pp;
}
__device__ __forceinline__ void minlab_init_at(int64_t s, const int32_t *__restrict__ parent,
                                               const int32_t *__restrict__ label,
                                               int32_t *__restrict__ minlab) {
    if (!active_node(label, s)) return;
    if (parent[s] == (int32_t)s) minlab[s] = (int32_t)s;
}
__device__ __forceinline__ void minlab_reduce_at(int64_t s, const int32_t *__restrict__ parent,
                                                 const int32_t *__restrict__ label,
                                                 int32_t *__restrict__ minlab) {
    if (!active_node(label, s)) return;
    atomicMin(&minlab[parent[s]], (int32_t)s);
}
// Eight doubling steps' worth of hops per launch: jout[s] is jin applied eight times, mout the
// largest label on the way (three steps of the one-hop form, whose launches were a quarter of a
// 9,001-point fit's). The first launch (jin null) starts from the proposals themselves.
constexpr int HOPS = 8;
__global__ void dbl_hops_kernel(const int32_t *__restrict__ next, const int32_t *__restrict__ jin,
                                const int32_t *__restrict__ min_, const int32_t *__restrict__ label,
                                int64_t n, int32_t *__restrict__ jout, int32_t *__restrict__ mout) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n || !active_node(label, s)) return;
    int32_t j = (int32_t)s, m = (int32_t)s;
#pragma unroll
    for (int h = 0; h < HOPS; ++h) {
        const int32_t a = jin ? min_[j] : j;
        m = a > m ? a : m;
        j = jin ? jin[j] : next[j];
    }
    jout[s] = j;
    mout[s] = m;
}

// keep_at, and the label minima of the roots (their own label) for minlab_reduce_kernel.
__global__ void keep_kernel(const int32_t *__restrict__ next, const int32_t *__restrict__ jmp,
                            const int32_t *__restrict__ mx, const int32_t *__restrict__ label,
                            int64_t n, int32_t *__restrict__ keep, int32_t *__restrict__ parent,
                            int32_t *__restrict__ minlab) {
    int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    keep_at(s, next, jmp, mx, label, keep, parent);
    if (!keep[s]) minlab[s] = (int32_t)s;  // a root (or an inactive node, whose entry is not read)
}

__global__ void emit_kernel(const int32_t *__restrict__ keep, const int32_t *__restrict__ pos,
                            const int32_t *__restrict__ sums, const uint32_t *__restrict__ esrc,
                            const uint32_t *__restrict__ edst, const float *__restrict__ ew,
                            int64_t n, const DevStatus *status, uint32_t *__restrict__ out_src,
                            uint32_t *__restrict__ out_dst, float *__restrict__ out_w,
                            int64_t capacity) {
    int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    emit_at(s, keep, pos, esrc, edst, ew, (int64_t)status->edges + sums[s / kScanTile], out_src,
            out_dst, out_w, capacity);
}

// Eight hops toward the root per launch, in place: a parent read while another thread moves it
// is an ancestor either way, so every launch at least multiplies the depth covered by eight.
__global__ void jump_kernel(int32_t *__restrict__ parent, const int32_t *__restrict__ label,
                            int64_t n) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n || !active_node(label, s)) return;
    const volatile int32_t *vp = parent;
    const int32_t p = vp[s];
    int32_t q = p;
#pragma unroll
    for (int h = 1; h < HOPS; ++h) {
        const int32_t up = vp[q];
        if (up == q) break;
        q = up;
    }
    if (q != p) parent[s] = q;
}

// minlab_reduce_at; one thread also adds the emitted edges to the status and clears the component
// count for relabel_kernel.
__global__ void minlab_reduce_kernel(const int32_t *__restrict__ parent,
                                     const int32_t *__restrict__ label, int64_t n,
                                     int32_t *__restrict__ minlab, DevStatus *status,
                                     const int32_t *kept_total, int require_progress) {
    int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s < n) minlab_reduce_at(s, parent, label, minlab);
    if (s == 0) {
        status->edges += *kept_total;
        status->components = 0;
        // "Boruvka round made no progress" (mst.rs:279-283)
        if (require_progress && *kept_total == 0) atomicCAS(&status->err_kind, 0, 4);
    }
}

// label[i] <- smallest label of the tree that holds i's old component; counts the components (the
// points that carry their own label).
__global__ void relabel_kernel(int32_t *__restrict__ label, const int32_t *__restrict__ parent,
                               const int32_t *__restrict__ minlab, int64_t n, DevStatus *status) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool root = false;
    if (i < n) {
        const int32_t l = minlab[parent[label[i]]];
        label[i] = l;
        root = l == (int32_t)i;
    }
    const int roots = __syncthreads_count(root);
    if (threadIdx.x == 0 && roots) atomicAdd(&status->components, (unsigned long long)roots);
}

// Start of a component sort: empty histogram and cursors, empty row and component keys for the
// round that follows, the scan's ticket and, where the sort counts them, the pair sum. The ticket
// is cleared by every sort: sorts outside a fit (sort_by_cells of a set's kNN or of a predictor's
// rows) run on a status block that nothing else has written.
__global__ void sort_clear_kernel(int32_t *__restrict__ cnt, int32_t *__restrict__ fill,
                                  unsigned long long *__restrict__ row_keys,
                                  unsigned long long *__restrict__ comp_keys, int64_t n,
                                  DevStatus *status, bool counts_pairs) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) {
        status->scan_ticket = 0;
        if (counts_pairs) status->same_pairs = 0.0;
    }
    if (i >= n) return;
    cnt[i] = 0;
    fill[i] = 0;
    row_keys[i] = ~0ull;
    comp_keys[i] = ~0ull;
}

// Labels and cores in the fit's spatial order, and the histogram of the labels.
__global__ void label_cells_kernel(const int32_t *__restrict__ label, const float *__restrict__ core,
                                   const int32_t *__restrict__ perm, int64_t n,
                                   int32_t *__restrict__ cnt, int32_t *__restrict__ labp,
                                   float *__restrict__ corep) {
    const int64_t pos = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int32_t l = -1;
    if (pos < n) {
        const int32_t i = perm[pos];
        l = label[i];
        labp[pos] = l;
        corep[pos] = core[i];
    }
    const unsigned peers = __match_any_sync(0xffffffffu, l);
    if (l >= 0 && (int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&cnt[l], __popc(peers));
}

// Counting sort of points by label: histogram with warp-aggregated atomics.
__global__ void hist_kernel(const int32_t *__restrict__ label, int64_t n, int32_t *__restrict__ cnt) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int32_t l = i < n ? label[i] : -1;
    unsigned peers = __match_any_sync(0xffffffffu, l);
    int lane = threadIdx.x & 31;
    if (l >= 0 && lane == __ffs(peers) - 1) atomicAdd(&cnt[l], __popc(peers));
}

// Histogram of the labels and flags of the roots (points that carry their own label).
__global__ void hist_roots_kernel(const int32_t *__restrict__ label, int64_t n,
                                  int32_t *__restrict__ cnt, int32_t *__restrict__ root) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int32_t l = i < n ? label[i] : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, l);
    if (l >= 0 && (int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&cnt[l], __popc(peers));
    if (i < n) root[i] = l == (int32_t)i;
}

// Level of a squared norm within the rows' range.
__device__ __forceinline__ int norm_level(float p, const unsigned int *range, int levels) {
    const float lo = __uint_as_float(range[0]), hi = __uint_as_float(range[1]);
    const float t = (p - lo) / (hi - lo) * (float)levels;  // NaN (one norm, overflow): level 0
    return t >= (float)levels ? levels - 1 : t > 0.0f ? (int)t : 0;
}

__global__ void norm_keys_kernel(const int32_t *__restrict__ label, const int32_t *__restrict__ rank,
                                 const int32_t *__restrict__ sums, const int32_t *__restrict__ cnt,
                                 const float *__restrict__ rnorm,
                                 const unsigned int *__restrict__ range, int64_t n, int levels,
                                 int32_t *__restrict__ key, DevStatus *status) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    double sq = 0.0;
    if (i < n) {
        const int32_t l = label[i];
        key[i] = (rank[l] + sums[l / kScanTile]) * levels + norm_level(rnorm[i], range, levels);
        sq = (double)cnt[i] * (double)cnt[i];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    if ((threadIdx.x & 31) == 0 && sq != 0.0) atomicAdd(&status->same_pairs, sq);
}

__global__ void cell_keys_kernel(const int32_t *__restrict__ cell, const float *__restrict__ rnorm,
                                 const unsigned int *__restrict__ range, int64_t n, int levels,
                                 int32_t *__restrict__ key) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) key[i] = cell[i] * levels + norm_level(rnorm[i], range, levels);
}

__global__ void scatter_kernel(const int32_t *__restrict__ label, int64_t n,
                               const int32_t *__restrict__ start,
                               const int32_t *__restrict__ sums, int32_t *__restrict__ fill,
                               int32_t *__restrict__ perm) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int32_t l = i < n ? label[i] : -1;
    unsigned peers = __match_any_sync(0xffffffffu, l);
    int lane = threadIdx.x & 31;
    int leader = __ffs(peers) - 1;
    int base = 0;
    if (l >= 0 && lane == leader) base = atomicAdd(&fill[l], __popc(peers));
    base = __shfl_sync(peers, base, leader);
    if (l < 0) return;
    int rank = __popc(peers & ((1u << lane) - 1u));
    perm[start[l] + sums[l / kScanTile] + base + rank] = (int32_t)i;
}

__global__ void gather_kernel(const float *__restrict__ x, const float *__restrict__ core,
                              const int32_t *__restrict__ label, const int32_t *__restrict__ perm,
                              int64_t n, int d, float *__restrict__ xp, float *__restrict__ corep,
                              int32_t *__restrict__ labp) {
    int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n * d) return;
    int64_t pos = e / d;
    int f = (int)(e - pos * d);
    int32_t i = perm[pos];
    xp[e] = x[(int64_t)i * d + f];
    if (f == 0) {
        if (core) corep[pos] = core[i];
        labp[pos] = label[i];
    }
}

// gather_kernel for rows of 16-byte pieces (d a multiple of 4, aligned rows): a thread per piece. What
// bounds it is HBM and the latency of the row index: 500,000 x 128 107 us against 322 us with
// a thread per element.
__global__ void gather4_kernel(const float4 *__restrict__ x, const float *__restrict__ core,
                               const int32_t *__restrict__ label, const int32_t *__restrict__ perm,
                               int64_t pieces, unsigned per_row, float4 *__restrict__ xp,
                               float *__restrict__ corep, int32_t *__restrict__ labp) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= pieces) return;
    const int64_t pos = e / per_row;
    const unsigned c = (unsigned)(e - pos * per_row);
    const int32_t i = perm[pos];
    xp[e] = x[(int64_t)i * per_row + c];
    if (c == 0) {
        if (core) corep[pos] = core[i];
        labp[pos] = label[i];
    }
}

// Per-component minimum of (row weight bits << 32 | row) over component-sorted positions:
// segmented warp reduction over the contiguous label runs, one atomic per run.
// Component key of the row at sorted position pos: (weight bits << 32 | row), ~0 for a row
// without a candidate (an error unless allow_empty) or with a non-finite weight (an error).
__device__ __forceinline__ unsigned long long comp_key_at(int64_t pos,
                                                          const int32_t *__restrict__ perm,
                                                          const unsigned long long *__restrict__ row_keys,
                                                          DevStatus *status, int allow_empty) {
    const int32_t i = perm[pos];
    const unsigned long long rk = row_keys[i];
    if (rk == ~0ull) {
        if (!allow_empty) atomicCAS(&status->err_kind, 0, 4);
        return ~0ull;
    }
    const uint32_t wb = (uint32_t)(rk >> 32);
    if (numerical_bits(wb)) {
        atomicCAS(&status->err_kind, 0, 1);
        return ~0ull;
    }
    return ((unsigned long long)wb << 32) | (uint32_t)i;
}

__global__ void component_min_kernel(const int32_t *__restrict__ perm,
                                     const int32_t *__restrict__ labp,
                                     const unsigned long long *__restrict__ row_keys, int64_t n,
                                     unsigned long long *__restrict__ comp_keys,
                                     DevStatus *status, int allow_empty) {
    int64_t pos = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    int32_t l = -1;
    unsigned long long v = ~0ull;
    if (pos < n) {
        l = labp[pos];
        v = comp_key_at(pos, perm, row_keys, status, allow_empty);
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned long long ov = __shfl_down_sync(0xffffffffu, v, o);
        int32_t ol = __shfl_down_sync(0xffffffffu, l, o);
        if (lane + o < 32 && ol == l && ov < v) v = ov;
    }
    int32_t prev = __shfl_up_sync(0xffffffffu, l, 1);
    bool head = l >= 0 && (lane == 0 || prev != l);
    if (head && v != ~0ull) atomicMin(&comp_keys[l], v);
}

// Winner of each active component: source = argmin row, destination = that row's candidate.
__device__ __forceinline__ void winner_at(int64_t s, const int32_t *label,
                                          const unsigned long long *__restrict__ comp_keys,
                                          const unsigned long long *__restrict__ row_keys,
                                          int64_t n, int32_t *__restrict__ next,
                                          uint32_t *__restrict__ esrc, uint32_t *__restrict__ edst,
                                          float *__restrict__ ew, DevStatus *status) {
    if (label[s] != (int32_t)s) return;
    unsigned long long ck = comp_keys[s];
    if (ck == ~0ull) {
        atomicCAS(&status->err_kind, 0, 4);
        next[s] = (int32_t)s;
        return;
    }
    uint32_t src = (uint32_t)ck;
    uint32_t dst = (uint32_t)row_keys[src];
    if ((int64_t)dst >= n) {
        atomicCAS(&status->err_kind, 0, 2);
        next[s] = (int32_t)s;
        return;
    }
    next[s] = label[dst];
    esrc[s] = src;
    edst[s] = dst;
    ew[s] = __uint_as_float((uint32_t)(ck >> 32));
}

__global__ void winner_kernel(const int32_t *__restrict__ label,
                              const unsigned long long *__restrict__ comp_keys,
                              const unsigned long long *__restrict__ row_keys, int64_t n,
                              int32_t *__restrict__ next, uint32_t *__restrict__ esrc,
                              uint32_t *__restrict__ edst, float *__restrict__ ew,
                              DevStatus *status) {
    int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s < n) winner_at(s, label, comp_keys, row_keys, n, next, esrc, edst, ew, status);
}

// ---- exclusive scan of int32: one launch; readers add their tile's offset ----
constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 4;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;
static_assert(SCAN_TILE == kScanTile, "tile of the scan offsets");

template <int THREADS = SCAN_THREADS>
__device__ __forceinline__ int block_exclusive_scan(int v, int *warp_sums, int &total) {
    static_assert(THREADS <= 1024, "one warp scans the warp sums");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int w = lane < (THREADS / 32) ? warp_sums[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < (THREADS / 32)) warp_sums[lane] = w;
    }
    __syncthreads();
    int warp_prefix = warp > 0 ? warp_sums[warp - 1] : 0;
    total = warp_sums[THREADS / 32 - 1];
    __syncthreads();
    return warp_prefix + x - v;
}

// Every block scans one tile into out and its total into tile_sums; the block that finishes last
// scans the totals (entry i's position is out[i] + tile_sums[i / kScanTile]). With `square_sum`
// the sum of squared inputs is added to it (exact in f64: integers below 2^53). The ticket wraps
// back to 0.
__global__ void __launch_bounds__(SCAN_THREADS)
    scan_kernel(const int32_t *__restrict__ in, int32_t *__restrict__ out, int64_t n,
                int32_t *tile_sums, int32_t *__restrict__ grand_total, DevStatus *status,
                double *square_sum) {
    __shared__ int warp_sums[SCAN_THREADS / 32];
    __shared__ double pair_sums[SCAN_THREADS / 32];
    __shared__ bool last;
    const int tid = threadIdx.x;
    const int64_t base = (int64_t)blockIdx.x * SCAN_TILE + (int64_t)tid * SCAN_ITEMS;
    int v[SCAN_ITEMS];
    int sum = 0;
    double sq = 0.0;
#pragma unroll
    for (int t = 0; t < SCAN_ITEMS; ++t) {
        v[t] = base + t < n ? in[base + t] : 0;
        sum += v[t];
        sq += (double)v[t] * (double)v[t];
    }
    int total;
    int prefix = block_exclusive_scan(sum, warp_sums, total);
#pragma unroll
    for (int t = 0; t < SCAN_ITEMS; ++t) {
        if (base + t < n) out[base + t] = prefix;
        prefix += v[t];
    }
    if (square_sum) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        if ((tid & 31) == 0) pair_sums[tid >> 5] = sq;
        __syncthreads();
        if (tid == 0) {
            double t = 0.0;
            for (int w = 0; w < SCAN_THREADS / 32; ++w) t += pair_sums[w];
            if (t != 0.0) atomicAdd(square_sum, t);
        }
    }
    if (tid == 0) {
        tile_sums[blockIdx.x] = total;
        __threadfence();
        last = atomicInc(&status->scan_ticket, gridDim.x - 1) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    int carry = 0;
    for (int64_t b = 0; b < gridDim.x; b += SCAN_THREADS) {
        const int64_t i = b + tid;
        const int x = i < gridDim.x ? __ldcg(tile_sums + i) : 0;
        int sums;
        const int p = block_exclusive_scan(x, warp_sums, sums);
        if (i < gridDim.x) tile_sums[i] = carry + p;
        carry += sums;
    }
    if (tid == 0 && grand_total) *grand_total = carry;
}

// ---- forests of fewer than 2048 points: each step of a fit in one CTA ----
//
// The same per-node steps in the same order as the kernel sequences below, with block barriers
// where the sequences have kernel boundaries, on arrays in shared memory. What bounds them is the
// chain of dependent loads and barriers (two per pointer-doubling or path-halving step, 24 steps
// at 2,000 points), so the arrays sit where a load takes tens of cycles instead of an L2 trip, and
// 1,024 threads (256 up to 512 rows) take two nodes each. Measured in a pack of eight fits of 500 to
// 2,047 rows on a GB300, against 256 threads on global arrays: seed 16.4 us (41.0), sort 10.9 us
// (18.6), merge 11.2 us (26.3).
constexpr int64_t SMALL_ROWS = 2048;  // nodes the arrays hold; fits of fewer points take this form
constexpr int SMALL_THREADS = 1024;
constexpr int SMALL_ITEMS = (int)(SMALL_ROWS / SMALL_THREADS);
// Fits of few rows take fewer threads, whose barriers cost less: a pack of 5, 9 and 30 rows 191 us
// instead of 201 us, eight fits of 250 rows 359 us instead of 371 us (128 threads 192 and 370 us).
constexpr int TINY_THREADS = 256;
constexpr int64_t TINY_ROWS = SMALL_ITEMS * (int64_t)TINY_THREADS;
inline int small_threads(int64_t n) { return n <= TINY_ROWS ? TINY_THREADS : SMALL_THREADS; }
// The instance of a one-CTA kernel for fits of up to n rows.
#define CUSCAN_SMALL(kernel, n) ((n) <= TINY_ROWS ? kernel<TINY_THREADS> : kernel<SMALL_THREADS>)

struct SmallForest {
    unsigned long long *comp_keys;
    int32_t *next, *ja, *ma, *jb, *mb, *keep, *pos, *parent, *minlab, *label;
    uint32_t *esrc, *edst;
    float *ew;
};
constexpr size_t kSmallSmem = (size_t)SMALL_ROWS * (8 + 13 * 4);
__device__ __forceinline__ SmallForest small_forest(void *smem) {
    SmallForest f;
    f.comp_keys = reinterpret_cast<unsigned long long *>(smem);
    int32_t *p = reinterpret_cast<int32_t *>(f.comp_keys + SMALL_ROWS);
    auto take = [&p]() {
        int32_t *at = p;
        p += SMALL_ROWS;
        return at;
    };
    f.next = take();
    f.ja = take();
    f.ma = take();
    f.jb = take();
    f.mb = take();
    f.keep = take();
    f.pos = take();
    f.parent = take();
    f.minlab = take();
    f.label = take();
    f.esrc = reinterpret_cast<uint32_t *>(take());
    f.edst = reinterpret_cast<uint32_t *>(take());
    f.ew = reinterpret_cast<float *>(take());
    return f;
}

// Cycle breaking, emit and union of the proposals in F.next/esrc/edst/ew (resolve_proposals).
// The points' labels are F.label, which are also the active labels of a round; the seed
// (active_label null) starts from labels 0..n-1. New labels leave to point_label.
template <int T>
__device__ __forceinline__ void resolve_block(const SmallForest &F, const int32_t *active_label,
                                              int32_t *__restrict__ point_label, int64_t n,
                                              int steps, DevStatus *status,
                                              uint32_t *__restrict__ out_src,
                                              uint32_t *__restrict__ out_dst,
                                              float *__restrict__ out_w, int64_t capacity,
                                              int require_progress) {
    __shared__ int warp_sums[T / 32];
    const int tid = threadIdx.x;
    int32_t *ja = F.ja, *ma = F.ma, *jb = F.jb, *mb = F.mb;
    // cycle breaking: pointer doubling with a running maximum, ping-pong buffers
    for (int64_t s = tid; s < n; s += T) dbl_init_at(s, F.next, active_label, ja, ma);
    __syncthreads();
    for (int t = 0; t < steps; ++t) {
        for (int64_t s = tid; s < n; s += T)
            dbl_step_at(s, ja, ma, active_label, jb, mb);
        __syncthreads();
        int32_t *tj = ja, *tm = ma;
        ja = jb;
        ma = mb;
        jb = tj;
        mb = tm;
    }
    for (int64_t s = tid; s < n; s += T)
        keep_at(s, F.next, ja, ma, active_label, F.keep, F.parent);
    __syncthreads();
    // exclusive scan of keep in node order: thread t holds nodes [t SMALL_ITEMS, +SMALL_ITEMS)
    int v[SMALL_ITEMS];
    int sum = 0;
    const int64_t base = (int64_t)tid * SMALL_ITEMS;
#pragma unroll
    for (int u = 0; u < SMALL_ITEMS; ++u) {
        v[u] = base + u < n ? F.keep[base + u] : 0;
        sum += v[u];
    }
    int total;
    int prefix = block_exclusive_scan<T>(sum, warp_sums, total);
#pragma unroll
    for (int u = 0; u < SMALL_ITEMS; ++u) {
        if (base + u < n) F.pos[base + u] = prefix;
        prefix += v[u];
    }
    __syncthreads();
    // append the kept edges in node order after the edges emitted so far
    const int64_t edges = (int64_t)status->edges;
    for (int64_t s = tid; s < n; s += T)
        emit_at(s, F.keep, F.pos, F.esrc, F.edst, F.ew, edges, out_src, out_dst, out_w, capacity);
    __syncthreads();
    if (tid == 0) {
        status->edges = (unsigned long long)(edges + total);
        // "Boruvka round made no progress" (mst.rs:279-283)
        if (require_progress && total == 0) atomicCAS(&status->err_kind, 0, 4);
    }
    // union: path halving, smallest point of every tree, relabel, count the components
    for (int t = 0; t < steps; ++t) {
        for (int64_t s = tid; s < n; s += T) jump_at(s, F.parent, active_label);
        __syncthreads();
    }
    for (int64_t s = tid; s < n; s += T)
        minlab_init_at(s, F.parent, active_label, F.minlab);
    __syncthreads();
    for (int64_t s = tid; s < n; s += T)
        minlab_reduce_at(s, F.parent, active_label, F.minlab);
    __syncthreads();
    int roots = 0;
    for (int64_t i0 = 0; i0 < n; i0 += T) {
        const int64_t i = i0 + tid;
        int32_t l = -1;
        if (i < n) {
            l = F.minlab[F.parent[active_label ? F.label[i] : (int32_t)i]];
            point_label[i] = l;
        }
        roots += __syncthreads_count(l == (int32_t)i);
    }
    if (tid == 0) status->components = (unsigned long long)roots;
}

// Core column, seed proposals and their merge (core_kernel, seed_kernel, resolve_proposals).
template <int T>
__device__ __forceinline__ void small_seed(const PackFit &f, void *smem) {
    const SmallForest F = small_forest(smem);
    const int64_t n = f.n;
    for (int64_t i = threadIdx.x; i < n; i += T)
        core_at(i, f.dsq, n, f.k, f.min_samples, f.core);
    __syncthreads();
    for (int64_t i = threadIdx.x; i < n; i += T)
        seed_at(i, f.core, f.ids, f.dsq, n, f.k, F.next, F.esrc, F.edst, F.ew, f.status);
    __syncthreads();
    resolve_block<T>(F, nullptr, f.label, n, log2_ceil_dev(n > 1 ? n : 2) + 1, f.status, f.src, f.dst,
                  f.w, n - 1, 0);
}

// Start of a round: counting sort by label (histogram, sum of squared sizes, exclusive scan and
// scatter; the order of points within a label is free, as in scatter_kernel), the sorted labels
// and core distances, cleared row keys and the label range of every 32-row tile.
template <int T>
__device__ __forceinline__ void small_sort(const PackFit &f, void *smem) {
    const SmallForest F = small_forest(smem);
    int32_t *cnt = F.next, *start = F.ja, *fill = F.ma, *perm = F.jb, *labp = F.mb;
    __shared__ int warp_sums[T / 32];
    __shared__ double pair_sums[T / 32];
    const int tid = threadIdx.x;
    const int64_t n = f.n;
    for (int64_t i = tid; i < n; i += T) {
        cnt[i] = 0;
        fill[i] = 0;
        F.label[i] = f.label[i];
    }
    __syncthreads();
    for (int64_t i = tid; i < n; i += T) atomicAdd(&cnt[F.label[i]], 1);
    __syncthreads();
    // sum of squared sizes (exact in f64: integers below 2^53)
    double v = 0.0;
    for (int64_t i = tid; i < n; i += T) {
        const double c = (double)cnt[i];
        v += c * c;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((tid & 31) == 0) pair_sums[tid >> 5] = v;
    int c[SMALL_ITEMS];
    int sum = 0;
    const int64_t base = (int64_t)tid * SMALL_ITEMS;
#pragma unroll
    for (int u = 0; u < SMALL_ITEMS; ++u) {
        c[u] = base + u < n ? cnt[base + u] : 0;
        sum += c[u];
    }
    int total;
    int prefix = block_exclusive_scan<T>(sum, warp_sums, total);
#pragma unroll
    for (int u = 0; u < SMALL_ITEMS; ++u) {
        if (base + u < n) start[base + u] = prefix;
        prefix += c[u];
    }
    if (tid == 0) {
        double t = 0.0;
        for (int w = 0; w < T / 32; ++w) t += pair_sums[w];
        f.status->same_pairs = t;
    }
    __syncthreads();
    for (int64_t i = tid; i < n; i += T) {
        const int32_t l = F.label[i];
        perm[start[l] + atomicAdd(&fill[l], 1)] = (int32_t)i;
    }
    __syncthreads();
    for (int64_t p = tid; p < n; p += T) {
        const int32_t i = perm[p], l = F.label[i];
        labp[p] = l;
        f.perm[p] = i;
        f.corep[p] = f.core[i];
        f.labp[p] = l;
        f.row_keys[p] = ~0ull;
    }
    __syncthreads();
    const int64_t tiles = ceil_div(n, SMALL_RANGE);
    for (int64_t t = tid; t < tiles; t += T) {
        const int64_t a = t * SMALL_RANGE, b = a + SMALL_RANGE < n ? a + SMALL_RANGE : n;
        int32_t mn = labp[a], mx = mn;
        for (int64_t i = a + 1; i < b; ++i) {
            const int32_t l = labp[i];
            mn = l < mn ? l : mn;
            mx = l > mx ? l : mx;
        }
        f.tile_lo[t] = mn;
        f.tile_hi[t] = mx;
    }
}

// End of a round: the per-component minimum key (component_min_kernel's keys, reduced with
// shared atomics), the winners (winner_kernel), then resolve_block over `components` components.
template <int T>
__device__ __forceinline__ void small_merge(const PackFit &f, int64_t components, void *smem) {
    const SmallForest F = small_forest(smem);
    const int tid = threadIdx.x;
    const int64_t n = f.n;
    for (int64_t i = tid; i < n; i += T) {
        F.comp_keys[i] = ~0ull;
        F.label[i] = f.label[i];
    }
    __syncthreads();
    for (int64_t p = tid; p < n; p += T) {
        const unsigned long long v = comp_key_at(p, f.perm, f.row_keys, f.status, f.allow_empty);
        if (v != ~0ull) atomicMin(&F.comp_keys[f.labp[p]], v);
    }
    __syncthreads();
    for (int64_t i = tid; i < n; i += T)
        winner_at(i, F.label, F.comp_keys, f.row_keys, n, F.next, F.esrc, F.edst, F.ew, f.status);
    __syncthreads();
    resolve_block<T>(F, F.label, f.label, n, log2_ceil_dev(components > 1 ? components : 2) + 1,
                  f.status, f.src, f.dst, f.w, n - 1, 1);
}

// One fit alone: its descriptor is a kernel argument.
template <int T>
__global__ void __launch_bounds__(T) small_seed_kernel(const PackFit f) {
    extern __shared__ __align__(16) unsigned char small_smem[];
    small_seed<T>(f, small_smem);
}
template <int T>
__global__ void __launch_bounds__(T) small_sort_kernel(const PackFit f) {
    extern __shared__ __align__(16) unsigned char small_smem[];
    small_sort<T>(f, small_smem);
}
template <int T>
__global__ void __launch_bounds__(T)
    small_merge_kernel(const PackFit f, int64_t components) {
    extern __shared__ __align__(16) unsigned char small_smem[];
    small_merge<T>(f, components, small_smem);
}
// Sorted copy of the rows only (labels and cores: small_sort).
__global__ void gather_rows_kernel(const float *__restrict__ x, const int32_t *__restrict__ perm,
                                   int64_t total, int d, float *__restrict__ xp) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= total) return;
    const int64_t pos = e / d;
    xp[e] = x[(int64_t)perm[pos] * d + (e - pos * d)];
}

inline unsigned blocks(int64_t n, int t = 256) { return (unsigned)ceil_div(n > 0 ? n : 1, t); }

}  // namespace

int scan_exclusive(cuscan_ctx *ctx, ForestBuffers &b, const int32_t *in, int32_t *out, int64_t n,
                   int32_t *grand_total, cudaStream_t s, double *square_sum) {
    const int64_t tiles = ceil_div(n > 0 ? n : 1, SCAN_TILE);
    int rc = ensure(ctx, b.scan_tmp, (size_t)tiles * sizeof(int32_t), "scan tile sums");
    if (rc) return rc;
    CUSCAN_KERNEL(scan_kernel, (unsigned)tiles, SCAN_THREADS, 0, s, in, out, n,
                  as<int32_t>(b.scan_tmp), grand_total, b.status, square_sum);
    CUSCAN_LAUNCH(ctx, "scan_kernel");
    return CUSCAN_OK;
}

static int log2_ceil(int64_t c) {
    int l = 0;
    while ((1ll << l) < c) ++l;
    return l;
}

// Common tail of the seed and of every round: break cycles of the proposals next[] over the
// active nodes, append the kept edges in node order, merge and relabel points.
static int resolve_proposals(cuscan_ctx *ctx, ForestBuffers &b, int64_t n, int64_t active,
                             const int32_t *active_label, int32_t *point_label,
                             uint32_t *out_src, uint32_t *out_dst, float *out_w,
                             int require_progress, cudaStream_t s) {
    int32_t *next = as<int32_t>(b.next);
    int32_t *ja = as<int32_t>(b.jmp_a), *ma = as<int32_t>(b.mx_a);
    int32_t *jb = as<int32_t>(b.jmp_b), *mb = as<int32_t>(b.mx_b);
    // launches of eight hops for 2^(log2(active) + 1) hops
    const int steps = (log2_ceil(active > 1 ? active : 2) + 1 + 2) / 3;
    for (int t = 0; t < steps; ++t) {
        CUSCAN_KERNEL(dbl_hops_kernel, blocks(n), 256, 0, s, next, t ? ja : nullptr,
                      t ? ma : nullptr, active_label, n, jb, mb);
        int32_t *tj = ja, *tm = ma;
        ja = jb;
        ma = mb;
        jb = tj;
        mb = tm;
    }
    int32_t *keep = as<int32_t>(b.keep), *pos = as<int32_t>(b.pos), *parent = as<int32_t>(b.parent);
    int32_t *minlab = as<int32_t>(b.minlab);
    CUSCAN_KERNEL(keep_kernel, blocks(n), 256, 0, s, next, ja, ma, active_label, n, keep, parent,
                  minlab);
    CUSCAN_LAUNCH(ctx, "cycle breaking");
    int rc = scan_exclusive(ctx, b, keep, pos, n, as<int32_t>(b.kept_total), s);
    if (rc) return rc;
    CUSCAN_KERNEL(emit_kernel, blocks(n), 256, 0, s, keep, pos, as<int32_t>(b.scan_tmp),
                  as<uint32_t>(b.esrc), as<uint32_t>(b.edst), as<float>(b.ew), n, b.status, out_src,
                  out_dst, out_w, n - 1);
    for (int t = 0; t < steps; ++t)
        CUSCAN_KERNEL(jump_kernel, blocks(n), 256, 0, s, parent, active_label, n);
    CUSCAN_KERNEL(minlab_reduce_kernel, blocks(n), 256, 0, s, parent, active_label, n, minlab,
                  b.status, as<int32_t>(b.kept_total), require_progress);
    CUSCAN_KERNEL(relabel_kernel, blocks(n), 256, 0, s, point_label, parent, minlab, n, b.status);
    CUSCAN_LAUNCH(ctx, "union/relabel");
    return CUSCAN_OK;
}

// The descriptor of a fit alone (fewer than SMALL_ROWS points) for the one-CTA steps.
static PackFit small_fit(ForestBuffers &b, int64_t n, int32_t *label, uint32_t *out_src,
                         uint32_t *out_dst, float *out_w) {
    PackFit f{};
    f.n = n;
    f.label = label;
    f.src = out_src;
    f.dst = out_dst;
    f.w = out_w;
    f.perm = as<int32_t>(b.perm);
    f.labp = as<int32_t>(b.labp);
    f.corep = as<float>(b.corep);
    f.row_keys = as<unsigned long long>(b.row_keys);
    f.tile_lo = as<int32_t>(b.tile_lo);
    f.tile_hi = as<int32_t>(b.tile_hi);
    f.status = b.status;
    return f;
}

bool forest_small(int64_t n) { return n < SMALL_ROWS; }

int forest_seed(cuscan_ctx *ctx, ForestBuffers &b, float *core, const int32_t *ids,
                const float *dsq, int64_t n, int k, int min_samples, int32_t *label,
                uint32_t *out_src, uint32_t *out_dst, float *out_w, cudaStream_t s) {
    if (forest_small(n)) {
        PackFit f = small_fit(b, n, label, out_src, out_dst, out_w);
        f.k = k;
        f.min_samples = min_samples;
        f.core = core;
        f.ids = const_cast<int32_t *>(ids);
        f.dsq = const_cast<float *>(dsq);
        const auto kernel = CUSCAN_SMALL(small_seed_kernel, n);
        if (int rc = allow_dynamic_smem(ctx, kernel, kSmallSmem)) return rc;
        CUSCAN_KERNEL(kernel, 1, small_threads(n), kSmallSmem, s, f);
        CUSCAN_LAUNCH(ctx, "small_seed_kernel");
        return CUSCAN_OK;
    }
    CUSCAN_KERNEL(core_kernel, blocks(n), 256, 0, s, dsq, n, k, min_samples, core);
    CUSCAN_KERNEL(seed_kernel, blocks(n), 256, 0, s, core, ids, dsq, n, k, as<int32_t>(b.next),
                                           as<uint32_t>(b.esrc), as<uint32_t>(b.edst),
                                           as<float>(b.ew), label, b.status);
    CUSCAN_LAUNCH(ctx, "seed_kernel");
    // all points are active nodes of the seed graph (active_label == nullptr)
    return resolve_proposals(ctx, b, n, n, nullptr, label, out_src, out_dst, out_w, 0, s);
}

int forest_norm_keys(cuscan_ctx *ctx, ForestBuffers &b, const int32_t *label, int64_t n,
                     int64_t components, cudaStream_t s) {
    RefinedBuffers &R = b.refined;
    int32_t *cnt = as<int32_t>(b.cnt), *rank = as<int32_t>(b.pos);
    int rc = ensure(ctx, R.key, sizeof(int32_t) * n, "row keys");
    if (rc) return rc;
    CUSCAN_KERNEL(sort_clear_kernel, blocks(n), 256, 0, s, cnt, as<int32_t>(b.fill),
                  as<unsigned long long>(b.row_keys), as<unsigned long long>(b.comp_keys), n,
                  b.status, true);
    CUSCAN_KERNEL(hist_roots_kernel, blocks(n), 256, 0, s, label, n, cnt, as<int32_t>(b.keep));
    // ranks of the component roots; the histogram's squares are same_pairs
    if ((rc = scan_exclusive(ctx, b, as<int32_t>(b.keep), rank, n, nullptr, s))) return rc;
    CUSCAN_KERNEL(norm_keys_kernel, blocks(n), 256, 0, s, label, rank, as<int32_t>(b.scan_tmp), cnt,
                  as<float>(R.rnorm), as<unsigned int>(R.norm_range), n,
                  norm_levels(n, components), as<int32_t>(R.key), b.status);
    CUSCAN_LAUNCH(ctx, "norm_keys_kernel");
    return CUSCAN_OK;
}

int forest_sort_by_component(cuscan_ctx *ctx, ForestBuffers &b, const float *x, const float *core,
                             const int32_t *label, int64_t n, int d, cudaStream_t s,
                             const int32_t *key) {
    int32_t *cnt = as<int32_t>(b.cnt), *start = as<int32_t>(b.start), *fill = as<int32_t>(b.fill);
    if (forest_small(n)) {
        PackFit f = small_fit(b, n, const_cast<int32_t *>(label), nullptr, nullptr, nullptr);
        f.core = const_cast<float *>(core);
        const auto kernel = CUSCAN_SMALL(small_sort_kernel, n);
        if (int rc = allow_dynamic_smem(ctx, kernel, kSmallSmem)) return rc;
        CUSCAN_KERNEL(kernel, 1, small_threads(n), kSmallSmem, s, f);
        CUSCAN_KERNEL(gather_rows_kernel, blocks(n * d), 256, 0, s, x, as<int32_t>(b.perm), n * d, d,
                      as<float>(b.xp));
        CUSCAN_LAUNCH(ctx, "component sort");
        return CUSCAN_OK;
    }
    CUSCAN_KERNEL(sort_clear_kernel, blocks(n), 256, 0, s, cnt, fill,
                  as<unsigned long long>(b.row_keys), as<unsigned long long>(b.comp_keys), n,
                  b.status, !key);
    CUSCAN_KERNEL(hist_kernel, blocks(n), 256, 0, s, key ? key : label, n, cnt);
    CUSCAN_LAUNCH(ctx, "hist_kernel");
    // same_pairs: the sum of squared component sizes, for the work counters
    int rc = scan_exclusive(ctx, b, cnt, start, n, nullptr, s,
                            key ? nullptr : &b.status->same_pairs);
    if (rc) return rc;
    CUSCAN_KERNEL(scatter_kernel, blocks(n), 256, 0, s, key ? key : label, n, start,
                  as<int32_t>(b.scan_tmp), fill, as<int32_t>(b.perm));
    if (d % 4 == 0 && reinterpret_cast<uintptr_t>(x) % 16 == 0)
        CUSCAN_KERNEL(gather4_kernel, blocks(n * (d / 4)), 256, 0, s,
                      reinterpret_cast<const float4 *>(x), core, label, as<int32_t>(b.perm),
                      n * (d / 4), (unsigned)(d / 4), reinterpret_cast<float4 *>(b.xp.ptr),
                      as<float>(b.corep), as<int32_t>(b.labp));
    else
        CUSCAN_KERNEL(gather_kernel, blocks(n * d), 256, 0, s, x, core, label, as<int32_t>(b.perm), n,
                      d, as<float>(b.xp), as<float>(b.corep), as<int32_t>(b.labp));
    CUSCAN_LAUNCH(ctx, "component sort");
    return CUSCAN_OK;
}

int forest_cell_keys(cuscan_ctx *ctx, ForestBuffers &b, int64_t n, int levels, cudaStream_t s) {
    RefinedBuffers &R = b.refined;
    if (int rc = ensure(ctx, R.key, sizeof(int32_t) * n, "row keys")) return rc;
    CUSCAN_KERNEL(cell_keys_kernel, blocks(n), 256, 0, s, as<int32_t>(R.cells), as<float>(R.rnorm),
                  as<unsigned int>(R.norm_range), n, levels, as<int32_t>(R.key));
    CUSCAN_LAUNCH(ctx, "cell_keys_kernel");
    return CUSCAN_OK;
}

int forest_label_cells(cuscan_ctx *ctx, ForestBuffers &b, const float *core, const int32_t *label,
                       int64_t n, cudaStream_t s) {
    int32_t *cnt = as<int32_t>(b.cnt);
    CUSCAN_KERNEL(sort_clear_kernel, blocks(n), 256, 0, s, cnt, as<int32_t>(b.fill),
                  as<unsigned long long>(b.row_keys), as<unsigned long long>(b.comp_keys), n,
                  b.status, true);
    CUSCAN_KERNEL(label_cells_kernel, blocks(n), 256, 0, s, label, core, as<int32_t>(b.perm), n, cnt,
                  as<int32_t>(b.labp), as<float>(b.corep));
    CUSCAN_LAUNCH(ctx, "label_cells_kernel");
    return scan_exclusive(ctx, b, cnt, as<int32_t>(b.start), n, nullptr, s, &b.status->same_pairs);
}

int forest_round(cuscan_ctx *ctx, ForestBuffers &b, int64_t n, int64_t components,
                 int32_t *label, uint32_t *out_src, uint32_t *out_dst, float *out_w,
                 cudaStream_t s, int allow_empty) {
    unsigned long long *comp_keys = as<unsigned long long>(b.comp_keys);
    if (forest_small(n)) {
        PackFit f = small_fit(b, n, label, out_src, out_dst, out_w);
        f.allow_empty = allow_empty;
        const auto kernel = CUSCAN_SMALL(small_merge_kernel, n);
        if (int rc = allow_dynamic_smem(ctx, kernel, kSmallSmem)) return rc;
        CUSCAN_KERNEL(kernel, 1, small_threads(n), kSmallSmem, s, f, components);
        CUSCAN_LAUNCH(ctx, "small_merge_kernel");
        return CUSCAN_OK;
    }
    CUSCAN_KERNEL(component_min_kernel, blocks(n), 256, 0, s, as<int32_t>(b.perm),
                  as<int32_t>(b.labp), as<unsigned long long>(b.row_keys), n, comp_keys, b.status,
                  allow_empty);
    CUSCAN_KERNEL(winner_kernel, blocks(n), 256, 0, s, label, comp_keys, as<unsigned long long>(b.row_keys),
                                             n, as<int32_t>(b.next), as<uint32_t>(b.esrc),
                                             as<uint32_t>(b.edst), as<float>(b.ew), b.status);
    CUSCAN_LAUNCH(ctx, "component winners");
    return resolve_proposals(ctx, b, n, components, label, label, out_src, out_dst, out_w, 1, s);
}

// Total MST weight in f64: the sum over the emitted edges of sqrt((double) w_sq), the per-edge
// weight that finalize_mst forms (crates/hdbscan-core/src/mst.rs:501-512). Every edge's f64
// weight is exact (IEEE square root of an exactly widened f32); only the order of the sum is
// this kernel's own: a fixed grid-stride assignment and a fixed shared-memory tree per block,
// then one block sums the partials the same way. The result depends only on the edge list.
constexpr int kWeightThreads = 256;
constexpr int kWeightBlocks = 256;

__device__ double block_tree_sum(double v, double *sh) {
    sh[threadIdx.x] = v;
    __syncthreads();
#pragma unroll
    for (int off = kWeightThreads / 2; off > 0; off >>= 1) {
        if ((int)threadIdx.x < off) sh[threadIdx.x] += sh[threadIdx.x + off];
        __syncthreads();
    }
    return sh[0];
}

__global__ void __launch_bounds__(kWeightThreads)
mst_weight_partials_kernel(const float *__restrict__ w, int64_t m, int grid,
                           double *__restrict__ partials) {
    __shared__ double sh[kWeightThreads];
    double acc = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * kWeightThreads + threadIdx.x; i < m;
         i += (int64_t)grid * kWeightThreads)
        acc += sqrt((double)w[i]);
    const double total = block_tree_sum(acc, sh);
    if (threadIdx.x == 0) partials[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kWeightThreads)
mst_weight_final_kernel(const double *__restrict__ partials, int grid, DevStatus *status) {
    __shared__ double sh[kWeightThreads];
    double acc = 0.0;
    for (int i = threadIdx.x; i < grid; i += kWeightThreads) acc += partials[i];
    const double total = block_tree_sum(acc, sh);
    if (threadIdx.x == 0) status->mst_weight = total;
}

int forest_mst_weight(cuscan_ctx *ctx, ForestBuffers &b, const float *w, int64_t m,
                      cudaStream_t s) {
    if (m <= 0) {
        CUSCAN_CUDA(ctx, cudaMemsetAsync(&b.status->mst_weight, 0, sizeof(double), s));
        return CUSCAN_OK;
    }
    // partials live in the component-key array (n 64-bit slots, idle once the rounds end);
    // the grid never exceeds the edge count, which is below n
    const int grid = (int)std::min<int64_t>(kWeightBlocks, ceil_div(m, kWeightThreads));
    double *partials = as<double>(b.comp_keys);
    CUSCAN_KERNEL(mst_weight_partials_kernel, grid, kWeightThreads, 0, s, w, m, grid, partials);
    CUSCAN_KERNEL(mst_weight_final_kernel, 1, kWeightThreads, 0, s, partials, grid, b.status);
    CUSCAN_LAUNCH(ctx, "MST weight");
    return CUSCAN_OK;
}

int forest_reserve(cuscan_ctx *ctx, ForestBuffers &b, int64_t n, int d) {
    const size_t ni = sizeof(int32_t) * (size_t)n;
    int rc = 0;
#define RES(buf, bytes, what) \
    if ((rc = ensure(ctx, b.buf, (bytes), what))) return rc;
    RES(next, ni, "forest proposals");
    RES(esrc, ni, "forest sources");
    RES(edst, ni, "forest destinations");
    RES(ew, sizeof(float) * (size_t)n, "forest weights");
    RES(jmp_a, ni, "pointer doubling");
    RES(mx_a, ni, "pointer doubling");
    RES(jmp_b, ni, "pointer doubling");
    RES(mx_b, ni, "pointer doubling");
    RES(keep, ni, "kept edges");
    RES(pos, ni, "edge positions");
    RES(parent, ni, "forest parents");
    RES(minlab, ni, "component labels");
    RES(kept_total, 64, "kept total");
    RES(cnt, ni, "component histogram");
    RES(start, ni, "component offsets");
    RES(fill, ni, "component cursors");
    RES(perm, ni, "component order");
    RES(xp, sizeof(float) * (size_t)n * (size_t)d, "component-sorted data");
    RES(corep, sizeof(float) * (size_t)n, "component-sorted core distances");
    RES(labp, ni, "component-sorted labels");
    RES(row_keys, sizeof(unsigned long long) * (size_t)n, "row candidates");
    RES(comp_keys, sizeof(unsigned long long) * (size_t)n, "component candidates");
    RES(tile_lo, sizeof(int32_t) * (size_t)(ceil_div(n, 32) + 1), "tile label ranges");
    RES(tile_hi, sizeof(int32_t) * (size_t)(ceil_div(n, 32) + 1), "tile label ranges");
    RES(status_buf, sizeof(DevStatus), "fit status");
    RES(scan_tmp, sizeof(int32_t) * (size_t)ceil_div(n, SCAN_TILE), "scan tile sums");
#undef RES
    b.status = as<DevStatus>(b.status_buf);
    return CUSCAN_OK;
}

int forest_buffers(ForestBuffers &b, Buffer **out) {
    RefinedBuffers &r = b.refined;
    Buffer *all[] = {&b.next, &b.esrc, &b.edst, &b.ew, &b.jmp_a, &b.mx_a, &b.jmp_b, &b.mx_b,
                     &b.keep, &b.pos, &b.parent, &b.minlab, &b.kept_total, &b.cnt, &b.start,
                     &b.fill, &b.perm, &b.xp, &b.corep, &b.labp, &b.row_keys, &b.comp_keys,
                     &b.tile_lo, &b.tile_hi, &b.status_buf, &b.scan_tmp, &b.knn_ids_tmp,
                     &b.knn_dist_tmp, &r.xt, &r.pnorm, &r.mnorm, &r.tile_mmax, &r.tile_lo,
                     &r.tile_hi, &r.cand_ids, &r.cand_lb, &r.fallback, &r.error,
                     &r.cbound, &r.rowcnt, &r.pivots, &r.cells, &r.cell_d, &r.absmax,
                     &r.qthr, &r.xq, &r.pq, &r.mq, &r.cand2, &r.rowcnt2, &r.fallback2,
                     &r.urow, &r.colcnt, &r.colbuf, &r.act_flag, &r.act_idx, &r.act_pos,
                     &r.rowlb, &r.lbtmp, &r.cursor, &r.colp, &r.colc, &r.cmin, &r.pivot_d,
                     &r.cell_scale, &r.tile_centre, &r.tile_radius, &r.thr0, &r.qorder,
                     &r.rnorm, &r.norm_range, &r.key, &r.qchunk_lo, &r.qchunk_hi,
                     &r.masks, &r.ball_thr, &r.vis, &r.vis_count};
    static_assert(sizeof(all) / sizeof(all[0]) == kForestBufferCount, "buffer list");
    const int count = (int)(sizeof(all) / sizeof(all[0]));
    if (out)
        for (int i = 0; i < count; ++i) out[i] = all[i];
    return count;
}

void forest_release_refined(ForestBuffers &b) {
    Buffer *all[kForestBufferCount];
    const int count = forest_buffers(b, all);
    int first = 0;
    while (all[first] != &b.knn_ids_tmp) ++first;  // the list above: the rest follows the forest's own
    for (int i = first; i < count; ++i) release(*all[i]);
}

void forest_release(ForestBuffers &b) {
    Buffer *all[kForestBufferCount];
    const int count = forest_buffers(b, all);
    for (int i = 0; i < count; ++i) release(*all[i]);
    b.status = nullptr;
}

// ---- packed small fits: the one-CTA steps of every fit of a pack, one launch each ----
namespace {

// Fit blockIdx.x: core column, seed proposals, labels and the seed's merge (small_seed, as a fit
// alone). Block 0 also clears the pack's per-round counters.
template <int T>
__global__ void __launch_bounds__(T)
    pack_seed_kernel(const PackFit *__restrict__ fits, int *more) {
    extern __shared__ __align__(16) unsigned char small_smem[];
    const PackFit f = fits[blockIdx.x];
    const int tid = threadIdx.x;
    DevStatus *st = f.status;
    if (blockIdx.x == 0 && tid < kPackMaxRounds + 2) more[tid] = 0;
    if (tid == 0) {
        *st = DevStatus{};
        f.kept_total[1] = 0;
    }
    __syncthreads();
    small_seed<T>(f, small_smem);
    if (tid == 0) {
        st->seed_edges = st->edges;
        st->components_after_seed = st->components;
    }
}

// Start of round r of fit blockIdx.x: whether it runs (more than one component, no error,
// within the round limit: the host driver's checks), then small_sort (pack_gather_kernel copies
// the rows).
template <int T>
__global__ void __launch_bounds__(T) pack_sort_kernel(const PackFit *__restrict__ fits) {
    extern __shared__ __align__(16) unsigned char small_smem[];
    const PackFit f = fits[blockIdx.x];
    DevStatus *st = f.status;
    __shared__ int run;
    if (threadIdx.x == 0) {
        int on = st->components > 1 && st->err_kind == 0;
        if (on && st->rounds > (unsigned long long)kPackMaxRounds) {
            st->err_kind = kPackErrNoConvergence;
            on = 0;
        }
        f.kept_total[1] = on;
        run = on;
    }
    __syncthreads();
    if (!run) return;
    small_sort<T>(f, small_smem);
}

// Sorted copy of the rows of fit blockIdx.y whose round runs (gather_kernel's copy), spread over
// the grid's x blocks: a single CTA per fit would wait on one dependent load pair per element.
__global__ void pack_gather_kernel(const PackFit *__restrict__ fits) {
    const PackFit &f = fits[blockIdx.y];
    if (!*(volatile int32_t *)&f.kept_total[1]) return;
    const int64_t n = f.n;
    const int d = f.d;
    const int64_t total = n * d;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t p = e / d;
        const int c = (int)(e - p * d);
        f.xp[e] = f.x[(int64_t)f.perm[p] * d + c];
    }
}

// End of round r of fit blockIdx.x: winners and merge (small_merge), then the round's
// bookkeeping (rounds run, ordered cross pairs entering it) and whether another round is due.
template <int T>
__global__ void __launch_bounds__(T)
    pack_merge_kernel(const PackFit *__restrict__ fits, int r, int *more) {
    extern __shared__ __align__(16) unsigned char small_smem[];
    const PackFit f = fits[blockIdx.x];
    if (!*(volatile int32_t *)&f.kept_total[1]) return;
    const int tid = threadIdx.x;
    const int64_t n = f.n;
    DevStatus *st = f.status;
    const int64_t comps = (int64_t)st->components;
    __syncthreads();  // every thread has the count before the merge rewrites it
    small_merge<T>(f, comps, small_smem);
    if (tid == 0) {
        st->rounds += 1;
        st->cross_pairs += (double)n * (double)n - st->same_pairs;
        if (st->components > 1 && st->err_kind == 0) atomicAdd(&more[r], 1);
    }
}

// f64 MST weight of fit blockIdx.x in forest_mst_weight's order: the partial of block b of its
// grid is the tree sum over edges b * 256 + t + i * grid * 256, then the partials' tree sum.
__global__ void __launch_bounds__(kWeightThreads)
    pack_weight_kernel(const PackFit *__restrict__ fits) {
    __shared__ double sh[kWeightThreads];
    __shared__ double partials[kWeightBlocks];
    const PackFit &f = fits[blockIdx.x];
    DevStatus *st = f.status;
    if (st->err_kind) return;
    // a complete forest has n - 1 edges (any other count is reported by the host)
    const int64_t m = (int64_t)st->edges < f.n - 1 ? (int64_t)st->edges : f.n - 1;
    if (m <= 0) {
        if (threadIdx.x == 0) st->mst_weight = 0.0;
        return;
    }
    const int64_t g = ceil_div(m, kWeightThreads);
    const int grid = (int)(g < kWeightBlocks ? g : kWeightBlocks);
    for (int b = 0; b < grid; ++b) {
        double acc = 0.0;
        for (int64_t i = (int64_t)b * kWeightThreads + threadIdx.x; i < m;
             i += (int64_t)grid * kWeightThreads)
            acc += sqrt((double)f.w[i]);
        const double total = block_tree_sum(acc, sh);
        if (threadIdx.x == 0) partials[b] = total;
        __syncthreads();
    }
    double acc = 0.0;
    for (int i = threadIdx.x; i < grid; i += kWeightThreads) acc += partials[i];
    const double total = block_tree_sum(acc, sh);
    if (threadIdx.x == 0) st->mst_weight = total;
}

}  // namespace

int pack_seed(cuscan_ctx *ctx, const PackFit *fits, int count, int64_t n_max, int *more,
              cudaStream_t s) {
    const auto kernel = CUSCAN_SMALL(pack_seed_kernel, n_max);
    if (int rc = allow_dynamic_smem(ctx, kernel, kSmallSmem)) return rc;
    CUSCAN_KERNEL(kernel, count, small_threads(n_max), kSmallSmem, s, fits, more);
    CUSCAN_LAUNCH(ctx, "pack_seed_kernel");
    return CUSCAN_OK;
}

int pack_round(cuscan_ctx *ctx, const PackFit *fits, int count, int64_t n_max, int d_max,
               int splits, int r, int *more, cudaStream_t s) {
    const auto sort = CUSCAN_SMALL(pack_sort_kernel, n_max);
    const auto merge = CUSCAN_SMALL(pack_merge_kernel, n_max);
    if (int rc = allow_dynamic_smem(ctx, sort, kSmallSmem)) return rc;
    if (int rc = allow_dynamic_smem(ctx, merge, kSmallSmem)) return rc;
    CUSCAN_KERNEL(sort, count, small_threads(n_max), kSmallSmem, s, fits);
    CUSCAN_LAUNCH(ctx, "pack_sort_kernel");
    const dim3 gg((unsigned)std::min<int64_t>(ceil_div(n_max * d_max, 256), 128), (unsigned)count);
    CUSCAN_KERNEL(pack_gather_kernel, gg, 256, 0, s, fits);
    CUSCAN_LAUNCH(ctx, "pack_gather_kernel");
    if (int rc = launch_pack_candidates(ctx, fits, count, n_max, d_max, splits, s)) return rc;
    CUSCAN_KERNEL(merge, count, small_threads(n_max), kSmallSmem, s, fits, r, more);
    CUSCAN_LAUNCH(ctx, "pack_merge_kernel");
    return CUSCAN_OK;
}

int pack_weight(cuscan_ctx *ctx, const PackFit *fits, int count, cudaStream_t s) {
    CUSCAN_KERNEL(pack_weight_kernel, count, kWeightThreads, 0, s, fits);
    CUSCAN_LAUNCH(ctx, "pack_weight_kernel");
    return CUSCAN_OK;
}

}  // namespace cuscan
