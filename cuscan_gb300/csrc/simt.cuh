// Exact f32 pair tiles on the SIMT cores, shared by the kNN sweep (knn.cu) and the Borůvka
// candidate sweep (boruvka.cu).
//
// One CTA of 128 threads computes 64 query x 128 reference tiles of squared distances, each pair
// accumulated in feature order as acc = fmaf(q_f - r_f, q_f - r_f, acc)
// (crates/cuscan-common/src/kernels/neighbors.rs:44-48). Both operands stream through a
// three-stage ring of 16-feature chunks, transposed on the way in ([feature][row], 4-byte
// cp.async), and every thread keeps an 8 x 8 block of pairs in registers.
//
// What bounds it: the FP32 pipe. A pair and feature cost one subtract and one FMA. Packed f32x2
// arithmetic (two references per instruction, each lane rounded as the scalar instruction)
// halves the issue slots, so the shared loads, the packing of the query value and the copies
// issue beside it: in registers alone the packed form sustains 18.1e12 pair-features/s on a
// GB300 against 14.3e12 for the scalar form. The 8 x 8 block reads 16 floats of shared memory for
// 64 pairs; one query per thread against 32 references (the layout before it) read 33 floats for
// 32 pairs and was bound by shared-memory bandwidth at 5.0e12. Streaming the queries
// as well, instead of holding all their features, keeps three CTAs on an SM up to the widest
// rows.
#pragma once

#include "common.cuh"

namespace cuscan {
namespace simt {

constexpr int QT = 64;        // query rows per tile
constexpr int RT = 128;       // reference rows per tile
constexpr int KC = 16;        // features per pipeline stage
constexpr int STAGES = 3;
constexpr int THREADS = 128;
constexpr int CTAS_PER_SM = 3;  // register limit: 168 per thread
constexpr int QS = QT + 4;    // padded rows: 16-byte alignment, transposing copies on two banks
constexpr int RS = RT + 4;
constexpr int STAGE_FLOATS = KC * (QS + RS);

__device__ __forceinline__ void cp_async4(float *smem, const float *gmem) {
    unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

using Packed = unsigned long long;  // two f32 values
__device__ __forceinline__ Packed pack2(float v) {
    Packed r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ void unpack2(Packed p, float &a, float &b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p));
}
__device__ __forceinline__ Packed sub2(Packed a, Packed b) {
    Packed r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ Packed fma2(Packed a, Packed b, Packed c) {
    Packed r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// The thread's place in the tile: queries 4 tq + {0..3} and 32 + 4 tq + {0..3}, references
// 4 tr + {0..3} and 64 + 4 tr + {0..3}. A warp covers 32 queries x 64 references, so its shared
// loads touch 64 and 128 distinct bytes.
struct Place {
    int tq, tr;
};
__device__ __forceinline__ Place place() {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    return {(warp & 1) * 4 + (lane >> 3), (warp >> 1) * 8 + (lane & 7)};
}
__device__ __forceinline__ int query_of(const Place &p, int i) { return (i >> 2) * 32 + p.tq * 4 + (i & 3); }
__device__ __forceinline__ int ref_of(const Place &p, int j) { return (j >> 2) * 64 + p.tr * 4 + (j & 3); }

// Features [f0, f0 + kc) of the 64 query rows rows_s[] (row indices in shared memory).
__device__ __forceinline__ void copy_queries(float *dst, const float *__restrict__ x,
                                             const int32_t *rows_s, int d, int f0, int kc) {
    const int f = threadIdx.x & (KC - 1), r = threadIdx.x / KC;
    if (f >= kc) return;
    constexpr int STEP = THREADS / KC;
#pragma unroll
    for (int i = 0; i < QT / STEP; ++i)
        cp_async4(dst + f * QS + r + i * STEP, x + (int64_t)rows_s[r + i * STEP] * d + f0 + f);
}

// The same of reference rows [row0, row0 + 128); rows at or past `end` repeat row end - 1 (the
// epilogues leave them out).
__device__ __forceinline__ void copy_refs(float *dst, const float *__restrict__ x, int64_t row0,
                                          int64_t end, int d, int f0, int kc) {
    const int f = threadIdx.x & (KC - 1), r = threadIdx.x / KC;
    if (f >= kc) return;
    constexpr int STEP = THREADS / KC;
    if (row0 + RT <= end) {
        const float *p = x + (row0 + r) * d + f0 + f;
        const int64_t step = (int64_t)STEP * d;
#pragma unroll
        for (int i = 0; i < RT / STEP; ++i) {
            cp_async4(dst + f * RS + r + i * STEP, p);
            p += step;
        }
    } else {
#pragma unroll 4
        for (int i = 0; i < RT / STEP; ++i) {
            int64_t row = row0 + r + i * STEP;
            if (row >= end) row = end - 1;
            cp_async4(dst + f * RS + r + i * STEP, x + row * d + f0 + f);
        }
    }
}

// acc[i][j / 2] += the features of one chunk.
__device__ __forceinline__ void accumulate(Packed (&acc)[8][4], const float *q, const float *r,
                                           int kc, const Place &p) {
    const float *qp = q + p.tq * 4, *rp = r + p.tr * 4;
#pragma unroll 4
    for (int f = 0; f < kc; ++f) {
        const float4 qa = *reinterpret_cast<const float4 *>(qp + f * QS);
        const float4 qb = *reinterpret_cast<const float4 *>(qp + f * QS + 32);
        const ulonglong2 ra = *reinterpret_cast<const ulonglong2 *>(rp + f * RS);
        const ulonglong2 rb = *reinterpret_cast<const ulonglong2 *>(rp + f * RS + 64);
        const float qv[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
        const Packed rv[4] = {ra.x, ra.y, rb.x, rb.y};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const Packed qq = pack2(qv[i]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const Packed t = sub2(qq, rv[j]);
                acc[i][j] = fma2(t, t, acc[i][j]);
            }
        }
    }
}

// Distances of query i of the thread to its eight references.
__device__ __forceinline__ void row_of(const Packed (&a)[4], float (&v)[8]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) unpack2(a[j], v[2 * j], v[2 * j + 1]);
}

// The sweep of 64 query rows over the tiles of [t_begin, t_end) that `next` visits (next(t) is
// the first visited tile at or after t, at least t_end when none is left), references below r_end.
// next is called once per visited tile, by the copy side (up to two tiles ahead), right after a
// barrier and before the following one. meta(tile, slot) copies a tile's row data (cp.async)
// into slot 0..3 with the tile's first chunk; epilogue(tile, slot, acc) runs once per tile, in
// order. Every thread of the CTA takes part.
template <class Next, class Meta, class Epilogue>
__device__ __forceinline__ void sweep(const float *__restrict__ query, const int32_t *rows_s,
                                      const float *__restrict__ ref, int d, int64_t t_begin,
                                      int64_t t_end, int64_t r_end, float *stages, Next next,
                                      Meta meta, Epilogue epilogue) {
    const Place p = place();
    const int chunks = (d + KC - 1) / KC;
    int64_t lt = next(t_begin);  // tile of the copy side
    int64_t ahead[STAGES - 1];   // tiles whose copies have begun after the compute side's tile
    int waiting = 0;
    int lc = 0, lstage = 0, stage = 0;
    int lslot = 0, slot = 0;
    auto load = [&]() {
        if (lt < t_end) {
            float *s = stages + lstage * STAGE_FLOATS;
            const int f0 = lc * KC, kc = d - f0 < KC ? d - f0 : KC;
            copy_queries(s, query, rows_s, d, f0, kc);
            copy_refs(s + KC * QS, ref, lt * RT, r_end, d, f0, kc);
            if (lc == 0) {
                meta(lt, lslot);
                // (unrolled: the queue stays in registers)
#pragma unroll
                for (int i = 0; i < STAGES - 1; ++i)
                    if (i == waiting) ahead[i] = lt;
                ++waiting;
            }
            if (++lc == chunks) {
                lc = 0;
                lslot = (lslot + 1) & 3;
                lt = next(lt + 1);
            }
        }
        cp_async_commit();
        lstage = lstage + 1 == STAGES ? 0 : lstage + 1;
    };
#pragma unroll
    for (int i = 0; i < STAGES - 1; ++i) load();
    while (waiting > 0) {
        const int64_t ct = ahead[0];
#pragma unroll
        for (int i = 0; i + 1 < STAGES - 1; ++i) ahead[i] = ahead[i + 1];
        --waiting;
        Packed acc[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
        for (int c = 0; c < chunks; ++c) {
            cp_async_wait<STAGES - 2>();
            __syncthreads();
            load();  // into the stage that every thread has finished with
            const float *s = stages + stage * STAGE_FLOATS;
            const int kc = d - c * KC < KC ? d - c * KC : KC;
            accumulate(acc, s, s + KC * QS, kc, p);
            stage = stage + 1 == STAGES ? 0 : stage + 1;
        }
        epilogue(ct, slot, acc);
        slot = (slot + 1) & 3;
    }
    cp_async_wait<0>();
}

// Reference chunks per query tile: `splits` CTAs for each of the query tiles, each over `chunk`
// references (a multiple of a tile), chunks of at least min_tiles tiles. The CTAs of a launch
// take about as long each, so its time is the waves over the resident slots times a CTA's tiles
// and start_tiles (its start and its results, in tiles); the count with the least such time is
// taken, among those of at most eight waves (partial results grow with the splits). 10,007 x 64 candidates (157 query tiles
// on 456 slots) took 787 us with at most 4 splits and take 562 us.
inline void split_plan(int sm_count, int64_t query_tiles, int64_t nr, int64_t min_tiles,
                       double start_tiles, int64_t &splits, int64_t &chunk,
                       int64_t limit = INT64_MAX) {
    const int64_t slots = (int64_t)CTAS_PER_SM * sm_count, tiles = ceil_div(nr, (int64_t)RT);
    if (query_tiles < 1) query_tiles = 1;
    int64_t most = ceil_div(8 * slots, query_tiles);
    if (most > ceil_div(tiles, min_tiles)) most = ceil_div(tiles, min_tiles);
    if (most > limit) most = limit;
    splits = 1;
    double best = 0.0;
    for (int64_t s = 1; s <= most; ++s) {
        const int64_t per = ceil_div(tiles, s);  // tiles of a CTA
        const double cost =
            (double)ceil_div(query_tiles * ceil_div(tiles, per), slots) * ((double)per + start_tiles);
        if (s == 1 || cost < best) {
            best = cost;
            splits = s;
        }
    }
    chunk = ceil_div(tiles, splits) * RT;
    splits = ceil_div(nr, chunk);
    if (splits < 1) splits = 1;
}
// Parts of a kNN sweep keep their partial lists within kSplitRows rows beyond the queries' own, and
// have at least two tiles.
constexpr int64_t kSplitRows = 512 * (int64_t)kSMs;
inline int64_t split_most(int64_t nq) { return (kSplitRows + nq) / nq; }
// Most rows of partial lists of up to nq queries against nr references.
inline int64_t split_max_rows(int64_t nq, int64_t nr) {
    const int64_t parts = nq * ceil_div(ceil_div(nr, (int64_t)RT), (int64_t)2);
    return kSplitRows + nq < parts ? kSplitRows + nq : parts;
}

}  // namespace simt
}  // namespace cuscan
