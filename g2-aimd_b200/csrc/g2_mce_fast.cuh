// g2_mce_fast.cuh - the Bron-Kerbosch walk of search-tree nodes with at most 96
// vertices in P and X (of P0) and 128 live back rows (included by mce.cu; same
// tree, same records).
//
// The general walk keeps rows in the warp's slab, one word per lane, and
// rebuilds candidate lists per node: about 600 warp instructions per node with
// most lanes idle at 1 to 4 words, and 7,000 per root to scan forward lists for
// members of P0.  Here
//  * P, X, Q and the set of live back rows are W + W + W + 4 words held by every
//    lane, a lane scores candidates lane, lane + 32, ... by W AND + POPC each
//    from shared memory, and one max-reduction over (score, rank) is the pivot;
//  * the children's back rows are one AND with the branch's column of B (kept
//    both ways round), so there are no lists to filter;
//  * a child without P is counted in place: no frame, no pop.
// Small roots start here (fast_root: rows from tiles of the core's bit matrix,
// g2_corebits.cuh); the general walk enters here (fast_sub) at the first node of a
// branch that is small enough, renumbering its P and X: the dense core's roots
// have hundreds of back rows and over a hundred vertices, their nodes at depth 1
// or 2 few.
//
// Measured (B200, us per call, general walk alone -> with this one): maximal
// cliques of Chung-Lu 2^18 6972 -> 4519, of R-MAT s13 with 50 planted cliques
// 9622 -> 6877, of G(2000, .01) 256 -> 121, of 24 power-law graphs with their
// triangles 5340 -> 2617.  What is left is the latency of the dependent steps of a
// node (a lone warp: about 1,500 cycles per node); the sets are sized so that 24
// warps' rows leave half of the L1 to the slabs (frames in shared memory: 7.4 ->
// 9.5 ms on the R-MAT graph, four CTAs per SM: 9.7 ms).
#pragma once

#include <cstdint>

#include "g2_corebits.cuh"
#include "g2_device.cuh"
#include "g2_handoff.cuh"
#include "g2_kernels.h"

namespace g2 {

namespace {

constexpr uint32_t kFastWords = 3;                // words of a set of vertices
constexpr uint32_t kFastN = 32u * kFastWords;     // vertices
constexpr uint32_t kFastB = 4;                    // words of a set of back rows
constexpr uint32_t kFastM = 32u * kFastB;         // back rows
constexpr uint32_t kFastHist = 104;               // clique sizes counted in shared memory (a small root's all)
constexpr uint32_t kFastRows = 32u * kFastWords * (kFastWords + 2u * kFastB);  // A, B and B transposed (words)
constexpr uint32_t kFastArea = kFastRows + kFastN / 2u;   // and the vertices' places in P0
static_assert(kFastHist >= kFastN + 2u, "a small root's sizes fit");
constexpr uint32_t kFastRecRows = 4;              // record: [task, depth, pool unit, nb] before P, X, R

template <int W>
constexpr uint32_t fast_frame() { return (3u * W + kFastB + 1u + 3u) & ~3u; }  // P, X, Q, back rows, branch

// State of a walk in the slab: the entry node, where the root's rows are (for
// the record pool), then the frames.
struct FastHead {
    uint32_t R[32];            // path of the entry node (bits over P0)
    uint32_t P[4], X[4], B[4];
    uint32_t unit;             // the rows' place in the pool (64-word units), ~0 while not there
    uint32_t nb_full;          // kept back rows of the root
    uint32_t d0;               // depth of the entry node
    uint32_t pad;
    const uint32_t *rowsA, *rowsB;  // the root's rows in memory (null: only in shared memory)
    uint64_t pad2[6];
};
constexpr uint32_t kFastHeadWords = sizeof(FastHead) / 4;
static_assert(sizeof(FastHead) % 64 == 0, "frames stay aligned");
// slab words of a walk
constexpr uint32_t kFastSlab = kFastHeadWords + (kFastN + 2u) * fast_frame<kFastWords>();

__device__ __forceinline__ uint16_t *fast_ids(uint32_t *sm) { return reinterpret_cast<uint16_t *>(sm + kFastRows); }

// Lane i's word, bit j  ->  lane j's word, bit i.
__device__ __forceinline__ uint32_t flip32(uint32_t x) {
    const uint32_t lane = lane_id();
    uint32_t m = 0x0000ffffu;
#pragma unroll
    for (uint32_t k = 16; k; k >>= 1, m ^= m << k) {
        const uint32_t y = __shfl_xor_sync(G2_FULL, x, k);
        x = (lane & k) ? (x & ~m) | ((y >> k) & m) : (x & m) | ((y & m) << k);
    }
    return x;
}

// A warp counts clique sizes in 32-bit shared words that live for many walks; word 0
// (no clique has size 0) carries the inner nodes walked from one walk to the next.
// An inner node adds at most its kFastN leaves, so emptying the counters at every
// a.hist_fold-th of them (2^24) keeps each below 2^32.

// To the run's histogram.
__device__ __noinline__ void fast_flush(const MceArgs &a, uint32_t *hist) {
    __syncwarp();
    for (uint32_t s = lane_id(); s < kFastHist; s += 32) {
        const uint32_t h = hist[s];
        hist[s] = 0;
        if (!h || !s) continue;
        if (s < a.hist_len) atomicAdd(a.out + 1 + s, (unsigned long long)h);
        else if (a.hist_len) atomicOr(a.status, kStatusHistOverflow);  // hist_len 0: no histogram
    }
    __syncwarp();
}

// To a root's own counters, which its commit adds to the run's.
__device__ __noinline__ void fast_keep(uint32_t *hist, unsigned long long *keep, uint32_t sizes) {
    __syncwarp();
    for (uint32_t s = lane_id(); s < sizes; s += 32) {
        if (s) keep[s] += hist[s];
        hist[s] = 0;
    }
    __syncwarp();
}

template <int W>
__device__ __forceinline__ uint32_t *fast_frame_at(FastHead *head, uint32_t l) {
    return reinterpret_cast<uint32_t *>(head) + kFastHeadWords + l * fast_frame<W>();
}

// Hand the pending branches of the shallowest open level to idle warps; frame d
// holds the current node (its first branch stays).  0 nothing to hand off,
// 1 done, 2 buffers full.
template <int W>
__device__ __noinline__ int fast_donate(const MceArgs &a, uint32_t task, uint32_t d, FastHead *head, uint32_t *sm,
                                        uint32_t p) {
    constexpr uint32_t N = 32u * W, M = kFastM;
    const uint32_t *A = sm, *B = A + W * N;
    const uint32_t lane = lane_id(), Wr = (p + 31u) >> 5, nb = head->nb_full, d0 = head->d0;
    uint32_t l = 0, cnt = 0;
    uint32_t *f = nullptr;
    for (; l <= d; l++) {
        f = fast_frame_at<W>(head, l);
        cnt = 0;
        for (uint32_t w = 0; w < W; w++) cnt += __popc(f[2 * W + w]);
        if (l == d) cnt = cnt ? cnt - 1u : 0u;  // the current node keeps its first branch
        if (cnt) break;
    }
    if (cnt == 0) return 0;
    uint32_t unit = head->unit;
    if (unit == 0xffffffffu) {  // the root's rows go to the pool once
        const uint64_t words = (uint64_t)(p + nb) * Wr, units = (words + 63u) >> 6;
        unsigned long long off = 0;
        if (lane == 0) off = atomicAdd(a.npool, (unsigned long long)units);
        off = __shfl_sync(G2_FULL, off, 0);
        if ((off + units) << 6 > a.pool_cap) return 2;
        uint32_t *dst = a.pool + (off << 6);
        if (head->rowsA) {
            for (uint64_t i = lane; i < (uint64_t)p * Wr; i += 32) dst[i] = head->rowsA[i];
            for (uint64_t i = lane; i < (uint64_t)nb * Wr; i += 32) dst[(uint64_t)p * Wr + i] = head->rowsB[i];
        } else {
            for (uint32_t j = lane; j < p; j += 32)
                for (uint32_t w = 0; w < Wr; w++) dst[j * Wr + w] = A[w * N + j];
            for (uint32_t i = lane; i < nb; i += 32)
                for (uint32_t w = 0; w < Wr; w++) dst[(p + i) * Wr + w] = B[w * M + i];
        }
        unit = (uint32_t)off;
        __syncwarp();
        if (lane == 0) head->unit = unit;
    }
    unsigned long long k = reserve_records(a, cnt);
    if (k == ~0ull) return 2;
    const unsigned long long k0 = k;
    const uint16_t *ids = fast_ids(sm);
    uint32_t P[W], X[W], Q[W], stay[W];
#pragma unroll
    for (int w = 0; w < W; w++) P[w] = f[w], X[w] = f[W + w], Q[w] = f[2 * W + w], stay[w] = 0;
    uint32_t path = lane < Wr ? head->R[lane] : 0u;  // lane w: word w
    for (uint32_t j = 0; j < l; j++) {
        const uint32_t id = ids[fast_frame_at<W>(head, j)[3 * W + kFastB]];
        if ((id >> 5) == lane) path |= 1u << (id & 31u);
    }
    auto next = [&]() {  // lowest branch; it moves from P to X and out of Q
        uint32_t q = 0xffffffffu;
#pragma unroll
        for (int w = W - 1; w >= 0; w--)
            if (Q[w]) q = 32u * w + (uint32_t)(__ffs(Q[w]) - 1);
#pragma unroll
        for (int w = 0; w < W; w++)
            if ((q >> 5) == (uint32_t)w) {
                const uint32_t bit = 1u << (q & 31u);
                P[w] &= ~bit;
                X[w] |= bit;
                Q[w] &= ~bit;
            }
        return q;
    };
    if (l == d) {
        const uint32_t q0 = next();
#pragma unroll
        for (int w = 0; w < W; w++)
            if ((q0 >> 5) == (uint32_t)w) stay[w] = 1u << (q0 & 31u);
    }
    for (uint32_t i = 0; i < cnt; i++, k++) {
        const uint32_t q = next();
        uint32_t *rec = a.records + k * a.rec_stride;
        if (lane == 0) {
            rec[0] = task;
            rec[1] = d0 + l + 1u;
            rec[2] = unit;
            rec[3] = nb;
        }
        uint32_t *rp = rec + kFastRecRows, *rx = rp + Wr, *rr = rx + Wr;
        if (lane < Wr) {
            const uint32_t id = ids[q];
            rp[lane] = rx[lane] = 0u;
            rr[lane] = path | ((id >> 5) == lane ? 1u << (id & 31u) : 0u);
        }
        __syncwarp();
#pragma unroll
        for (int w = 0; w < W; w++) {  // the child's P and X, back in P0's numbering
            const uint32_t aq = A[w * N + q], id = ids[32u * w + lane], bit = 1u << (id & 31u);
            if (((P[w] & aq) >> lane) & 1u) atomicOr(rp + (id >> 5), bit);
            if (((X[w] & aq) >> lane) & 1u) atomicOr(rx + (id >> 5), bit);
        }
    }
    publish_records(a, k0, k);
    if (lane == 0)
        for (int w = 0; w < W; w++) f[2 * W + w] = stay[w];
    __syncwarp();
    return 1;
}

// Rows of a root for the general walk, in memory, from the core's bit matrix: A
// (p rows of W words) and the non-zero rows of the back neighbours (at most cap,
// in order).  staged: shared memory for P0.  Returns the kept rows, ~0 if there may be more than cap.  A dense
// root of Chung-Lu 2^18 has 2,000 back neighbours: scanning their lists, a lane
// each and twice, kept its warp 1.6 ms before any branch could be handed off.
__device__ __noinline__ uint32_t core_rows_of_root(const MceArgs &a, uint32_t v, uint64_t split, uint32_t p,
                                                   uint32_t nx, uint32_t *A, uint32_t *B, uint32_t cap,
                                                   uint32_t *staged) {
    const uint32_t lane = lane_id(), W = (p + 31u) >> 5;
    const Csr g{a.rp, a.ci, a.fo, a.core.bits};
    const CoreBlock b = core_block(a.core, v);
    for (uint32_t i = lane; i < p; i += 32) staged[i] = ldg(a.ci + split + i);
    __syncwarp();
    const uint32_t *ids = staged, *xids = a.ci + split - nx;
    uint32_t nb = 0;
    const uint32_t nback = (nx + 31u) >> 5;
    for (uint32_t h = 0; h < W + nback; h++) {  // heads 32 at a time: tiles of P0, then the back neighbours
        const bool back = h >= W;
        const uint32_t i0 = 32u * (back ? h - W : h), m0 = back ? nx : p;
        const uint32_t m = m0 - i0 < 32u ? m0 - i0 : 32u;
        const uint32_t at = i0 + (lane < m ? lane : m - 1u);
        const uint32_t hid = back ? ldg(xids + at) : ids[at];
        uint32_t any = 0;
        bool skip = false;  // no head of the chunk has a bit row
        if (back) {
            if (nb + 32u > cap) return 0xffffffffu;
            uint32_t *mine = B + (uint64_t)(nb + lane) * W;
            for (uint32_t s = 0; s < W; s++) mine[s] = 0u;
            list_rows(g, ids, p, hid, lane < m && hid < b.base, [&](uint32_t j) {
                mine[j >> 5] |= 1u << (j & 31u);
                any = 1u;
            });
            skip = !__any_sync(G2_FULL, lane < m && hid >= b.base);
        }
#pragma unroll 1
        for (uint32_t s = back ? 0u : h; s < W && !skip; s++) {
            const uint32_t j = 32u * s + lane, cid = ids[j < p ? j : p - 1u];
            // lane = column, bits = heads
            uint32_t x = back ? core_tile<false>(g, b, hid, m, cid) : core_tile(g, b, hid, m, cid);
            if (j >= p) x = 0;
            if (!back && s == h) x &= (1u << lane) - 1u;
            const uint32_t y = flip32(x);  // lane = head, bits = columns
            if (back) {
                any |= y;
                B[(uint64_t)(nb + lane) * W + s] |= y;  // (rows past the chunk's are zero and overwritten)
            } else if (s == h) {
                if (j < p) A[(uint64_t)j * W + s] = x | y;
            } else {
                if (j < p) A[(uint64_t)j * W + h] = x;
                A[(uint64_t)(i0 + lane) * W + s] = y;
            }
        }
        if (!back) continue;
        uint32_t tot;
        const uint32_t pos = warp_scan(any != 0, tot);
        if (tot < m)  // close the gaps (rows only move down)
            for (uint32_t s = 0; s < W; s++) {
                __syncwarp();
                const uint32_t y = B[(uint64_t)(nb + lane) * W + s];
                __syncwarp();
                if (any) B[(uint64_t)(nb + pos) * W + s] = y;
            }
        nb += tot;
        __syncwarp();
    }
    return nb;
}

// Rows of a set of back rows for a walk: B (row-major words, given) both ways
// round; lanes hold 32 rows at a time.
__device__ __forceinline__ void fast_put_b(uint32_t *B, uint32_t *T, uint32_t N, uint32_t w, uint32_t b2, uint32_t x) {
    B[w * kFastM + 32u * b2 + lane_id()] = x;
    T[b2 * N + 32u * w + lane_id()] = flip32(x);
}

// A root's rows and entry node from the core's bit matrix.  sm: kFastArea words;
// returns the kept back rows, ~0 if there are more than kFastM.
__device__ __noinline__ uint32_t fast_root(const MceArgs &a, uint32_t v, uint64_t split, uint32_t p, uint32_t nx,
                                           FastHead *head, uint32_t *sm) {
    const uint32_t lane = lane_id(), W = (p + 31u) >> 5, N = 32u * W;
    uint32_t *A = sm, *B = A + W * N, *T = B + W * kFastM;
    const Csr g{a.rp, a.ci, a.fo, a.core.bits};
    const CoreBlock b = core_block(a.core, v);
    // B is filled last: until then it holds a chunk's words, P0 and list rows
    uint32_t *chunk = B, *ids = B + N, *list = B + 2u * N;
    const uint32_t *xids = a.ci + split - nx;
    uint32_t nb = 0;
    __syncwarp();  // the area is free
    for (uint32_t i = lane; i < N; i += 32) ids[i] = ldg(a.ci + split + (i < p ? i : p - 1u));
    for (uint32_t i = lane; i < kFastB * N; i += 32) T[i] = 0u;
    __syncwarp();
    // heads 32 at a time: first the tiles of P0 (the upper ones), then the back neighbours
    const uint32_t nback = (nx + 31u) >> 5;
    for (uint32_t h = 0; h < W + nback; h++) {
        const bool back = h >= W;
        const uint32_t i0 = 32u * (back ? h - W : h), m0 = back ? nx : p;
        const uint32_t m = m0 - i0 < 32u ? m0 - i0 : 32u;
        const uint32_t at = i0 + (lane < m ? lane : m - 1u);
        const uint32_t hid = back ? ldg(xids + at) : ids[at];
        uint32_t any = 0;
        const bool lists = back && __any_sync(G2_FULL, lane < m && hid < b.base);
        if (lists) {
            for (uint32_t s = 0; s < W; s++) list[32u * s + lane] = 0u;
            list_rows(g, ids, p, hid, lane < m && hid < b.base,
                      [&](uint32_t j) { list[(j & ~31u) + lane] |= 1u << (j & 31u); });
        }
#pragma unroll 1
        for (uint32_t s = back ? 0u : h; s < W; s++) {
            const uint32_t j = 32u * s + lane;
            // lane = column, bits = heads
            uint32_t x = back ? core_tile<false>(g, b, hid, m, ids[j]) : core_tile(g, b, hid, m, ids[j]);
            if (lists) x |= flip32(list[32u * s + lane]);
            if (j >= p) x = 0;
            if (back) {
                any |= x;
                chunk[s * 32u + lane] = x;
            } else if (s == h) {
                x &= (1u << lane) - 1u;
                A[s * N + j] = x | flip32(x);
            } else {
                A[h * N + j] = x;
                A[s * N + 32u * h + lane] = flip32(x);
            }
        }
        if (!back) continue;
        const uint32_t mask = __reduce_or_sync(G2_FULL, any);  // those with a neighbour in P0 are kept
        const uint32_t cnt = __popc(mask);
        if (!cnt) continue;
        if (nb + cnt > kFastM) return 0xffffffffu;
        const uint32_t wb = nb >> 5, sh = nb & 31u;
        for (uint32_t s = 0; s < W; s++) {
            const uint32_t x = chunk[s * 32u + lane];
            uint32_t t = x, k = 0;
            if (mask & (mask + 1u)) {  // squeeze out the others
                t = 0;
                for (uint32_t mm = mask; mm; mm &= mm - 1, k++) t |= ((x >> (__ffs(mm) - 1)) & 1u) << k;
            }
            T[wb * N + 32u * s + lane] |= t << sh;
            if (sh + cnt > 32u) T[(wb + 1u) * N + 32u * s + lane] |= t >> (32u - sh);
        }
        nb += cnt;
    }
    for (uint32_t b2 = 0; 32u * b2 < nb; b2++)
        for (uint32_t s = 0; s < W; s++) B[s * kFastM + 32u * b2 + lane] = flip32(T[b2 * N + 32u * s + lane]);
    head->R[lane] = 0u;
    for (uint32_t i = lane; i < kFastN; i += 32) fast_ids(sm)[i] = (uint16_t)i;
    if (lane < 4u) {
        head->P[lane] = p >= 32u * (lane + 1u) ? G2_FULL : p > 32u * lane ? (1u << (p - 32u * lane)) - 1u : 0u;
        head->X[lane] = 0u;
        head->B[lane] = nb >= 32u * (lane + 1u) ? G2_FULL : nb > 32u * lane ? (1u << (nb - 32u * lane)) - 1u : 0u;
    }
    if (lane == 0) {
        head->unit = 0xffffffffu;
        head->nb_full = nb;
        head->d0 = 0;
        head->rowsA = head->rowsB = nullptr;
    }
    __syncwarp();
    return nb;
}

// Bits of a row at the members' places, in order: word(w) = the row's word w, mask
// = lane w's word of the members (the same places for every lane, so each costs
// two shifts for 32 rows); put(o, word) takes the squeezed words.
template <class Word, class Put>
__device__ __forceinline__ void squeeze(uint32_t mask, uint32_t W, Word word, Put put) {
    uint32_t acc = 0, done = 0;
    for (uint32_t w = 0; w < W; w++) {
        uint32_t m = __shfl_sync(G2_FULL, mask, w);
        if (!m) continue;
        const uint32_t x = word(w);
        for (; m; m &= m - 1) {
            acc = __funnelshift_r(acc, x >> (__ffs(m) - 1), 1);
            if ((++done & 31u) == 0) put((done >> 5) - 1u, acc);
        }
    }
    if (done & 31u) put(done >> 5, acc >> (32u - (done & 31u)));
}

// Vertices of the node (P, X) of a general walk (lane w holds word w).
__device__ __forceinline__ uint32_t fast_members(uint32_t P, uint32_t X) {
    return __reduce_add_sync(G2_FULL, (uint32_t)__popc(P | X));
}

// The node (P, X, path R; lane w holds word w) of cnt <= kFastN vertices with the
// live back rows list[0..n), n <= kFastM, of a root whose rows are rowsA / rowsB
// (over p vertices): renumbered, or (cnt = p) as it is, which is cheaper to set up
// and is taken whenever P0 itself is small enough (Chung-Lu 2^18 4.4 against
// 5.4 ms renumbered; R-MAT s13 with planted cliques, P0 up to 150: 7.5 ms in the
// general walk, 6.0 renumbered).
__device__ __noinline__ void fast_sub(uint32_t p, uint32_t cnt, uint32_t P, uint32_t X, uint32_t R, uint32_t d0,
                                      uint32_t unit, uint32_t nb_full, const uint32_t *rowsA, const uint32_t *rowsB,
                                      const uint32_t *list, uint32_t n, FastHead *head, uint32_t *sm) {
    const uint32_t lane = lane_id(), lt = (1u << lane) - 1u, Wr = (p + 31u) >> 5, W = (cnt + 31u) >> 5, N = 32u * W;
    uint32_t *A = sm, *B = A + W * N, *T = B + W * kFastM;
    uint16_t *ids = fast_ids(sm);
    const uint32_t member = P | X;
    __syncwarp();
    if (cnt == p) {  // P0's own numbering
        for (uint32_t i = lane; i < kFastN; i += 32) ids[i] = (uint16_t)i;
        for (uint32_t j = lane; j < N; j += 32)
            for (uint32_t w = 0; w < W; w++) A[w * N + j] = j < p ? rowsA[j * W + w] : 0u;
        for (uint32_t b2 = 0; b2 < kFastB; b2++) {
            const uint32_t i = 32u * b2 + lane, bi = i < n ? list[i] : 0u;
            for (uint32_t w = 0; w < W; w++) {
                if (32u * b2 < n) fast_put_b(B, T, N, w, b2, i < n ? rowsB[(uint64_t)bi * W + w] : 0u);
                else T[b2 * N + 32u * w + lane] = 0u;
            }
        }
        if (lane < W) head->P[lane] = P, head->X[lane] = X;
    }
    uint32_t k = 0;
    for (uint32_t w = 0; w < Wr && cnt != p; w++) {
        const uint32_t m = __shfl_sync(G2_FULL, member, w);
        if ((m >> lane) & 1u) ids[k + __popc(m & lt)] = (uint16_t)((w << 5) + lane);
        k += __popc(m);
    }
    __syncwarp();
    for (uint32_t s = 0; s < W && cnt != p; s++) {
        const uint32_t j = 32u * s + lane, id = ids[j < cnt ? j : cnt - 1u];
        const uint32_t pw = __shfl_sync(G2_FULL, P, id >> 5), xw = __shfl_sync(G2_FULL, X, id >> 5);
        const uint32_t ps = __ballot_sync(G2_FULL, j < cnt && ((pw >> (id & 31u)) & 1u));
        const uint32_t xs = __ballot_sync(G2_FULL, j < cnt && ((xw >> (id & 31u)) & 1u));
        if (lane == 0) head->P[s] = ps, head->X[s] = xs;
        const uint32_t *row = rowsA + (uint64_t)id * Wr;
        squeeze(member, Wr, [&](uint32_t w) { return j < cnt ? row[w] : 0u; },
                [&](uint32_t o, uint32_t x) { A[o * N + j] = x; });
    }
    for (uint32_t b2 = 0; b2 < kFastB && cnt != p; b2++) {
        if (32u * b2 < n) {
            const uint32_t i = 32u * b2 + lane;
            const uint32_t *row = rowsB + (uint64_t)(i < n ? list[i] : 0u) * Wr;
            squeeze(member, Wr, [&](uint32_t w) { return i < n ? row[w] : 0u; },
                    [&](uint32_t o, uint32_t x) { fast_put_b(B, T, N, o, b2, x); });
        } else {
            for (uint32_t w = 0; w < W; w++) T[b2 * N + 32u * w + lane] = 0u;
        }
    }
    head->R[lane] = lane < Wr ? R : 0u;
    if (lane < 4u)
        head->B[lane] = n >= 32u * (lane + 1u) ? G2_FULL : n > 32u * lane ? (1u << (n - 32u * lane)) - 1u : 0u;
    if (lane == 0) {
        head->unit = unit;
        head->nb_full = nb_full;
        head->d0 = d0;
        head->rowsA = rowsA;
        head->rowsB = rowsB;
    }
    __syncwarp();
}

// What a walk found.
struct FastSum {
    unsigned long long nodes, cliques;
    bool donated;
};

// Walk from the entry node in `head` (nb live back rows); hist: sizes found
// (shared memory; emptied into `keep`, or without one into the run's histogram).
template <int W>
__device__ __noinline__ FastSum fast_walk(const MceArgs &a, uint32_t task, uint32_t p, uint32_t nb, FastHead *head,
                                          uint32_t *sm, uint32_t *hist, unsigned long long *keep, long long c0) {
    constexpr uint32_t FW = fast_frame<W>(), N = 32u * W, M = kFastM;
    const uint32_t lane = lane_id();
    const uint32_t *A = sm, *B = A + W * N, *T = B + W * M;
    uint32_t P[W], X[W], Q[W], XB[kFastB];
    const uint32_t d0 = head->d0;
    bool donated = false;
#pragma unroll
    for (int w = 0; w < W; w++) P[w] = head->P[w], X[w] = head->X[w];
#pragma unroll
    for (uint32_t b2 = 0; b2 < kFastB; b2++) XB[b2] = head->B[b2];
#pragma unroll
    for (int w = 0; w < W; w++) Q[w] = 0;
    __syncwarp();
    const uint32_t nbw = (nb + 31u) >> 5;
    uint32_t d = 0;
    unsigned long long nodes = 0, cliques = 0;
    bool may_spill = a.spill_cycles != 0 && ((p + 31u) >> 5) <= a.rec_words;
    long long next_check = 0;
    if (may_spill) {  // (a branch of a longer walk checks on its own clock)
        if (lane == 0) next_check = clock64() - c0;
        next_check = __shfl_sync(G2_FULL, next_check, 0) / (long long)a.spill_cycles * (long long)a.spill_cycles +
                     (long long)a.spill_cycles;
    }
    uint32_t inner = hist[0];
    const uint32_t fold = a.hist_fold - 1u;
    // a maximal clique of `size` vertices.  Sizes beyond the counters (a branch deep in
    // a large root) go to the root's own: keeping such branches out of this walk
    // instead made Chung-Lu 2*10^5 (exponent 2.2) 34 ms where it takes 19
    auto found = [&](uint32_t size) {
        cliques++;
        if (lane == 0) {
            if (size < kFastHist) hist[size]++;
            else keep[size]++;
        }
    };
    auto save = [&](uint32_t at, uint32_t q) {
        uint32_t f[FW];
#pragma unroll
        for (int w = 0; w < W; w++) f[w] = P[w], f[W + w] = X[w], f[2 * W + w] = Q[w];
#pragma unroll
        for (uint32_t b2 = 0; b2 < kFastB; b2++) f[3 * W + b2] = XB[b2];
        f[3 * W + kFastB] = q;
#pragma unroll
        for (uint32_t i = 3 * W + kFastB + 1; i < FW; i++) f[i] = 0;
        if (lane == 0) {
            uint4 *to = reinterpret_cast<uint4 *>(fast_frame_at<W>(head, at));
#pragma unroll
            for (uint32_t i = 0; i < FW / 4; i++) to[i] = make_uint4(f[4 * i], f[4 * i + 1], f[4 * i + 2], f[4 * i + 3]);
        }
    };
    bool enter = true;
    for (;;) {
        if (enter) {
            enter = false;
            nodes++;
            uint32_t anyp = 0, anyx = 0;
#pragma unroll
            for (int w = 0; w < W; w++) anyp |= P[w], anyx |= X[w];
#pragma unroll
            for (uint32_t b2 = 0; b2 < kFastB; b2++) anyx |= XB[b2];
            if (!anyp) {  // an entry's own node only (children without P are counted below)
                if (!anyx) found(d0 + d + 1u);
            } else {
                // pivot: max (|P ∩ row|, rank) over P, X and the live back rows
                uint32_t best = 0;
#pragma unroll
                for (int s = 0; s < W; s++) {
                    const uint32_t px = P[s] | X[s];
                    if (!px) continue;
                    uint32_t sc = 0;
#pragma unroll
                    for (int w = 0; w < W; w++) sc += __popc(P[w] & A[w * N + 32u * s + lane]);
                    const uint32_t key = (sc << 16) | (nb + 32u * s + lane);
                    if (((px >> lane) & 1u) && key > best) best = key;
                }
                for (uint32_t b2 = 0; b2 < nbw; b2++) {
                    uint32_t xb = 0;
#pragma unroll
                    for (uint32_t t = 0; t < kFastB; t++)
                        if (t == b2) xb = XB[t];
                    if (!xb) continue;
                    uint32_t sc = 0;
#pragma unroll
                    for (int w = 0; w < W; w++) sc += __popc(P[w] & B[w * M + 32u * b2 + lane]);
                    const uint32_t key = (sc << 16) | (32u * b2 + lane);
                    if (((xb >> lane) & 1u) && key > best) best = key;
                }
                best = __reduce_max_sync(G2_FULL, best) & 0xffffu;
                const uint32_t *row = best >= nb ? A + (best - nb) : B + best;
                const uint32_t step = best >= nb ? N : M;
#pragma unroll
                for (int w = 0; w < W; w++) Q[w] = P[w] & ~row[w * step];
                inner++;
                if ((inner & fold) == 0) {
                    if (keep) fast_keep(hist, keep, p + 2u < kFastHist ? p + 2u : kFastHist);
                    else fast_flush(a, hist);
                }
                if (may_spill && (nodes & 15u) == 0) {
                    long long el = 0;
                    if (lane == 0) el = clock64() - c0;
                    el = __shfl_sync(G2_FULL, el, 0);
                    if (el > next_check) {
                        if (handoff_wanted(a)) {
                            save(d, 0u);
                            __syncwarp();
                            const int got = fast_donate<W>(a, task, d, head, sm, p);
                            donated |= got == 1;
                            if (got == 2) may_spill = false;  // buffers full: finish the walk here
#pragma unroll
                            for (int w = 0; w < W; w++) Q[w] = fast_frame_at<W>(head, d)[2 * W + w];
                            __syncwarp();
                        }
                        next_check = el + (long long)a.spill_cycles;
                    }
                }
            }
        }
        // next branch: lowest bit of Q
        uint32_t q = 0xffffffffu;
#pragma unroll
        for (int w = W - 1; w >= 0; w--)
            if (Q[w]) q = 32u * w + (uint32_t)(__ffs(Q[w]) - 1);
        if (q == 0xffffffffu) {  // level done
            if (d == 0) break;
            d--;
            __syncwarp();
            const uint4 *from = reinterpret_cast<const uint4 *>(fast_frame_at<W>(head, d));
            uint32_t f[FW];
#pragma unroll
            for (uint32_t i = 0; i < FW / 4; i++) {
                const uint4 x = from[i];
                f[4 * i] = x.x, f[4 * i + 1] = x.y, f[4 * i + 2] = x.z, f[4 * i + 3] = x.w;
            }
#pragma unroll
            for (int w = 0; w < W; w++) P[w] = f[w], X[w] = f[W + w], Q[w] = f[2 * W + w];
#pragma unroll
            for (uint32_t b2 = 0; b2 < kFastB; b2++) XB[b2] = f[3 * W + b2];
            __syncwarp();
            continue;
        }
        // the child, from the sets before q moves (row q has no bit q)
        uint32_t cp[W], cx[W], cb[kFastB], anyp = 0, anyx = 0;
#pragma unroll
        for (int w = 0; w < W; w++) {
            const uint32_t aq = A[w * N + q];
            cp[w] = P[w] & aq;
            cx[w] = X[w] & aq;
            anyp |= cp[w];
            anyx |= cx[w];
        }
#pragma unroll
        for (uint32_t b2 = 0; b2 < kFastB; b2++) {
            cb[b2] = b2 < nbw ? XB[b2] & T[b2 * N + q] : 0u;
            anyx |= cb[b2];
        }
#pragma unroll
        for (int w = 0; w < W; w++)
            if ((q >> 5) == (uint32_t)w) {  // q moves from P to X
                const uint32_t bit = 1u << (q & 31u);
                P[w] &= ~bit;
                X[w] |= bit;
                Q[w] &= ~bit;
            }
        if (!anyp) {  // a leaf: counted here
            nodes++;
            if (!anyx) found(d0 + d + 2u);
            continue;
        }
        save(d, q);
#pragma unroll
        for (int w = 0; w < W; w++) P[w] = cp[w], X[w] = cx[w];
#pragma unroll
        for (uint32_t b2 = 0; b2 < kFastB; b2++) XB[b2] = cb[b2];
        d++;
        enter = true;
    }
    if (lane == 0) hist[0] = inner;
    __syncwarp();
    return FastSum{nodes, cliques, donated};
}

// n: vertices of the entry node's numbering.
__device__ __forceinline__ FastSum fast_any(const MceArgs &a, uint32_t task, uint32_t p, uint32_t n, uint32_t nb,
                                            FastHead *head, uint32_t *sm, uint32_t *hist, unsigned long long *keep, long long c0) {
    switch ((n + 31u) >> 5) {
        case 1: return fast_walk<1>(a, task, p, nb, head, sm, hist, keep, c0);
        case 2: return fast_walk<2>(a, task, p, nb, head, sm, hist, keep, c0);
        default: return fast_walk<3>(a, task, p, nb, head, sm, hist, keep, c0);
    }
}

}  // namespace

}  // namespace g2
