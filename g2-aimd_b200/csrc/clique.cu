// clique.cu - counts of 3-, 4- and 5-cliques (plans whose every position is
// adjacent to all earlier ones with images strictly increasing: presets 0, 24,
// 25) on bit rows of the root's forward neighbourhood, for sm_100a.
//
// Replaces GMatchApp (app_gmatch/gmatch.h:15-736) for these plans; the count
// of a root v is the number of (k-1)-cliques of the local graph on
// P0 = N(v) ∩ (v, ∞).  Two launches:
//
//  1. clique_prepare_kernel writes the bit matrix of the graph's dense core
//     (g2_corebits.cuh) and drops the tasks whose root cannot hold a clique
//     (|P0| < k - 1; two thirds of the roots of R-MAT s20), listing the others.
//  2. clique_kernel, a persistent grid, builds each root's rows 32 heads
//     by 32 columns at a time and counts pairs of rows by AND + popc.
//
// How a root is walked depends on p = |P0|:
//   p <= 32          one warp, a row per lane in registers;
//   p <= kWarpP      one warp, rows in the warp's shared memory;
//   larger, ordered  the CTA's warps share the root: rows in the CTA's shared
//                    memory, chunks of work taken from a shared counter (for
//                    5-cliques from 65 vertices on: 2.5 -> 1.7 ms on R-MAT s16);
//   larger, in order one warp, rows in the warp's slab (runs in the caller's
//                    order, which take the roots one by one as given).
// Measured (B200, forward lists and one warp per root -> this): 4-cliques of R-MAT
// s20 15.3 -> 3.6 ms (13.1 -> 2.5 G warp instructions; logic pipe and probe
// latency bound it), triangles of s18 6.1 -> 0.28 ms, 5-cliques of s16 31 -> 1.5 ms.
// A warp per root for all widths in schedule order was slower (5.2 ms on s20: the
// heavy roots' rows fight for the L1), fewer than 8 warps per CTA too (5.4 ms).
// Rows are stored as a packed triangle (row i keeps words 0 .. i / 32, at
// an odd stride so that lanes reading rows of one tile hit different banks),
// which halves the shared memory of a root: p = 658 takes 31 KB, so five CTAs of
// 8 warps stay resident.
#include <cstdint>

#include "g2_bitrows.cuh"
#include "g2_corebits.cuh"
#include "g2_device.cuh"
#include "g2_kernels.h"

namespace g2 {

CoreBlock core_block_of(uint32_t lo, uint32_t n, uint64_t bytes, uint32_t row0, uint64_t off) {
    uint32_t k = 0;
    while (k < n && (uint64_t)(k + 128u) * (k + 128u) / 8u <= bytes) k += 128u;
    if (k > n) k = n;
    CoreBlock b{};
    b.base = lo + n - k;
    b.end = lo + n;
    b.stride = ((k + 127u) / 128u) * 4u;
    b.row0 = row0;
    b.off = off;
    return b;
}

namespace {

constexpr uint32_t kWarpP = 128;      // roots up to this are walked by one warp in shared memory
constexpr uint32_t kQueue = 64;       // candidate queue of a warp (entries)
constexpr uint32_t kSub = 256;        // 5-cliques: largest neighbourhood compressed into its own rows
constexpr uint32_t kMaxQWords = 512;  // 5-clique candidate rows up to |P0| = 16384

// sum over t = 1..q of t | 1: words of the first q row tiles, per row of a tile
__host__ __device__ __forceinline__ constexpr uint32_t tri_f(uint32_t q) { return q * (q + 1u) / 2u + (q >> 1); }
__host__ __device__ __forceinline__ constexpr uint64_t tri_words(uint32_t W) { return 32ull * tri_f(W); }

// Lower rows of a local graph: row j keeps words 0 .. j / 32 (its neighbours
// before it) at an odd stride.
struct Tri {
    uint32_t *a;
    __device__ __forceinline__ uint32_t *row(uint32_t j) const {
        const uint32_t r = j >> 5;
        return a + 32u * tri_f(r) + (j & 31u) * ((r + 1u) | 1u);
    }
};

// Checks inside a root's tiles stand in the BUDGET build only (deadline set): in the
// other they cost 4 % of the 4-cliques of R-MAT s20.
__device__ __forceinline__ bool past_deadline(const CliqueArgs &a) {
    if (!a.deadline) return false;
    unsigned long long now = 0;
    if (lane_id() == 0) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
    now = __shfl_sync(G2_FULL, now, 0);
    return now > *a.deadline;
}

// Word r of the rows of tile w (lane = row 32 w + lane) from P0 (one warp).
template <class P0>
__device__ __forceinline__ uint32_t local_word(const Csr &g, const CoreBlock &b, P0 ids, uint32_t p, uint32_t w,
                                               uint32_t r) {
    const uint32_t lane = lane_id(), j = 32u * w + lane, i = 32u * r + lane;
    const uint32_t cid = ids[j < p ? j : p - 1u], hid = r == w ? cid : ids[i];
    uint32_t x = core_tile(g, b, hid, p - 32u * r < 32u ? p - 32u * r : 32u, cid);
    if (r == w) x &= (1u << lane) - 1u;
    return j < p ? x : 0u;
}

// Triangles through the pairs (y, z) with y in row tile w: lane y keeps words
// j0 .. j0 + N - 1 of its row in registers, the rows z >= y pass by (broadcast
// reads), and popc(row y & row z) is summed where y is in row z.  POPC issues
// at a quarter of the rate of logic, so two words and a running one are first
// added as bits (a full adder is two LOP3): one POPC per two words.
// Rows y with y % nparts == part.  Per-lane count.
template <int N>
__device__ __forceinline__ uint32_t pair_chunk(const Tri &t, uint32_t p, uint32_t w, uint32_t j0, uint32_t part,
                                               uint32_t nparts) {
    const uint32_t lane = lane_id(), top = 0x80000000u >> lane;  // x * top = x << (31 - lane), off the logic pipe
    uint32_t r[N];
    {
        const uint32_t *y = t.row(32u * w + lane) + j0;
        const bool own = nparts <= 1 || (32u * w + lane) % nparts == part;
#pragma unroll
        for (int i = 0; i < N; i++) r[i] = own ? y[i] : 0u;
    }
    uint32_t ones = 0, twos = 0;
    const uint32_t W = (p + 31u) >> 5;
    for (uint32_t tz = w; tz < W; tz++) {
        const uint32_t s = (tz + 1u) | 1u;
        const uint32_t *z = t.a + 32u * tri_f(tz);
        const uint32_t nz = p - 32u * tz < 32u ? p - 32u * tz : 32u;
#pragma unroll 1
        for (uint32_t k = 0; k < nz; k += 2, z += 2u * s) {  // tiles hold 32 rows: an odd last pair reads a zero row
            const uint32_t m0 = (uint32_t)((int)(z[w] * top) >> 31), m1 = (uint32_t)((int)(z[s + w] * top) >> 31);
#pragma unroll
            for (int i = 0; i < N; i++) {
                const uint32_t x0 = z[j0 + i] & r[i] & m0, x1 = z[s + j0 + i] & r[i] & m1;
                twos += __popc((x0 & x1) | (ones & (x0 ^ x1)));
                ones ^= x0 ^ x1;
            }
        }
    }
    return 2u * twos + __popc(ones);
}

__device__ __forceinline__ uint32_t pair_chunk_n(const Tri &t, uint32_t p, uint32_t w, uint32_t j0, uint32_t n,
                                                 uint32_t part, uint32_t nparts) {
    switch (n) {
        case 1: return pair_chunk<1>(t, p, w, j0, part, nparts);
        case 2: return pair_chunk<2>(t, p, w, j0, part, nparts);
        case 3: return pair_chunk<3>(t, p, w, j0, part, nparts);
        case 4: return pair_chunk<4>(t, p, w, j0, part, nparts);
        case 5: return pair_chunk<5>(t, p, w, j0, part, nparts);
        case 6: return pair_chunk<6>(t, p, w, j0, part, nparts);
        case 7: return pair_chunk<7>(t, p, w, j0, part, nparts);
        default: return pair_chunk<8>(t, p, w, j0, part, nparts);
    }
}

// Chunks of row tile w: its w + 1 words in equal pieces of at most 8.
__device__ __forceinline__ uint32_t chunks_of(uint32_t w) { return (w + 8u) >> 3; }
__device__ __forceinline__ uint32_t tile_chunk(const Tri &t, uint32_t p, uint32_t w, uint32_t c, uint32_t part,
                                               uint32_t nparts) {
    const uint32_t nc = chunks_of(w), j0 = (w + 1u) * c / nc, j1 = (w + 1u) * (c + 1u) / nc;
    return pair_chunk_n(t, p, w, j0, j1 - j0, part, nparts);
}

// Triangles of a local graph of p vertices, by one warp.  Per-lane count; ~0 if the
// time budget of `budget` ran out.
template <bool BUDGET>
__device__ __forceinline__ uint64_t triangles(const Tri &t, uint32_t p, uint32_t part, uint32_t nparts,
                                              const CliqueArgs *budget = nullptr) {
    uint64_t c = 0;
    for (uint32_t w = 0; 32u * w < p; w++) {
        if (BUDGET && past_deadline(*budget)) return ~0ull;
        for (uint32_t k = 0; k < chunks_of(w); k++) c += tile_chunk(t, p, w, k, part, nparts);
    }
    return c;
}

// Shared memory of a warp's 5-clique work: the compressed neighbourhood's
// members and rows, and the queue and candidate row of larger ones.
struct Sub {
    uint32_t cap;     // largest neighbourhood compressed
    uint16_t *list;   // cap entries
    uint32_t *rows;   // tri_words(cap / 32)
    uint32_t *queue;  // kQueue
    uint32_t *q;      // words of a row
};

// 4-cliques of the local graph whose highest vertex is `top` = triangles among
// the members of row `top`.  Up to cap members the induced graph is compressed
// into rows of its own: a member's new row is its old row's bits at the
// members' places, which are the same places for every lane, so each costs two
// shifts for 32 rows.  Larger neighbourhoods are walked per edge.  Per-lane count.
__device__ uint64_t count_below(const Tri &t, uint32_t top, const Sub &sub) {
    const uint32_t lane = lane_id(), lt = (1u << lane) - 1u;
    const uint32_t *at = t.row(top);
    const uint32_t W = (top >> 5) + 1u;
    uint32_t q = 0;
    for (uint32_t w = lane; w - lane < W; w += 32) {
        const uint32_t n = w < W ? __popc(at[w]) : 0u;
        q += __reduce_add_sync(G2_FULL, n);
    }
    if (q < 3) return 0;
    if (q <= sub.cap) {
        uint32_t n = 0;
        for (uint32_t w = 0; w < W; w++) {
            const uint32_t bits = at[w];
            if ((bits >> lane) & 1u) sub.list[n + __popc(bits & lt)] = (uint16_t)((w << 5) + lane);
            n += __popc(bits);
        }
        __syncwarp();
        const Tri s{sub.rows};
        for (uint32_t c0 = 0; c0 < q; c0 += 32) {  // 32 members, a lane each
            const uint32_t j = c0 + lane, y = sub.list[j < q ? j : q - 1u];
            const uint32_t *old = t.row(y), ow = j < q ? (y >> 5) + 1u : 0u;
            const uint32_t last = __shfl_sync(G2_FULL, y, 31) >> 5;
            uint32_t *row = s.row(j);
            uint32_t acc = 0, done = 0;
            for (uint32_t w = 0; w <= last; w++) {
                const uint32_t x = w < ow ? old[w] : 0u;
                for (uint32_t m = at[w]; m; m &= m - 1) {  // uniform
                    acc = __funnelshift_r(acc, x >> (__ffs(m) - 1), 1);
                    if ((++done & 31u) == 0 && done <= c0 + 32u) row[(done >> 5) - 1u] = acc;
                }
            }
            if (done < c0 + 32u && (done & 31u)) row[done >> 5] = acc >> (32u - (done & 31u));
        }
        __syncwarp();
        const uint64_t c = triangles<false>(s, q, 0u, 1u);
        __syncwarp();  // the list and rows are free again
        return c;
    }
    uint64_t c = 0;
    for (uint32_t wz = 0; wz < W; wz++) {
        for (uint32_t m = at[wz]; m; m &= m - 1) {
            const uint32_t z = (wz << 5) + (uint32_t)(__ffs(m) - 1);
            const uint32_t *az = t.row(z);
            for (uint32_t w = lane; w <= wz; w += 32) sub.q[w] = at[w] & az[w];
            __syncwarp();
            uint32_t qn = 0;
            auto batch = [&](uint32_t n) {
                const uint32_t y = lane < n ? sub.queue[lane] : 0u, wy = y >> 5;
                const uint32_t *ay = t.row(y);
                const uint32_t wl = __shfl_sync(G2_FULL, wy, n - 1u);
                uint32_t k = 0;
                for (uint32_t w = 0; w <= wl; w++)
                    if (lane < n && w <= wy) k += __popc(sub.q[w] & ay[w]);
                c += k;
            };
            for (uint32_t w = 0; w <= wz; w++) {
                const uint32_t bits = sub.q[w];
                if (!bits) continue;
                if ((bits >> lane) & 1u) sub.queue[qn + __popc(bits & lt)] = (w << 5) + lane;
                qn += __popc(bits);
                __syncwarp();
                if (qn >= 32u) {
                    batch(32u);
                    const uint32_t keep = sub.queue[32u + lane];
                    __syncwarp();
                    sub.queue[lane] = keep;
                    qn -= 32u;
                    __syncwarp();
                }
            }
            if (qn) batch(qn);
            __syncwarp();  // queue and candidate row are free again
        }
    }
    return c;
}

struct Root {
    uint32_t task, v, p, part, nparts;
    uint64_t ids;  // P0 = ci[ids, ids + p)
};

__device__ __forceinline__ Root load_root(const CliqueArgs &a, uint32_t task) {
    Root r;
    r.task = task;
    r.v = a.tasks[task];
    const uint32_t tp = a.task_part ? a.task_part[task] : (1u << 16);
    r.nparts = tp >> 16;
    r.part = tp & 0xffffu;
    const uint64_t lo = ldg(a.rp + r.v), hi = ldg(a.rp + r.v + 1);
    r.ids = lo + ldg(a.fo + r.v);
    r.p = (uint32_t)(hi - r.ids);
    return r;
}

// Roots that leave the tiles to the general kernel's forward lists (the rest list).
// The tiles' cost does not depend on what they hold; the lists' follows the entries
// (`mean` per head, from 32 heads):
//  * far: more than a quarter of the heads (8 of a small root) have no bit row.  They
//    cost a binary search per column, the lists mean / 32 steps and a search each.
//    G(10^6, 4e-5) 4-cliques 2.4 ms by lists, 2.9 by tiles; G(2*10^5, 10^-3) 7.2 / 13.2.
//  * Roots of more than 64 vertices with hardly an entry: 4,000 roots over 800 vertices
//    without an edge, triangles 0.18 / 0.72 ms, 4-cliques 0.69 / 3.5, at a mean of 20
//    entries 2.8 / 0.72 and 5.5 / 3.5.
// A warp takes such a root's heads one after the other (0.4 ms for 600), so up to
// kManySparse of more than 64 vertices in a run stay with the tiles, but for very wide
// ones (a hub of 20,000 forward neighbours in generator ids: 24 / 102 to 371 ms).
constexpr uint32_t kFewHeads = 8;
constexpr uint32_t kSparseP = 64;  // up to here six tiles
constexpr uint32_t kWideP = 1024;
constexpr uint32_t kManySparse = 1024;
__device__ __forceinline__ bool heads_far(const CliqueArgs &a, const CoreBlock &b, uint64_t ids, uint64_t p) {
    return p > kFewHeads && ldg(a.ci + ids + (p <= 32u ? kFewHeads : p / 4u)) < b.base;
}
__device__ __forceinline__ uint32_t forward_length(const CliqueArgs &a, uint32_t u) {
    const uint64_t len = ldg(a.rp + u + 1) - ldg(a.rp + u) - ldg(a.fo + u);
    return (uint32_t)(len < (1u << 26) ? len : 1u << 26);
}
// A root of up to kSparseP vertices, per lane (from 4 heads).
__device__ __forceinline__ bool small_leaves_tiles(const CliqueArgs &a, const CoreBlock &b, uint64_t ids, uint64_t p) {
    if (!heads_far(a, b, ids, p)) return false;
    uint64_t sum = 0;
#pragma unroll
    for (uint32_t i = 0; i < 4; i++) sum += forward_length(a, ldg(a.ci + ids + p * (2 * i + 1) / 8u));
    return sum / 4u + 32u < 3u * p;
}
// A wider one (one warp).
__device__ __forceinline__ bool wide_leaves_tiles(const CliqueArgs &a, uint32_t k, const CoreBlock &b, uint64_t ids,
                                                  uint64_t p) {
    const uint32_t len = forward_length(a, ldg(a.ci + ids + p * lane_id() / 32u));
    const uint64_t mean = __reduce_add_sync(G2_FULL, len) / 32u;
    return mean * (k == 3 ? 128u : k == 4 ? 64u : 16u) < p || (mean + 32u < 3u * p && heads_far(a, b, ids, p));
}
// Does root r leave the tiles?  many: the run holds many such roots.  Warp-uniform.
__device__ __forceinline__ bool leaves_tiles(const CliqueArgs &a, uint32_t k, const CoreBlock &b, const Root &r,
                                             bool many) {
    if (r.p <= (many ? kSparseP : kWideP) || !a.by_cost) return false;  // (small ones: by the preparation)
    return wide_leaves_tiles(a, k, b, r.ids, r.p);
}
__device__ __forceinline__ bool many_sparse(const CliqueArgs &a) { return a.by_cost && a.counts[5] > kManySparse; }

// A root to the rest list (one lane).
__device__ __forceinline__ void to_rest(const CliqueArgs &a, uint32_t task) {
    a.lists[3 * a.list_cap + atomicAdd(a.counts + 3, 1ull)] = task;
    atomicOr(a.status, kStatusRest);
}

// p <= 32: lane j holds P0[j] and its row.  Warp total.
template <int K>
__device__ uint64_t root_small(const Csr &g, const CoreBlock &b, const Root &r, uint32_t id) {
    const uint32_t lane = lane_id(), p = r.p;
    const uint32_t last = __shfl_sync(G2_FULL, id, p - 1u);
    const uint32_t x = core_tile(g, b, lane < p ? id : last, p, lane < p ? id : last);
    const uint32_t row = lane < p ? x & ((1u << lane) - 1u) : 0u;
    uint32_t n = 0;
    if (K == 3) {
        if (r.nparts <= 1 || lane % r.nparts == r.part) n = __popc(row);
    } else {
        for (uint32_t z = K - 2; z < p; z++) {
            if (r.nparts > 1 && z % r.nparts != r.part) continue;
            const uint32_t rz = __shfl_sync(G2_FULL, row, z);
            if (K == 4) {
                if ((rz >> lane) & 1u) n += __popc(rz & row);
            } else {
                for (uint32_t m = rz & ~3u; m; m &= m - 1) {  // the vertex below z, with two more below it
                    const uint32_t q = rz & __shfl_sync(G2_FULL, row, __ffs(m) - 1);
                    if ((q >> lane) & 1u) n += __popc(q & row);
                }
            }
        }
    }
    return __reduce_add_sync(G2_FULL, n);
}

// Triangles of root r: edges of its local graph, by tiles k = first, first + step, ...
// Per-lane count; ~0 if the time budget ran out (looked at once per row of tiles).
template <bool BUDGET, class P0>
__device__ __forceinline__ uint64_t count_edges(const CliqueArgs &a, const Csr &g, const CoreBlock &b, P0 ids, const Root &r,
                                                uint32_t first, uint32_t step) {
    const uint32_t lane = lane_id();
    uint32_t c = 0, k = 0;
    for (uint32_t w = 0; 32u * w < r.p; w++) {
        if (BUDGET && past_deadline(a)) return ~0ull;
        const bool mine = r.nparts <= 1 || (32u * w + lane) % r.nparts == r.part;
        for (uint32_t q = 0; q <= w; q++, k++) {
            if (k % step != first) continue;
            const uint32_t x = local_word(g, b, ids, r.p, w, q);
            if (mine) c += __popc(x);
        }
    }
    return c;
}

// Rows of root r into t, by tiles k = first, first + step, ...  false if the time
// budget ran out (looked at once per row of tiles).
template <bool BUDGET, class P0>
__device__ __forceinline__ bool build_rows(const CliqueArgs &a, const Csr &g, const CoreBlock &b, P0 ids, uint32_t p, const Tri &t,
                                           uint32_t first, uint32_t step) {
    uint32_t k = 0;
    for (uint32_t w = 0; 32u * w < p; w++) {
        if (BUDGET && past_deadline(a)) return false;
        uint32_t *row = t.row(32u * w + lane_id());
        for (uint32_t q = 0; q <= w; q++, k++)
            if (k % step == first) row[q] = local_word(g, b, ids, p, w, q);
    }
    return true;
}

// One warp: rows in `A`, P0 at `ids`.  Warp total; ~0 if the time budget ran out.
template <int K, bool BUDGET, class P0>
__device__ __forceinline__ uint64_t root_warp(const CliqueArgs &a, const Csr &g, const CoreBlock &b, const Root &r,
                                              P0 ids, uint32_t *A, const Sub &sub) {
    if constexpr (K == 3) {
        const uint64_t n = count_edges<BUDGET>(a, g, b, ids, r, 0u, 1u);
        return BUDGET && n == ~0ull ? n : warp_sum_u64(n);
    }
    const Tri t{A};
    if (!build_rows<BUDGET>(a, g, b, ids, r.p, t, 0u, 1u) && BUDGET) return ~0ull;
    __syncwarp();
    uint64_t c = 0;
    if constexpr (K == 4) {
        c = triangles<BUDGET>(t, r.p, r.part, r.nparts, &a);
        if (BUDGET && c == ~0ull) return c;
    } else {
        for (uint32_t x = 3; x < r.p; x++) {
            if (r.nparts > 1 && x % r.nparts != r.part) continue;
            if (a.deadline && past_deadline(a)) return ~0ull;
            c += count_below(t, x, sub);
        }
    }
    __syncwarp();
    return warp_sum_u64(c);
}

// Credit a finished root (one lane).  Roots of budgeted runs are marked
// finished by a cost of at least 1.
__device__ __forceinline__ void credit(const CliqueArgs &a, uint32_t task, uint64_t c, long long c0) {
    if (a.root_nodes && c) atomicAdd(reinterpret_cast<unsigned long long *>(a.root_nodes + task), (unsigned long long)c);
    if (a.root_cost)
        atomicAdd(reinterpret_cast<unsigned long long *>(a.root_cost + task),
                  (unsigned long long)(clock64() - c0) + 1ull);
}

// Shared memory (words) of a warp's 5-clique work, of a warp that walks roots by
// itself, and of a warp of a CTA that shares a root (P0 and the rows follow).
__host__ __device__ __forceinline__ constexpr uint32_t sub_words(uint32_t cap, uint32_t q_words) {
    return cap / 2u + (uint32_t)tri_words(cap / 32u) + (q_words ? kQueue + q_words : 0u);
}
// in order, a warp also walks roots of more than kWarpP (rows in its slab)
__host__ __device__ __forceinline__ constexpr uint32_t warp_area(uint32_t k, bool in_order, uint32_t q_words) {
    return k == 3 ? kWarpP
                  : kWarpP + (uint32_t)tri_words(kWarpP / 32u) +
                        (k < 5 ? 0u : in_order ? sub_words(kSub, q_words) : sub_words(kWarpP, 0u));
}
__host__ __device__ __forceinline__ constexpr uint32_t cta_area(uint32_t k, uint32_t q_words) {
    return k < 5 ? 0u : sub_words(kSub, q_words);
}
__device__ __forceinline__ Sub make_sub(uint32_t *at, uint32_t cap) {
    Sub s;
    s.cap = cap;
    s.list = reinterpret_cast<uint16_t *>(at);
    s.rows = at + cap / 2u;
    s.queue = s.rows + (uint32_t)tri_words(cap / 32u);
    s.q = s.queue + kQueue;
    return s;
}

// One warp takes root r.  area: the warp's shared memory (P0, rows, 5-clique work).
template <int K, bool ORDER, bool BUDGET>
__device__ __forceinline__ void warp_task(const CliqueArgs &a, const Csr &g, const Root &r, uint32_t id,
                                          uint32_t *area, uint32_t *slab, bool many, uint64_t &total) {
    long long c0 = 0;
    if (a.root_cost) c0 = clock64();
    uint32_t *p0s = area, *A = area + kWarpP;
    const Sub sub = make_sub(A + (uint32_t)tri_words(kWarpP / 32u), ORDER ? kSub : kWarpP);  // (by size, 5-cliques: p <= kWarpP here)
    const uint32_t lane = lane_id();
    const CoreBlock b = core_block(a.core, r.v);
    uint64_t c = 0;
    if (past_deadline(a)) {
        c = ~0ull;
    } else if (leaves_tiles(a, K, b, r, many)) {
        if (lane == 0) to_rest(a, r.task);
        return;
    } else if (r.p <= 32u) {
        c = root_small<K>(g, b, r, id);
    } else if (r.p <= kWarpP) {
        p0s[lane] = id;
        for (uint32_t i = 32u + lane; i < r.p; i += 32) p0s[i] = ldg(a.ci + r.ids + i);
        __syncwarp();
        c = root_warp<K, BUDGET>(a, g, b, r, (const uint32_t *)p0s, A, sub);
        __syncwarp();
    } else if (ORDER) {
        c = root_warp<K, BUDGET>(a, g, b, r, a.ci + r.ids, slab, sub);
    }
    if (c == ~0ull) {
        if (lane == 0) atomicOr(a.status, kStatusDeadline);
    } else {
        total += c;
        if (lane == 0) credit(a, r.task, c, c0);
    }
}

// Warps take runs of `chunk` tasks of a list; the lanes read the tasks' roots
// (and the first 32 ids of P0 of the next one) ahead of the walk.
template <int K, bool ORDER, bool BUDGET>
__device__ __forceinline__ void warp_list(const CliqueArgs &a, const Csr &g, uint32_t list, uint32_t chunk,
                                          uint32_t *area, uint32_t *slab, bool many, uint64_t &total) {
    const uint32_t lane = lane_id();
    const uint32_t *ids = a.lists + (uint64_t)list * a.list_cap;
    const uint64_t n = a.counts[list];
    for (;;) {
        const uint64_t t0 = grab(a.heads + list, chunk);
        if (t0 >= n) break;
        const uint32_t m = (uint32_t)(t0 + chunk < n ? chunk : n - t0);
        Root mine{};
        if (lane < m) mine = load_root(a, ids[t0 + lane]);
        uint32_t next = 0;
        auto fetch = [&](uint32_t t) {
            const uint64_t at = __shfl_sync(G2_FULL, mine.ids, t);
            const uint32_t p = __shfl_sync(G2_FULL, mine.p, t);
            next = lane < p ? ldg(a.ci + at + lane) : 0u;
        };
        fetch(0);
        for (uint32_t t = 0; t < m; t++) {
            Root r;
            r.task = __shfl_sync(G2_FULL, mine.task, t);
            r.v = __shfl_sync(G2_FULL, mine.v, t);
            r.p = __shfl_sync(G2_FULL, mine.p, t);
            r.part = __shfl_sync(G2_FULL, mine.part, t);
            r.nparts = __shfl_sync(G2_FULL, mine.nparts, t);
            r.ids = __shfl_sync(G2_FULL, mine.ids, t);
            const uint32_t id = next;
            if (t + 1 < m) fetch(t + 1);
            warp_task<K, ORDER, BUDGET>(a, g, r, id, area, slab, many, total);
        }
    }
}

// The CTA's warps share each root of list 0.
template <int K, bool BUDGET>
__device__ __forceinline__ uint64_t cta_list(const CliqueArgs &a, const Csr &g, uint32_t *smem, bool many) {
    __shared__ uint32_t s_entry, s_next, s_expired, s_late, s_rest;
    __shared__ unsigned long long s_count;
    const uint32_t lane = lane_id(), wib = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint32_t *slab = a.scratch + (uint64_t)blockIdx.x * nw * a.words_per_warp;
    uint32_t *room = smem + nw * cta_area(K, a.q_words);
    const uint32_t room_words = a.smem_words - nw * cta_area(K, a.q_words);
    const Sub sub = make_sub(smem + wib * cta_area(K, a.q_words), kSub);
    const uint64_t n = a.counts[0];
    uint64_t sum = 0;
    for (;;) {
        if (wib == 0) {
            const bool late = past_deadline(a);
            if (lane == 0) {
                const unsigned long long t = atomicAdd(a.heads, 1ull);
                s_entry = t < n ? (uint32_t)t : 0xffffffffu;
                s_next = 0;
                s_late = s_expired = late;
                s_count = 0;
            }
        }
        __syncthreads();
        const uint32_t entry = s_entry;
        if (entry == 0xffffffffu) break;
        Root r = load_root(a, a.lists[entry]);
        bool first = true;  // of the root's pieces
        if (K == 5 && a.pieces) {  // piece of a heavy root
            const uint32_t piece = a.pieces[entry];
            first = (piece & 0xffffu) == 0;
            r.part += r.nparts * (piece & 0xffffu);
            r.nparts *= piece >> 16;
        }
        long long c0 = 0;
        if (a.root_cost) c0 = clock64();
        const CoreBlock b = core_block(a.core, r.v);
        const uint32_t W = (r.p + 31u) >> 5;
        const bool staged = r.p <= room_words;
        if (staged)
            for (uint32_t i = threadIdx.x; i < r.p; i += blockDim.x) room[i] = ldg(a.ci + r.ids + i);
        if (wib == nw - 1) {  // (while the others still load)
            const bool rest = !s_late && leaves_tiles(a, K, b, r, many);
            if (lane == 0) {
                s_rest = rest;  // (read by all before the next iteration's first barrier, written after it)
                if (rest && first) to_rest(a, r.task);
            }
        }
        __syncthreads();
        if (s_rest) continue;
        uint64_t c = 0;
        if (!s_late) {  // (else the time budget is spent: start no new root)
            if constexpr (K == 3) {
                if (staged) c = count_edges<BUDGET>(a, g, b, (const uint32_t *)room, r, wib, nw);
                else c = count_edges<BUDGET>(a, g, b, a.ci + r.ids, r, wib, nw);
                if (BUDGET && c == ~0ull) {
                    c = 0;
                    if (lane == 0) s_expired = 1;
                }
            } else {
                uint32_t *A = staged && tri_words(W) <= room_words - r.p ? room + r.p : slab;
                const Tri t{A};
                const bool built = staged ? build_rows<BUDGET>(a, g, b, (const uint32_t *)room, r.p, t, wib, nw)
                                          : build_rows<BUDGET>(a, g, b, a.ci + r.ids, r.p, t, wib, nw);
                if (BUDGET && !built && lane == 0) s_expired = 1;  // (the loop below ends at its first check, for all warps)
                __syncthreads();
                for (;;) {
                    uint32_t x = 0;
                    if (lane == 0) x = atomicAdd(&s_next, 1u);
                    x = __shfl_sync(G2_FULL, x, 0);
                    if (a.deadline && past_deadline(a)) {
                        if (lane == 0) s_expired = 1;
                        break;
                    }
                    if constexpr (K == 4) {  // chunk x of the row tiles
                        uint32_t w = 0;
                        while (w < W && x >= chunks_of(w)) x -= chunks_of(w), w++;
                        if (w >= W) break;
                        c += tile_chunk(t, r.p, w, x, r.part, r.nparts);
                    } else {  // highest vertex, the dearest first
                        if (x + 3 >= r.p) break;
                        const uint32_t top = r.p - 1u - x;
                        if (r.nparts > 1 && top % r.nparts != r.part) continue;
                        c += count_below(t, top, sub);
                    }
                }
            }
        }
        c = warp_sum_u64(c);
        if (lane == 0 && c) atomicAdd(&s_count, (unsigned long long)c);
        __syncthreads();
        if (threadIdx.x == 0) {
            if (s_expired) {
                atomicOr(a.status, kStatusDeadline);
            } else {
                sum += s_count;
                credit(a, r.task, s_count, c0);
            }
        }
    }
    __syncthreads();  // the warps' areas overlap the root's rows
    return sum;       // thread 0's
}

template <int K, bool ORDER, bool BUDGET>
__global__ void __launch_bounds__(256, K == 5 ? 4 : 5) clique_kernel(const __grid_constant__ CliqueArgs a) {
    extern __shared__ uint32_t smem[];
    const uint32_t lane = lane_id(), wib = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const Csr g{a.rp, a.ci, a.fo, a.core.bits};
    uint64_t total = 0;
    const bool many = many_sparse(a);
    if (!ORDER) total = cta_list<K, BUDGET>(a, g, smem, many);
    uint32_t *area = smem + wib * warp_area(K, ORDER, a.q_words);
    uint32_t *slab = a.scratch + ((uint64_t)blockIdx.x * nw + wib) * a.words_per_warp;
    uint64_t mine = 0;
    if (ORDER) {
        warp_list<K, true, BUDGET>(a, g, 0, a.chunk, area, slab, many, mine);
    } else {
        warp_list<K, false, BUDGET>(a, g, 1, 1u, area, slab, many, mine);
        warp_list<K, false, BUDGET>(a, g, 2, 8u, area, slab, many, mine);
    }
    if (lane == 0) total += mine;
    if (lane == 0 && total) atomicAdd(a.out, (unsigned long long)total);
}

// |P0| times the square of its vertices' neighbourhoods per CTA piece of a 5-clique root.
constexpr uint64_t kPieceCube = 1ull << 20;

// Segment of a bit row kept in a warp's shared memory while it is filled (words).
constexpr uint32_t kSeg = 512;

// Bit rows of the core (a warp per row, from row gw on): the forward list's
// entries set bits of a segment in shared memory, which is then stored whole.
__device__ __forceinline__ void core_rows(const CoreBits &c, const uint64_t *rp, const uint32_t *ci,
                                          const uint32_t *fo, uint32_t *out, uint32_t *seg, uint64_t gw,
                                          uint64_t nwarps) {
    const uint32_t lane = lane_id();
    for (uint64_t r = gw; r < c.rows; r += nwarps) {
        CoreBlock b = c.one;
        if (c.nblocks > 1) {  // last block with row0 <= r
            uint32_t lo = 0, hi = c.nblocks;
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) >> 1;
                if (c.blocks[mid].row0 <= r) lo = mid;
                else hi = mid;
            }
            b = c.blocks[lo];
        }
        const uint32_t x = (uint32_t)(r - b.row0), u = b.base + x;
        uint32_t *row = out + b.off + (uint64_t)x * b.stride;
        uint64_t e = ldg(rp + u) + ldg(fo + u);
        const uint64_t end = ldg(rp + u + 1);
        for (uint32_t w0 = (x >> 5) & ~3u; w0 < b.stride; w0 += kSeg) {  // words below the row's own are never read
            const uint32_t nw = b.stride - w0 < kSeg ? b.stride - w0 : kSeg;
            for (uint32_t w = 4u * lane; w < nw; w += 128) *reinterpret_cast<uint4 *>(seg + w) = make_uint4(0, 0, 0, 0);
            __syncwarp();
            const uint64_t stop = (uint64_t)b.base + 32ull * (w0 + nw);
            for (;;) {
                const uint32_t y = e + lane < end ? ldg(ci + e + lane) : 0xffffffffu;
                const bool in = e + lane < end && y < b.end && y < stop;
                const uint32_t c = y - b.base - 32u * w0;
                if (in && c < 32u * nw) atomicOr(seg + (c >> 5), 1u << (c & 31u));
                const uint32_t m = __popc(__ballot_sync(G2_FULL, in));
                e += m;
                if (m < 32u) break;
            }
            __syncwarp();
            for (uint32_t w = 4u * lane; w < nw; w += 128)
                *reinterpret_cast<uint4 *>(row + w0 + w) = *reinterpret_cast<const uint4 *>(seg + w);
            __syncwarp();
        }
    }
}

__global__ void __launch_bounds__(256) core_rows_kernel(const __grid_constant__ CoreBits c, const uint64_t *rp,
                                                        const uint32_t *ci, const uint32_t *fo, uint32_t *out) {
    __shared__ __align__(16) uint32_t seg_all[8][kSeg];
    core_rows(c, rp, ci, fo, out, seg_all[threadIdx.x >> 5],
              ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5, ((uint64_t)gridDim.x * blockDim.x) >> 5);
}

// Roots of a loaded graph that may leave the tiles (4 heads each; a very wide one
// counts as 1024).
__global__ void __launch_bounds__(256) sparse_roots_kernel(const __grid_constant__ CliqueArgs a, uint64_t n,
                                                           unsigned int *count) {
    unsigned int c = 0;
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t ids = ldg(a.rp + v) + ldg(a.fo + v), p = ldg(a.rp + v + 1) - ids;
        if (p <= kFewHeads) continue;
        if (p <= kSparseP) {
            c += small_leaves_tiles(a, a.core.one, ids, p);
            continue;
        }
        uint64_t sum = 0;
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) sum += forward_length(a, ldg(a.ci + ids + p * (2 * i + 1) / 8u));
        if (sum / 4u * 16u < p || (sum / 4u + 32u < 3u * p && heads_far(a, a.core.one, ids, p))) c += p > kWideP ? 1024u : 1u;
    }
    c = __reduce_add_sync(G2_FULL, c);
    if (lane_id() == 0 && c) atomicAdd(count, c < (1u << 20) ? c : 1u << 20);
}

// The task lists and the core's bit rows.
__global__ void __launch_bounds__(256) clique_prepare_kernel(const __grid_constant__ CliqueArgs a, uint32_t k) {
    __shared__ __align__(16) uint32_t seg_all[8][kSeg];
    const uint32_t lane = lane_id();
    const uint64_t gw = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    // ---- task lists
    const uint64_t nt = a.ntasks_dev ? (*a.ntasks_dev < a.ntasks ? *a.ntasks_dev : a.ntasks) : a.ntasks;
    for (uint64_t t0 = gw * 32; t0 < nt; t0 += nwarps * 32) {
        const uint64_t t = t0 + lane;
        int list = -1;
        uint32_t copies = 1;
        uint32_t v = 0;
        uint64_t ids = 0, p = 0;
        if (t < nt) {
            v = a.tasks[t];
            ids = ldg(a.rp + v) + ldg(a.fo + v);
            p = ldg(a.rp + v + 1) - ids;
        }
        bool sparse = false;
        if (a.by_cost) {
            const CoreBlock b = core_block(a.core, v);
            if (p + 1 >= k && p <= kSparseP) sparse = small_leaves_tiles(a, b, ids, p);
            // how many wider roots leave the tiles: the first of the 32 stands for all
            const uint32_t m = __ballot_sync(G2_FULL, p > kSparseP && p <= a.p_fit), l = m ? __ffs(m) - 1 : 0;
            const uint32_t lv = __shfl_sync(G2_FULL, v, l);
            if (m && wide_leaves_tiles(a, k, core_block(a.core, lv), __shfl_sync(G2_FULL, ids, l),
                                       __shfl_sync(G2_FULL, p, l)) && lane == 0)
                atomicAdd(a.counts + 5, (unsigned long long)__popc(m));
        }
        // share of the pairs in P0 that are edges, of 32 (5-cliques of wide roots, for their pieces)
        uint32_t share = 32;
        if (a.pieces && !a.in_order) {
            const bool look = p > a.cta_min && p <= a.p_fit && p * p * p > kPieceCube;
            for (uint32_t m = __ballot_sync(G2_FULL, look); m; m &= m - 1) {
                const uint32_t l = __ffs(m) - 1;
                const uint64_t half = __shfl_sync(G2_FULL, p, l) / 2u, at = __shfl_sync(G2_FULL, ids, l);
                const uint32_t u = ldg(a.ci + at + half * lane / 32u);
                const uint32_t y = ldg(a.ci + at + half + half * ((7u * lane + 3u) & 31u) / 32u);
                const bool hit = contains(a.ci, ldg(a.rp + u) + ldg(a.fo + u), ldg(a.rp + u + 1), y);
                const uint32_t hits = __popc(__ballot_sync(G2_FULL, hit));
                if (l == lane) share = hits ? hits : 1u;
            }
        }
        if (t < nt) {
            if (p + 1 < k) {  // no k-clique rooted here: finished
                if (a.root_cost) a.root_cost[t] = 1;
            } else if (p > a.p_fit || sparse) {
                list = 3;
            } else {
                list = a.in_order ? 0 : p > a.cta_min ? 0 : p > 32u ? 1 : 2;
                // 5-cliques of a wide root cost about p times the square of its
                // vertices' neighbourhoods: pieces of about kPieceCube, each a CTA's
                // share of the highest vertices
                const uint64_t in = p * share / 32u;
                if (a.pieces && list == 0 && !a.in_order && p * in * in > kPieceCube) {
                    const uint64_t want = p * in * in / kPieceCube + 1;
                    copies = (uint32_t)(want < 64 ? want : 64);
                    if (atomicAdd(a.counts + 4, copies - 1ull) + copies - 1 > a.extra_cap) copies = 1;
                }
            }
        }
        for (int l = 0; l < 4; l++) {
            const uint32_t m = __ballot_sync(G2_FULL, list == l);
            if (!m) continue;
            uint32_t incl = list == l ? copies : 0u;  // entries up to this lane's
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(G2_FULL, incl, o);
                if (lane >= (uint32_t)o) incl += y;
            }
            unsigned long long at = 0;
            if (lane == 31) {
                at = atomicAdd(a.counts + l, (unsigned long long)incl);
                if (l == 3) atomicOr(a.status, kStatusRest);
            }
            at = __shfl_sync(G2_FULL, at, 31);
            if (list != l) continue;
            at += incl - copies;
            for (uint32_t j = 0; j < copies; j++) {
                a.lists[(uint64_t)l * a.list_cap + at + j] = (uint32_t)t;
                if (a.pieces && l == 0) a.pieces[at + j] = (copies << 16) | j;
            }
        }
    }
    core_rows(a.core, a.rp, a.ci, a.fo, a.bits_out, seg_all[threadIdx.x >> 5], gw, nwarps);
}

}  // namespace

uint32_t clique_cta_min(uint32_t k) {
    return k == 5 ? 64u : kWarpP;
}

uint32_t clique_smem_words(uint32_t k, bool in_order, uint32_t max_fwd, int warps_per_block, uint32_t *q_words) {
    const uint32_t nw = (uint32_t)warps_per_block, W = (max_fwd + 31u) >> 5;
    // roots wider than kSub + 1 may hold neighbourhoods that are not compressed
    const uint32_t qw = k == 5 && max_fwd > kSub ? (W < kMaxQWords ? W : kMaxQWords) : 0u;
    *q_words = qw;
    uint32_t words = nw * warp_area(k, in_order, qw);
    if (!in_order) {
        // rows of the widest root in shared memory up to 44 KB per CTA (five CTAs
        // of 8 warps per SM), beyond that in the slab
        uint64_t need = max_fwd + (k == 3 ? 0ull : tri_words(W));
        const uint64_t cap = 11u * 1024u;
        if (need > cap) need = cap;
        const uint64_t cta = (uint64_t)nw * cta_area(k, qw) + need;
        if (cta > words) words = (uint32_t)cta;
    }
    return words;
}

bool clique_by_cost(uint32_t max_fwd, bool whole) { return !whole || max_fwd > kSparseP; }

uint32_t clique_p_fit(uint32_t k, bool in_order, uint64_t words_per_warp, int warps_per_block) {
    if (k == 3) return 1u << 18;  // (a lane counts a root's edges in 32 bits)
    uint64_t words = in_order ? words_per_warp : words_per_warp * (uint64_t)warps_per_block;
    uint32_t W = 0;
    const uint32_t wmax = k == 5 ? kMaxQWords : 4096u;
    while (W < wmax && tri_words(W + 1) <= words) W++;
    const uint32_t p = 32u * W;
    return p > kWarpP ? p : kWarpP;
}

template <int K, bool O>
static int clique_occ(int wpb, size_t sm) {
    cudaFuncSetAttribute(clique_kernel<K, O, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynamicSmem);
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, clique_kernel<K, O, false>, 32 * wpb, sm) != cudaSuccess) return 0;
    return nb;
}

int clique_blocks_per_sm(uint32_t k, bool in_order, int wpb, uint32_t smem_words) {
    const size_t sm = 4ull * smem_words;
    switch (k) {
        case 3: return in_order ? clique_occ<3, true>(wpb, sm) : clique_occ<3, false>(wpb, sm);
        case 4: return in_order ? clique_occ<4, true>(wpb, sm) : clique_occ<4, false>(wpb, sm);
        case 5: return in_order ? clique_occ<5, true>(wpb, sm) : clique_occ<5, false>(wpb, sm);
        default: return 0;
    }
}

cudaError_t core_rows_launch(const CoreBits &core, uint32_t *bits, const uint64_t *rp, const uint32_t *ci,
                             const uint32_t *fo, int sms, cudaStream_t st) {
    const uint64_t blocks = ((uint64_t)core.rows + 7) / 8, cap = 8ull * (uint64_t)sms;
    if (blocks) core_rows_kernel<<<(unsigned)(blocks < cap ? blocks : cap), 256, 0, st>>>(core, rp, ci, fo, bits);
    return cudaGetLastError();
}

cudaError_t sparse_roots_launch(const uint64_t *rp, const uint32_t *ci, const uint32_t *fo, uint64_t n,
                                const CoreBlock &core, int sms, unsigned int *count) {
    CliqueArgs a{};
    a.rp = rp, a.ci = ci, a.fo = fo, a.core.one = core;
    sparse_roots_kernel<<<8 * sms, 256>>>(a, n, count);
    return cudaGetLastError();
}

cudaError_t clique_prepare_launch(const CliqueArgs &a, uint32_t k, int sms, cudaStream_t st) {
    const uint64_t warps = (a.ntasks + 31) / 32 > a.core.rows ? (a.ntasks + 31) / 32 : a.core.rows;
    const uint64_t blocks = (warps + 7) / 8, cap = 8ull * (uint64_t)sms;
    clique_prepare_kernel<<<(unsigned)(blocks < 1 ? 1 : blocks < cap ? blocks : cap), 256, 0, st>>>(a, k);
    return cudaGetLastError();
}

cudaError_t clique_preload(uint32_t k, bool in_order) {
    cudaFuncAttributes fa;
    const cudaError_t e = cudaFuncGetAttributes(&fa, clique_prepare_kernel);
    if (e != cudaSuccess) return e;
    switch (k) {
        case 3: return in_order ? cudaFuncGetAttributes(&fa, clique_kernel<3, true, true>) : cudaFuncGetAttributes(&fa, clique_kernel<3, false, true>);
        case 4: return in_order ? cudaFuncGetAttributes(&fa, clique_kernel<4, true, true>) : cudaFuncGetAttributes(&fa, clique_kernel<4, false, true>);
        case 5: return in_order ? cudaFuncGetAttributes(&fa, clique_kernel<5, true, true>) : cudaFuncGetAttributes(&fa, clique_kernel<5, false, true>);
        default: return cudaErrorInvalidValue;
    }
}

template <int K, bool O, bool B>
static void clique_go_budget(const CliqueArgs &a, int blocks, int wpb, cudaStream_t st) {
    cudaFuncSetAttribute(clique_kernel<K, O, B>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynamicSmem);
    clique_kernel<K, O, B><<<blocks, 32 * wpb, 4ull * a.smem_words, st>>>(a);
}

template <int K, bool O>
static void clique_go(const CliqueArgs &a, int blocks, int wpb, cudaStream_t st) {
    if (a.deadline) clique_go_budget<K, O, true>(a, blocks, wpb, st);
    else clique_go_budget<K, O, false>(a, blocks, wpb, st);
}

cudaError_t clique_launch(const CliqueArgs &a, uint32_t k, int blocks, int wpb, cudaStream_t st) {
    switch (k) {
        case 3: a.in_order ? clique_go<3, true>(a, blocks, wpb, st) : clique_go<3, false>(a, blocks, wpb, st); break;
        case 4: a.in_order ? clique_go<4, true>(a, blocks, wpb, st) : clique_go<4, false>(a, blocks, wpb, st); break;
        case 5: a.in_order ? clique_go<5, true>(a, blocks, wpb, st) : clique_go<5, false>(a, blocks, wpb, st); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace g2
