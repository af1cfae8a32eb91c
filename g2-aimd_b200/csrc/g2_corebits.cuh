// g2_corebits.cuh - adjacency of the graph's last ids (its dense core, in
// degeneracy order) as a bit matrix, and tiles of a root's local adjacency
// read from it.
//
// The local graph of a root v lives on P0 = N(v) ∩ (v, ∞), p sorted ids; row j
// of it is the set of i < j with P0[j] in N+(P0[i]).  Scanning N+(P0[i]) for
// members of P0 reads every entry of it (4.4e9 entries over the roots of R-MAT
// s20) to find the 10 % that are in P0.  With N+(u) as a bit row, 32 columns j
// are tested against a head i by one load and two shifts: 7.1e7 warp steps for
// the same graph.  Only the last K ids have bit rows (K^2 bits); ids grow with
// the core number, so on R-MAT s20 93 % of the heads have one.  Columns of an
// earlier head binary-search in its (short) forward list, 32 at a time.
//
// The matrix is a workspace: every run builds it from the CSR.
#pragma once

#include <cstdint>

#include "g2_device.cuh"
#include "g2_kernels.h"

namespace g2 {

// The block whose graph holds vertex v (one block, or one per graph of a batch).
__device__ __forceinline__ CoreBlock core_block(const CoreBits &c, uint32_t v) {
    if (c.nblocks <= 1) return c.one;
    uint32_t lo = 0, hi = c.nblocks;  // first block with end > v
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(&c.blocks[mid].end) <= v) lo = mid + 1;
        else hi = mid;
    }
    if (lo >= c.nblocks) lo = c.nblocks - 1;
    return c.blocks[lo];
}

struct Csr {
    const uint64_t *rp;
    const uint32_t *ci;
    const uint32_t *fo;
    const uint32_t *bits;
};

// Tile of a local graph: lane = column (id `cid`, in order after or among the
// heads), heads = the first nh lanes' `hid`; on return bit i of a lane's word
// says whether its column is a forward neighbour of head i.  Bits of columns
// that do not come after the head in P0 are unspecified (the caller masks
// them).  Lanes beyond P0 pass any id of P0 and mask their word.  With LISTS =
// false the bits of heads without a bit row stay 0 (see list_rows).
template <bool LISTS = true>
__device__ __forceinline__ uint32_t core_tile(const Csr &g, const CoreBlock &b, uint32_t hid, uint32_t nh,
                                              uint32_t cid) {
    const uint32_t nout = __popc(__ballot_sync(G2_FULL, hid < b.base) & (nh >= 32u ? G2_FULL : (1u << nh) - 1u));
    // ids below the block only occur as columns before the head: any column will do
    const uint32_t c = cid >= b.base ? cid - b.base : 0u;
    const char *bits = reinterpret_cast<const char *>(g.bits + b.off);
    const uint32_t col = (c >> 5) * 4u;
    const uint32_t hrow = (hid - b.base) * (b.stride * 4u);  // K^2 / 8 < 2^32 bytes
    uint32_t acc = 0;
    auto word = [&](uint32_t h) {
        return ldg(reinterpret_cast<const uint32_t *>(bits + (col + __shfl_sync(G2_FULL, hrow, h))));
    };
    if (nout == 0 && nh >= 32u) {
#pragma unroll
        for (int h = 0; h < 32; h += 8) {  // eight independent loads in flight
            uint32_t x[8];
#pragma unroll
            for (int t = 0; t < 8; t++) x[t] = word(h + t);
#pragma unroll
            for (int t = 0; t < 8; t++) acc = __funnelshift_r(acc, x[t] >> (c & 31u), 1);
        }
        return acc;
    }
    // heads without a bit row come first (ids are sorted): four binary searches
    // in step, so that four loads are in flight
    uint32_t h = 0;
    for (; LISTS && h < nout; h += 4) {
        const uint32_t *list[4];
        uint32_t len[4], pos[4], most = 0;
#pragma unroll
        for (int t = 0; t < 4; t++) {
            const uint32_t u = __shfl_sync(G2_FULL, hid, h + t < nout ? h + t : h);
            const uint64_t e0 = ldg(g.rp + u) + ldg(g.fo + u);
            list[t] = g.ci + e0;
            len[t] = (uint32_t)(ldg(g.rp + u + 1) - e0);
            pos[t] = 0;
            most = len[t] > most ? len[t] : most;
        }
        for (uint32_t step = most ? 1u << (31 - __clz(most)) : 0u; step; step >>= 1) {
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const uint32_t q = pos[t] + step;
                if (q <= len[t] && ldg(list[t] + (q - 1u)) < cid) pos[t] = q;
            }
        }
#pragma unroll
        for (int t = 0; t < 4; t++) {
            const bool hit = pos[t] < len[t] && ldg(list[t] + pos[t]) == cid;
            if (h + t < nout) acc = __funnelshift_r(acc, hit ? 1u : 0u, 1);
        }
    }
    for (h = nout; h + 4 <= nh; h += 4) {
        uint32_t x[4];
#pragma unroll
        for (int t = 0; t < 4; t++) x[t] = word(h + t);
#pragma unroll
        for (int t = 0; t < 4; t++) acc = __funnelshift_r(acc, x[t] >> (c & 31u), 1);
    }
    for (; h < nh; h++) acc = __funnelshift_r(acc, word(h) >> (c & 31u), 1);
    return nh >= 32u ? acc : acc >> (32u - nh);
}

// Rows over P0 (ids, p of them) of up to 32 heads before P0, a lane each, from
// their forward lists: put(j) sets bit j of the lane's row.  For heads without a
// bit row that come in numbers (back neighbours of the dense core: short lists,
// which 32 lanes read at once where core_tile would search them four at a time).
template <class F>
__device__ __forceinline__ void list_rows(const Csr &g, const uint32_t *ids, uint32_t p, uint32_t head, bool on, F put) {
    if (on) {
        const uint32_t first = ids[0], last = ids[p - 1u];
        const uint64_t end = ldg(g.rp + head + 1);
        uint64_t e = lower_bound(g.ci, ldg(g.rp + head) + ldg(g.fo + head), end, first);
        uint32_t j = 0;
        for (; e < end && j < p; e++) {
            const uint32_t y = ldg(g.ci + e);
            if (y > last) break;
            uint32_t hi = p;
            while (j < hi) {
                const uint32_t mid = (j + hi) >> 1;
                if (ids[mid] < y) j = mid + 1;
                else hi = mid;
            }
            if (j < p && ids[j] == y) put(j);
        }
    }
    __syncwarp();
}

}  // namespace g2
