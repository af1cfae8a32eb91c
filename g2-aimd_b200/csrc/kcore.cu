// kcore.cu - degeneracy order of the loaded graph on the device, and the
// recode that renames vertices by it.
//
// Replaces the host preprocessing of kmeans/kcore.cpp:39-191 (k-core peeling,
// then a degree sort inside each shell and a recode): core numbers by peeling
// level after level in one launch (every vertex of remaining degree <= k leaves,
// its live neighbours lose one degree each; core numbers are unique, so any
// peeling order gives the same ones), then the order (core, degree, id)
// ascending by a stable radix sort of core above degree over ids, of the bits in
// use only.  The
// result equals g2_degeneracy_order's (csrc/host/graph_host.cpp) exactly.
#include <cub/cub.cuh>

#include <algorithm>
#include <climits>
#include <cstdint>
#include <cstdlib>
#include <vector>

#include "g2_device.cuh"
#include "g2_kernels.h"

namespace g2 {

namespace {

// Peeling in one launch.  A level-synchronous peel in separate launches took a
// thousand rounds of three launches and two host round trips each (R-MAT s18:
// about 30 ms; this kernel 3.4 ms, bound by the barriers of some 400 levels and
// their rounds and the latency of each round's dependent accesses).  Here one CTA
// per SM stays resident
// and the levels are separated by a grid barrier; within a level no order
// matters, so a warp that drops a neighbour to degree k claims it and walks on
// from its own queue (the rounds inside a level disappear).
//
//  * deg[u] of an unclaimed vertex is its live degree and stays above the level
//    k; a vertex is claimed once, by whoever swaps its core number in (the scan
//    at the level's start, or the warp whose decrement returned k + 1);
//  * every warp keeps its share of the vertices as a list that each scan compacts;
//  * a warp walks narrow vertices from its own queue, a few per round; the others
//    (and every vertex of more than kNarrow neighbours) become pieces of kPiece
//    neighbours on a list that all warps share in the next round, so a collapsing
//    core is spread over the chip (left to the warps that claimed its vertices,
//    one warp walked most of it alone: 40 ms on R-MAT s18);
//  * per-round counters rotate through four slots: written in round r, read after
//    its barrier, cleared in round r + 2 (when every CTA has read them).
constexpr uint32_t kPeelThreads = 1024, kPeelWarps = kPeelThreads / 32;
constexpr uint32_t kPeelQueue = 64;       // vertices in a warp's queue
constexpr uint32_t kNarrow = 64;          // neighbours of a vertex its claimer walks
constexpr uint32_t kPeelLocal = 24;       // vertices a warp walks from its queue per round
constexpr uint32_t kPiece = 256;          // neighbours per entry of the shared list
constexpr uint32_t kNoCore = 0xffffffffu;
constexpr long long kPeelWait = 1ll << 37;  // longest wait at the grid barrier (SM cycles, ~70 s)

struct PeelCtl {
    unsigned long long arrived;      // grid barrier: arrivals so far
    unsigned long long claims[4];    // vertices claimed in the round
    unsigned long long nshared[4];   // entries of the round's shared list
    unsigned int min_inv[4];         // ~(smallest degree left by the scan), 0 = none
    unsigned int max_deg, max_core;  // for the sort's bit count
    unsigned int timeout;            // a barrier wait ran out
    unsigned int rounds;
};

__device__ __forceinline__ unsigned long long peel_load(const unsigned long long *p) {
    return *reinterpret_cast<const volatile unsigned long long *>(p);
}

__global__ void __launch_bounds__(kPeelThreads, 1) peel_kernel(const uint64_t *rp, const uint32_t *ci, uint64_t n,
                                                              uint32_t *deg, uint32_t *core, uint32_t *list,
                                                              uint64_t share, uint64_t *shared_list,
                                                              uint64_t shared_cap, PeelCtl *ctl,
                                                              long long wait_cycles) {
    __shared__ uint32_t s_queue[kPeelWarps][kPeelQueue];
    __shared__ unsigned long long s_claims, s_nshared;
    __shared__ unsigned int s_min, s_bad;
    const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5, lt = (1u << lane) - 1u;
    const uint64_t w = (uint64_t)blockIdx.x * kPeelWarps + wib, nw = (uint64_t)gridDim.x * kPeelWarps;
    uint32_t *queue = s_queue[wib];
    uint32_t qn = 0;
    uint64_t claimed = 0;                  // by this warp in this round
    // this warp's share: ids lane + 32 (w + nw j), at list + w * share
    uint32_t *mine = list + w * share;
    uint64_t left = 0;
    {
        uint32_t top = 0;
        for (uint64_t c = w; c * 32 < n; c += nw) {
            const uint64_t v = c * 32 + lane;
            const bool in = v < n;
            if (in) {
                const uint32_t d = (uint32_t)(rp[v + 1] - rp[v]);
                deg[v] = d;
                core[v] = kNoCore;
                mine[left + lane] = (uint32_t)v;
                top = d > top ? d : top;
            }
            left += __popc(__ballot_sync(G2_FULL, in));
        }
        top = __reduce_max_sync(G2_FULL, top);
        if (lane == 0 && top) atomicMax(&ctl->max_deg, top);
    }
    unsigned long long barriers = 0;
    // all CTAs have arrived, or (false) the wait ran out: everybody leaves
    auto barrier = [&]() -> bool {
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) {
            const unsigned long long want = ++barriers * gridDim.x;
            atomicAdd(&ctl->arrived, 1ull);
            const long long t0 = clock64();
            s_bad = 0;
            while (peel_load(&ctl->arrived) < want) {
                if (clock64() - t0 > wait_cycles || *reinterpret_cast<volatile unsigned int *>(&ctl->timeout)) {
                    atomicExch(&ctl->timeout, 1u);
                    s_bad = 1;
                    break;
                }
            }
            __threadfence();
        }
        __syncthreads();
        return s_bad == 0;
    };
    if (!barrier()) return;
    uint32_t k = 0;
    uint64_t removed = 0, level_claims = 0;
    uint64_t coop = 0;  // shared entries of this round (0: a scan)
    for (uint32_t r = 0;; r++) {
        uint64_t *out = shared_list + (uint64_t)((r + 1) & 1u) * shared_cap;
        const uint64_t *in_list = shared_list + (uint64_t)(r & 1u) * shared_cap;
        unsigned long long *nout = ctl->nshared + (r + 1) % 4;
        uint32_t budget = kPeelLocal;
        if (blockIdx.x == 0 && threadIdx.x == 0) {  // the slots of round r + 2
            ctl->claims[(r + 2) % 4] = 0;
            ctl->nshared[(r + 2) % 4] = 0;
            ctl->min_inv[(r + 2) % 4] = 0;
        }
        // one vertex per lane (where `on`) onto the shared list, in pieces: entry =
        // piece above the vertex
        auto publish = [&](bool on, uint32_t v) {
            const uint32_t pieces = on ? ((uint32_t)(rp[v + 1] - rp[v]) + kPiece - 1u) / kPiece : 0u;
            uint32_t inc = pieces;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(G2_FULL, inc, o);
                if (lane >= (uint32_t)o) inc += y;
            }
            unsigned long long at = 0;
            if (lane == 31 && inc) at = atomicAdd(nout, (unsigned long long)inc);
            at = __shfl_sync(G2_FULL, at, 31) + inc - pieces;
            for (uint32_t j = 0; j < pieces; j++) out[at + j] = ((uint64_t)j << 32) | v;
            __syncwarp();
        };
        // claimed vertices (one per lane where `on`) onto the queue or the shared list
        auto push = [&](bool on, uint32_t v) {
            const bool narrow = on && (uint32_t)(rp[v + 1] - rp[v]) <= kNarrow;
            const uint32_t m = __ballot_sync(G2_FULL, narrow);
            const uint32_t at = qn + __popc(m & lt);
            const bool fits = narrow && at < kPeelQueue;
            if (fits) queue[at] = v;
            qn += __popc(m);
            if (qn > kPeelQueue) qn = kPeelQueue;
            claimed += __popc(__ballot_sync(G2_FULL, on));
            if (__any_sync(G2_FULL, on && !fits)) publish(on && !fits, v);
            __syncwarp();
        };
        // entries [e, end) of the adjacency: each live neighbour loses one degree
        // (four per lane at a time, so that four chains of dependent accesses overlap)
        auto walk = [&](uint64_t e, uint64_t end) {
            for (; e < end; e += 128) {  // warp-uniform
                uint32_t u[4], d[4];
                bool live[4], got[4];
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    const uint64_t x = e + 32 * t + lane;
                    live[t] = x < end;
                    u[t] = live[t] ? ldg(ci + x) : 0u;
                }
#pragma unroll
                for (int t = 0; t < 4; t++) live[t] = live[t] && __ldcg(deg + u[t]) > k;
#pragma unroll
                for (int t = 0; t < 4; t++) d[t] = live[t] ? atomicSub(deg + u[t], 1u) : 0u;
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    got[t] = live[t] && d[t] == k + 1u && atomicCAS(core + u[t], kNoCore, k) == kNoCore;
                    if (live[t] && d[t] <= k) atomicAdd(deg + u[t], 1u);  // claimed meanwhile
                }
#pragma unroll
                for (int t = 0; t < 4; t++)
                    if (__any_sync(G2_FULL, got[t])) push(got[t], u[t]);
            }
        };
        auto drain = [&]() {  // the queue, as far as the round's budget goes
            while (qn && budget) {
                const uint32_t v = queue[--qn];
                budget--;
                __syncwarp();
                walk(rp[v], rp[v + 1]);
            }
        };
        if (coop) {  // the shared list, a piece per warp in turn
            for (uint64_t i = w; i < coop; i += nw) {
                const uint64_t x = __ldcg(reinterpret_cast<const unsigned long long *>(in_list + i));
                const uint32_t v = (uint32_t)x;
                const uint64_t e = rp[v] + (x >> 32) * kPiece, end = rp[v + 1];
                walk(e, e + kPiece < end ? e + kPiece : end);
                drain();
            }
        } else {  // this warp's vertices: degree <= k leaves, the others stay listed
            uint64_t kept = 0;
            uint32_t low = 0;  // ~(smallest degree kept)
            for (uint64_t i = 0; i < left; i += 32) {
                const bool in = i + lane < left;
                const uint32_t v = in ? mine[i + lane] : 0u;
                const uint32_t d = in ? __ldcg(deg + v) : 0u;
                const bool stay = in && d > k;
                const bool got = in && !stay && atomicCAS(core + v, kNoCore, k) == kNoCore;
                const uint32_t m = __ballot_sync(G2_FULL, stay);  // all lanes have read their entries
                if (stay) {
                    mine[kept + __popc(m & lt)] = v;
                    low = ~d > low ? ~d : low;
                }
                kept += __popc(m);
                if (__any_sync(G2_FULL, got)) push(got, v);
            }
            left = kept;
            low = __reduce_max_sync(G2_FULL, low);
            if (lane == 0 && low) atomicMax(&ctl->min_inv[r % 4], low);
            drain();
        }
        for (; qn; qn -= qn < 32u ? qn : 32u) {  // what the budget left is shared
            const bool on = lane < qn;
            publish(on, on ? queue[qn - 1u - lane] : 0u);
        }
        if (lane == 0 && claimed) atomicAdd(&ctl->claims[r % 4], (unsigned long long)claimed);
        claimed = 0;
        const bool scan = coop == 0;
        if (!barrier()) return;
        if (threadIdx.x == 0) {
            s_claims = peel_load(&ctl->claims[r % 4]);
            s_nshared = peel_load(nout);
            s_min = ~*reinterpret_cast<volatile unsigned int *>(&ctl->min_inv[r % 4]);
        }
        __syncthreads();
        removed += s_claims;
        level_claims += s_claims;
        coop = s_nshared;
        if (coop) continue;
        if (removed >= n) {
            if (blockIdx.x == 0 && threadIdx.x == 0) {
                ctl->max_core = k;
                ctl->rounds = r + 1;
            }
            return;
        }
        // a level that removed nothing left every degree as its scan saw it
        k = scan && level_claims == 0 && s_min > k ? s_min : k + 1;
        level_claims = 0;
    }
}

// Sort keys (core number above the degree, dbits bits) and ids.
template <class Key>
__global__ void order_keys_kernel(const uint64_t *rp, const uint32_t *core, uint64_t n, int dbits, Key *keys,
                                  uint32_t *ids) {
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
        keys[v] = ((Key)core[v] << dbits) | (Key)(rp[v + 1] - rp[v]);
        ids[v] = (uint32_t)v;
    }
}

__global__ void scatter_perm_kernel(const uint32_t *ord, uint64_t n, uint32_t *perm) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        perm[ord[i]] = (uint32_t)i;
}

// Row length of each vertex under its new name (entry n stays 0 for the scan).
__global__ void recode_degrees_kernel(const uint64_t *rp, const uint32_t *perm, uint64_t n, uint64_t *deg) {
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x)
        deg[perm[v]] = rp[v + 1] - rp[v];
}

// Row of v, renamed, written unsorted at its new place (a warp per row; rows of
// big_min entries or more are listed instead).
__global__ void recode_scatter_kernel(const uint64_t *rp, const uint32_t *ci, const uint32_t *perm,
                                      const uint64_t *new_rp, uint64_t n, uint64_t big_min, uint32_t *big,
                                      unsigned long long *nbig, uint32_t *out) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t w0 = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t v = w0; v < n; v += nw) {
        const uint64_t lo = rp[v], len = rp[v + 1] - lo, base = new_rp[perm[v]];
        if (len >= big_min) {
            if (lane == 0) big[atomicAdd(nbig, 1ull)] = (uint32_t)v;
            continue;
        }
        for (uint64_t i = lane; i < len; i += 32) out[base + i] = perm[ci[lo + i]];
    }
}

// Listed rows (distinct ids), renamed and sorted by a bitmap of the new ids in
// shared memory, a CTA per row and kSpan ids at a time: the cost is the row's
// entries plus one look at every word of the bitmap, whatever the order.  A row
// that names a neighbour twice (not a deduplicated list) yields fewer ids than it
// has entries: *repeated is set and the caller sorts all rows instead.  CUB's
// segmented sort gives such a row to one CTA for four radix passes over global
// memory (R-MAT s18: 978 us, and 756 us to scatter the rows a warp each; measured
// with rows of 1024 entries on here: 85 + 135 us, and 846 us left in the segmented
// sort; the line stands at n / 1024 entries, 256 there).
constexpr uint32_t kSpanWords = 32768, kSpan = 32u * kSpanWords;  // 128 KB of shared memory
// rows from here on: a row costs a look at n / 32 words, so longer rows for more vertices
inline uint64_t big_row(uint64_t n) { return n >> 10 > 256 ? n >> 10 : 256; }
constexpr uint64_t kBigVertices = 4ull * kSpan;  // more vertices: too many passes over the row
__global__ void __launch_bounds__(1024, 1) recode_big_rows_kernel(const uint64_t *rp, const uint32_t *ci,
                                                                  const uint32_t *perm, const uint64_t *new_rp,
                                                                  uint64_t n, const uint32_t *big,
                                                                  const unsigned long long *nbig,
                                                                  unsigned long long *repeated, uint32_t *out) {
    extern __shared__ uint32_t s_map[];
    __shared__ uint32_t s_count[32];
    const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
    const uint64_t nb = *nbig;
    for (uint64_t i = blockIdx.x; i < nb; i += gridDim.x) {
        const uint32_t v = big[i];
        const uint64_t lo = rp[v], hi = rp[v + 1];
        uint64_t base = new_rp[perm[v]];
        for (uint64_t id0 = 0; id0 < n; id0 += kSpan) {
            const uint32_t words = (uint32_t)(n - id0 < kSpan ? (n - id0 + 31) / 32 : kSpanWords);
            for (uint32_t x = threadIdx.x; x < words; x += blockDim.x) s_map[x] = 0u;
            __syncthreads();
            for (uint64_t e = lo + threadIdx.x; e < hi; e += blockDim.x) {
                const uint64_t y = (uint64_t)ldg(perm + ldg(ci + e)) - id0;  // wraps below the span
                if (y < kSpan) atomicOr(s_map + (y >> 5), 1u << (y & 31u));
            }
            __syncthreads();
            // the warps' runs of words: bits before each, then the ids
            const uint32_t per = ((words + 31u) / 32u + 31u) & ~31u, x0 = wib * per, x1 = x0 + per < words ? x0 + per : words;
            uint32_t c = 0;
            for (uint32_t x = x0 + lane; x < x1; x += 32) c += __popc(s_map[x]);
            c = __reduce_add_sync(G2_FULL, c);
            if (lane == 0) s_count[wib] = c;
            __syncthreads();
            const uint32_t mine = s_count[lane];
            uint64_t at = base + __reduce_add_sync(G2_FULL, lane < wib ? mine : 0u);
            base += __reduce_add_sync(G2_FULL, mine);
            for (uint32_t x = x0; x < x1; x += 32) {
                uint32_t m = x + lane < x1 ? s_map[x + lane] : 0u;
                const uint32_t cnt = __popc(m);
                uint32_t inc = cnt;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(G2_FULL, inc, o);
                    if (lane >= (uint32_t)o) inc += y;
                }
                uint64_t q = at + inc - cnt;
                for (; m; m &= m - 1) out[q++] = (uint32_t)(id0 + 32ull * (x + lane) + (uint32_t)(__ffs(m) - 1));
                at += __shfl_sync(G2_FULL, inc, 31);
            }
            __syncthreads();  // the bitmap is free again
        }
        if (threadIdx.x == 0 && base != new_rp[perm[v]] + (hi - lo)) *repeated = 1ull;
    }
}

// Offsets of rows [r0, r0 + rows) relative to row r0 (segmented sort of one
// chunk): where each begins, and where it ends (at its start, so that nothing
// is sorted, for rows of big_min entries or more).
__global__ void chunk_offsets_kernel(const uint64_t *new_rp, uint64_t r0, uint64_t rows, uint64_t big_min, int *off,
                                     int *end) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < rows; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t a = new_rp[r0 + i], b = new_rp[r0 + i + 1];
        off[i] = (int)(a - new_rp[r0]);
        end[i] = (int)((b - a < big_min ? b : a) - new_rp[r0]);
    }
}

}  // namespace

// Sort every row of a CSR whose row pointers (device, n+1) are rp: the rows of
// `in` are sorted into `out`, in CUB segmented-sort calls of at most max_chunk
// entries (CUB counts items and segments in int).  A row longer than max_chunk:
// cudaErrorNotSupported.  Rows of big_min entries or more are left alone.
// Synchronous.
cudaError_t sort_rows_device(const uint64_t *rp, uint64_t n, uint64_t m, const uint32_t *in, uint32_t *out,
                             uint64_t max_chunk, int sms, uint64_t big_min) {
    max_chunk = std::min<uint64_t>(std::max<uint64_t>(max_chunk, 1), (uint64_t)INT_MAX);
    int *off = nullptr;
    uint64_t off_cap = 0;
    void *cub_tmp = nullptr;
    size_t cub_bytes = 0, need = 0;
    cudaError_t e = cudaSuccess;
    auto ok = [&](cudaError_t r) {
        if (e == cudaSuccess) e = r;
        return e == cudaSuccess;
    };
    const int G = sms * 8;
    uint32_t *tmp = const_cast<uint32_t *>(in);
    const uint64_t *nrp = rp;
    std::vector<uint64_t> cuts;  // row boundaries of the sort calls
    if (m <= max_chunk) {
        cuts = {0, n};
    } else {
        std::vector<uint64_t> h(n + 1);
        if (!ok(cudaMemcpy(h.data(), nrp, 8 * (n + 1), cudaMemcpyDeviceToHost))) goto done;
        cuts.push_back(0);
        uint64_t r = 0;
        while (r < n) {
            if (h[r + 1] - h[r] > max_chunk) {
                e = cudaErrorNotSupported;
                goto done;
            }
            // the last row r1 with h[r1] - h[r] <= max_chunk
            const uint64_t r1 =
                (uint64_t)(std::upper_bound(h.begin() + r, h.end(), h[r] + max_chunk) - h.begin()) - 1;
            r = std::min<uint64_t>(r1, n);
            cuts.push_back(r);
        }
    }
    for (size_t k = 0; k + 1 < cuts.size(); k++) {
        const uint64_t r0 = cuts[k], rows = cuts[k + 1] - r0;
        if (!rows) continue;
        uint64_t base = 0, items = m;
        if (cuts.size() > 2) {
            if (!ok(cudaMemcpy(&base, nrp + r0, 8, cudaMemcpyDeviceToHost)) ||
                !ok(cudaMemcpy(&items, nrp + r0 + rows, 8, cudaMemcpyDeviceToHost)))
                goto done;
            items -= base;
        }
        if (!items) continue;
        if (rows + 1 > (uint64_t)INT_MAX) {
            e = cudaErrorNotSupported;
            goto done;
        }
        if (rows > off_cap) {
            cudaFree(off);
            off = nullptr;
            off_cap = rows;
            if (!ok(cudaMalloc(&off, 2 * sizeof(int) * rows))) goto done;
        }
        chunk_offsets_kernel<<<G, 256>>>(nrp, r0, rows, big_min, off, off + rows);
        need = 0;
        if (!ok(cub::DeviceSegmentedSort::SortKeys(nullptr, need, tmp + base, out + base, (int)items, (int)rows, off,
                                                    off + rows)))
            goto done;
        if (need > cub_bytes) {
            cudaFree(cub_tmp);
            cub_tmp = nullptr;
            cub_bytes = need;
            if (!ok(cudaMalloc(&cub_tmp, cub_bytes))) goto done;
        }
        if (!ok(cub::DeviceSegmentedSort::SortKeys(cub_tmp, need, tmp + base, out + base, (int)items, (int)rows, off,
                                                    off + rows)))
            goto done;
    }
    ok(cudaGetLastError());
    ok(cudaDeviceSynchronize());
done:
    cudaFree(off);
    cudaFree(cub_tmp);
    return e;
}

cudaError_t recode_device(const uint64_t *rp, const uint32_t *ci, uint64_t n, uint64_t m, const uint32_t *perm,
                          uint64_t max_chunk, int sms, uint64_t **new_rp, uint32_t **new_ci) {
    *new_rp = nullptr;
    *new_ci = nullptr;
    if (n + 1 > (uint64_t)INT_MAX) return cudaErrorNotSupported;  // the scan counts items in int
    max_chunk = std::min<uint64_t>(std::max<uint64_t>(max_chunk, 1), (uint64_t)INT_MAX);
    uint64_t *nrp = nullptr, *deg = nullptr;
    uint32_t *tmp = nullptr, *nci = nullptr, *big = nullptr;
    unsigned long long *nbig = nullptr, repeated = 0;  // device: listed rows, and whether one repeats an id
    char *work = nullptr;
    void *scan = nullptr;
    size_t need = 0;
    uint64_t at = 0;
    const uint64_t big_min = n <= kBigVertices ? big_row(n) : ~0ull;
    cudaError_t e = cudaSuccess;
    auto ok = [&](cudaError_t r) {
        if (e == cudaSuccess) e = r;
        return e == cudaSuccess;
    };
    auto place = [&](uint64_t bytes) {  // offset of the next workspace array
        const uint64_t o = at;
        at += (bytes + 255) & ~255ull;
        return o;
    };
    const int G = sms * 8;
    const uint64_t o_deg = place(8 * (n + 1)), o_tmp = place(4 * std::max<uint64_t>(m, 1)), o_nbig = place(16);
    // a listed row has at least big_min of the m entries
    const uint64_t o_big = place(4 * (m / big_min + 1));
    if (!ok(cub::DeviceScan::ExclusiveSum(nullptr, need, deg, nrp, (int)(n + 1)))) return e;
    const uint64_t o_scan = place(std::max<size_t>(need, 16));
    if (!ok(cudaMalloc(&nrp, 8 * (n + 1))) || !ok(cudaMalloc(&nci, 4 * std::max<uint64_t>(m, 1))) ||
        !ok(cudaMalloc(&work, at)))
        goto done;
    deg = reinterpret_cast<uint64_t *>(work + o_deg);
    tmp = reinterpret_cast<uint32_t *>(work + o_tmp);
    nbig = reinterpret_cast<unsigned long long *>(work + o_nbig);
    big = reinterpret_cast<uint32_t *>(work + o_big);
    scan = work + o_scan;
    if (!ok(cudaMemsetAsync(deg + n, 0, 8)) || !ok(cudaMemsetAsync(nbig, 0, 16))) goto done;
    recode_degrees_kernel<<<G, 256>>>(rp, perm, n, deg);
    // exclusive scan: row pointers of the renamed rows (entry n = m)
    if (!ok(cub::DeviceScan::ExclusiveSum(scan, need, deg, nrp, (int)(n + 1)))) goto done;
    recode_scatter_kernel<<<G, 256>>>(rp, ci, perm, nrp, n, big_min, big, nbig, tmp);
    if (!ok(cudaGetLastError())) goto done;
    if (big_min != ~0ull && m >= big_min) {
        const size_t sm = 4ull * std::min<uint64_t>((n + 31) / 32, kSpanWords);
        if (!ok(cudaFuncSetAttribute(recode_big_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     4 * (int)kSpanWords)))
            goto done;
        recode_big_rows_kernel<<<sms, 1024, sm>>>(rp, ci, perm, nrp, n, big, nbig, nbig + 1, nci);
        if (!ok(cudaGetLastError())) goto done;
    }
    // sort the other rows, in calls of at most max_chunk entries
    if (!ok(sort_rows_device(nrp, n, m, tmp, nci, max_chunk, sms, big_min))) goto done;
    if (big_min != ~0ull && m >= big_min && ok(cudaMemcpy(&repeated, nbig + 1, 8, cudaMemcpyDeviceToHost)) && repeated) {
        recode_scatter_kernel<<<G, 256>>>(rp, ci, perm, nrp, n, ~0ull, big, nbig, tmp);
        if (ok(cudaGetLastError())) ok(sort_rows_device(nrp, n, m, tmp, nci, max_chunk, sms));
    }
done:
    cudaFree(work);
    if (e != cudaSuccess) {
        cudaFree(nrp);
        cudaFree(nci);
        return e;
    }
    *new_rp = nrp;
    *new_ci = nci;
    return cudaSuccess;
}

// perm (new id of each vertex) and core numbers of the CSR (rp, ci) with n
// vertices; device buffers.  *launches = kernels launched.  Synchronous (the
// sort's bit count is read back).  cudaErrorTimeout: the peel's barrier gave up
// (after kPeelWait, or G2_PEEL_WAIT SM cycles where that is set).
cudaError_t degeneracy_order_device(const uint64_t *rp, const uint32_t *ci, uint64_t n, uint64_t m, uint32_t *perm,
                                    uint32_t *core, int sms, uint64_t *launches) {
    *launches = 0;
    if (n == 0) return cudaSuccess;
    cudaError_t e = cudaSuccess;
    auto ok = [&](cudaError_t r) {
        if (e == cudaSuccess) e = r;
        return e == cudaSuccess;
    };
    const int G = sms * 8;
    unsigned blocks = (unsigned)sms;
    if (const char *env = getenv("G2_PEEL_BLOCKS")) blocks = std::max(1u, std::min(blocks, (unsigned)strtoul(env, nullptr, 10)));
    uint64_t share = 0;
    uint64_t at = 0;
    auto place = [&](uint64_t bytes) {
        const uint64_t o = at;
        at += (bytes + 255) & ~255ull;
        return o;
    };
    // peel: degrees, the warps' lists, two shared lists of pieces (each vertex is
    // listed once at most); sort: keys and ids twice
    uint64_t shared_cap = n + m / kPiece;
    const uint64_t o_ctl = place(sizeof(PeelCtl)), o_deg = place(4 * n), o_list = place(4 * (n + 32ull * kPeelWarps * blocks + 64)),
                   o_shared = place(16 * shared_cap), o_keys = place(16 * n), o_ids = place(8 * n);
    size_t need64 = 0, need32 = 0;
    {
        cub::DoubleBuffer<unsigned long long> k64(nullptr, nullptr);
        cub::DoubleBuffer<uint32_t> k32(nullptr, nullptr), v(nullptr, nullptr);
        if (!ok(cub::DeviceRadixSort::SortPairs(nullptr, need64, k64, v, (int)n)) ||
            !ok(cub::DeviceRadixSort::SortPairs(nullptr, need32, k32, v, (int)n)))
            return e;
    }
    size_t need = std::max<size_t>(std::max(need64, need32), 16);
    const uint64_t o_tmp = place(need);
    char *work = nullptr;
    if (!ok(cudaMalloc(&work, at))) return e;
    PeelCtl *ctl = reinterpret_cast<PeelCtl *>(work + o_ctl);
    uint32_t *deg = reinterpret_cast<uint32_t *>(work + o_deg), *list = reinterpret_cast<uint32_t *>(work + o_list),
             *ids = reinterpret_cast<uint32_t *>(work + o_ids);
    uint64_t *shared_list = reinterpret_cast<uint64_t *>(work + o_shared);
    PeelCtl h{};
    int dbits = 0, bits = 0;
    long long wait_cycles = kPeelWait;
    if (const char *env = getenv("G2_PEEL_WAIT")) wait_cycles = strtoll(env, nullptr, 10);
    void *args[] = {&rp, &ci, &n, &deg, &core, &list, &share, &shared_list, &shared_cap, &ctl, &wait_cycles};
    if (!ok(cudaMemsetAsync(ctl, 0, sizeof(PeelCtl)))) goto done;
    // one CTA per SM, or as many as this context may keep resident (part of a GPU)
    for (;; blocks = (blocks + 1) / 2) {
        const uint64_t nw = (uint64_t)blocks * kPeelWarps;
        share = ((n + 31) / 32 + nw - 1) / nw * 32;
        const cudaError_t r = cudaLaunchCooperativeKernel((const void *)peel_kernel, dim3(blocks), dim3(kPeelThreads), args, 0, nullptr);
        if (r == cudaErrorCooperativeLaunchTooLarge && blocks > 1) {
            cudaGetLastError();
            continue;
        }
        if (!ok(r)) goto done;
        break;
    }
    if (!ok(cudaMemcpy(&h, ctl, sizeof(h), cudaMemcpyDeviceToHost)))
        goto done;
    if (h.timeout) {
        e = cudaErrorTimeout;
        goto done;
    }
    // order by (core, degree, id): a stable sort of the bits that are in use
    while (dbits < 32 && (h.max_deg >> dbits)) dbits++;
    bits = dbits;
    while (bits < dbits + 32 && ((unsigned long long)h.max_core >> (bits - dbits))) bits++;
    {
        cub::DoubleBuffer<uint32_t> v(ids, ids + n);
        if (bits <= 32) {
            uint32_t *keys = reinterpret_cast<uint32_t *>(work + o_keys);
            order_keys_kernel<<<G, 256>>>(rp, core, n, dbits, keys, ids);
            cub::DoubleBuffer<uint32_t> kb(keys, keys + n);
            if (!ok(cub::DeviceRadixSort::SortPairs(work + o_tmp, need, kb, v, (int)n, 0, std::max(bits, 1)))) goto done;
        } else {
            unsigned long long *keys = reinterpret_cast<unsigned long long *>(work + o_keys);
            order_keys_kernel<<<G, 256>>>(rp, core, n, dbits, keys, ids);
            cub::DoubleBuffer<unsigned long long> kb(keys, keys + n);
            if (!ok(cub::DeviceRadixSort::SortPairs(work + o_tmp, need, kb, v, (int)n, 0, bits))) goto done;
        }
        scatter_perm_kernel<<<G, 256>>>(v.Current(), n, perm);
    }
    *launches = 3 + 2 + (uint64_t)(bits + 7) / 8;
    ok(cudaGetLastError());
    ok(cudaDeviceSynchronize());
done:
    cudaFree(work);
    return e;
}

}  // namespace g2
