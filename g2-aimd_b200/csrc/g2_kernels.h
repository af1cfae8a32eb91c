// g2_kernels.h - argument blocks and launchers of the device kernels
// (internal to libg2aimd.so; the public surface is include/g2_aimd.h).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "g2_aimd.h"

namespace g2 {

// Bits of the device status word.
constexpr int kStatusDeferOverflow = 1;  // deferred-task list full
constexpr int kStatusHistOverflow = 2;   // clique larger than the histogram
constexpr int kStatusStackOverflow = 4;  // GMatch candidate stack exhausted
constexpr int kStatusBadPlan = 8;        // plan arrays inconsistent
constexpr int kStatusWaitLimit = 16;     // a bounded device wait ran out
constexpr int kStatusDeadline = 32;      // the run's time budget ran out (MCE)

constexpr int kStatusRest = 64;          // (no error) a clique run's rest list has entries

// An MCE pass entry with this bit set is a spilled record id, else a task id.
constexpr uint32_t kRecordBit = 0x80000000u;
// Depth word of a record slot whose reservation ran past the buffer's end.
constexpr uint32_t kVoidRecord = 0xffffffffu;

// The dynamic shared memory limit set on the kernels (not the size of a launch): the
// same value every time, so that contexts of several threads do not take it from one
// another between setting it and launching.
constexpr int kMaxDynamicSmem = 200 * 1024;

// Bit rows of the last ids of a graph (g2_corebits.cuh): row of vertex u in
// [base, end) = bits of N+(u) over the ids base, base + 1, ..., `stride` words
// (a multiple of 4) each, from word `off` of the matrix.  A batch of graphs has
// one block per graph; row0 = rows of the blocks before it.
struct CoreBlock {
    uint32_t base, end, stride, row0;
    uint64_t off;
};
struct CoreBits {
    const uint32_t *bits;
    const CoreBlock *blocks;  // device; used if nblocks > 1
    uint32_t nblocks, rows;   // rows = sum of the blocks' rows
    CoreBlock one;            // the block if there is only one
};
// Block geometry of a graph of n vertices and m entries whose ids [lo, lo + n)
// get bit rows on the last K, K^2 bits at most about `bytes` (K a multiple of 128
// unless K = n); row0 / off continue from the previous block.
CoreBlock core_block_of(uint32_t lo, uint32_t n, uint64_t bytes, uint32_t row0, uint64_t off);

struct MceArgs {
    static constexpr uint32_t kPollCycles = 6000, kMaxSleepNs = 4096;  // of waiting warps (g2_handoff.cuh)
    const uint64_t *rp;
    const uint32_t *ci;
    const uint32_t *fo;             // fo[v]: offset in N(v) of the first neighbour > v
    const uint32_t *tasks;          // root vertex of each task
    const uint32_t *task_index;     // optional: the task ids this pass runs (else 0..ntasks-1)
    const uint32_t *task_part;      // optional per task id: (nparts << 16) | part of a split root
    uint32_t split_depth;           // split roots deal out their depth-split_depth subtrees (>= 1)
    uint64_t *root_cost;            // optional per task id: SM cycles spent on the task
    uint64_t ntasks;                // tasks in this pass (if ntasks_dev is null)
    const unsigned long long *ntasks_dev;  // else: task count read from device memory
    unsigned long long *head;       // device queue head
    uint32_t chunk;                 // tasks grabbed per atomic (0: 1, more among the light tasks)
    uint32_t hist_len;
    uint32_t *scratch;              // warps * words_per_warp words
    uint64_t words_per_warp;        // multiple of 64
    unsigned long long *out;        // [0] count, [1 + s] hist[s]
    uint32_t *deferred;             // task ids deferred to a larger pass
    unsigned long long *ndeferred;
    uint64_t deferred_cap;
    uint64_t *root_nodes;           // optional, per task id
    uint64_t *root_cliques;         // optional: maximal cliques found per task id
    unsigned long long *hist_dev;   // optional: per-root histogram here (a one-warp pass
                                    // whose slab is the spill slab) instead of the slab's head
    unsigned long long *work;       // optional: work model W in bytes (metrics kernel)
    int *status;
    // handed-off search-tree nodes (record: task, depth, pool offset / 64, nb,
    // then P, X, R rows of rec_words words; rec_stride words each)
    uint32_t *records;
    uint32_t *ready;                // per record slot: epoch of the run that published it
    unsigned long long *nrec;       // records written in this run (append-only)
    uint64_t rec_cap;
    uint32_t rec_stride, rec_words;
    uint32_t *pool;                 // A and B rows of the roots whose tasks spilled
    unsigned long long *npool;      // 64-word units used
    uint64_t pool_cap;              // words
    uint64_t spill_cycles;          // 0: no hand-off in this pass
    unsigned long long *qctl;       // record queue: [kQHead] tickets taken, [kQOut] outstanding work
    uint32_t epoch;                 // ready word of records published in this run (read from epoch_dev)
    const uint32_t *epoch_dev;      // the run's epoch, bumped on the device at the run's start
    uint64_t wait_cycles;           // longest wait of a warp for its ticket's record
    const unsigned long long *deadline;  // optional: %globaltimer (ns) past which roots are
                                         // dropped (set on the device by deadline_set)
    CoreBits core;                  // bit rows (core.bits null: every root takes the general walk)
    uint32_t sorted;                // tasks in descending cost (chunk 0)
    uint32_t hist_fold;             // inner nodes after which a warp empties its 32-bit size counters (a power of two)
};
constexpr int kQHead = 0, kQOut = 1;
constexpr uint32_t kMatchRecordWords = 32;  // stride of a plan-walk record

size_t mce_smem_bytes(int wpl, int warps_per_block);
// Resident CTAs per SM of the kernel a launch with these parameters runs (0 on error).
int mce_blocks_per_sm(int wpl, int warps_per_block, bool metrics);
int match_blocks_per_sm(int wpl, int warps_per_block, bool metrics, int ctas_per_sm, uint32_t p0_words);
// Load the code of a budgeted launch (kernels load on their first use, which takes
// milliseconds that would count against the budget).
cudaError_t mce_preload(int wpl);
cudaError_t clique_preload(uint32_t k, bool in_order);
cudaError_t mce_launch(int wpl, const MceArgs &a, int blocks, int warps_per_block, cudaStream_t st);
// Advance a run's hand-off epoch in stream order (skipping 0, the value of a
// never-published ready word), so runs captured in a CUDA graph stay distinct
// when the graph is replayed.
cudaError_t epoch_bump(uint32_t *epoch_dev, cudaStream_t st);
// *deadline = the device's %globaltimer now + budget_ns, in stream order.
cudaError_t deadline_set(unsigned long long *deadline, unsigned long long budget_ns, cudaStream_t st);
// In stream order: kStatusDeferOverflow into *status if *left (entries no pass
// walked) is nonzero.
cudaError_t flag_left(const unsigned long long *left, int *status, cudaStream_t st);

// Plan in device-friendly form: everything by POSITION.
struct DevPlan {
    uint32_t k;
    uint32_t bn_count[G2_MAX_QUERY];
    uint32_t bn_pos[G2_MAX_QUERY][G2_MAX_QUERY];       // back neighbours as positions
    uint32_t cond_count[G2_MAX_QUERY];
    uint32_t cond_op[G2_MAX_QUERY][G2_MAX_QUERY];      // condition of position p vs ...
    uint32_t cond_pos[G2_MAX_QUERY][G2_MAX_QUERY];     // ... the vertex matched at this position
    uint32_t share[G2_MAX_QUERY];                      // prefix intersection computed one level early
    uint32_t pre_bn_count[G2_MAX_QUERY];
    uint32_t pre_bn_pos[G2_MAX_QUERY][G2_MAX_QUERY];
    uint32_t pre_cond_count[G2_MAX_QUERY];
    uint32_t pre_cond_op[G2_MAX_QUERY][G2_MAX_QUERY];
    uint32_t pre_cond_pos[G2_MAX_QUERY][G2_MAX_QUERY];
    uint32_t after_bn_count[G2_MAX_QUERY];
    uint32_t after_bn_pos[G2_MAX_QUERY][G2_MAX_QUERY];
    uint32_t after_cond_count[G2_MAX_QUERY];
    uint32_t after_cond_op[G2_MAX_QUERY][G2_MAX_QUERY];
    uint32_t after_cond_pos[G2_MAX_QUERY][G2_MAX_QUERY];
    uint32_t clique;        // 1: every position adjacent to all earlier ones, strictly increasing images
};

struct MatchArgs {
    static constexpr uint32_t kPollCycles = 24000, kMaxSleepNs = 16384;  // of waiting warps (g2_handoff.cuh)
    const uint64_t *rp;
    const uint32_t *ci;
    const uint32_t *fo;
    const uint32_t *tasks;
    const uint32_t *task_index;
    const uint32_t *task_part;      // optional per task: (nparts << 16) | part of a split root
    uint64_t *root_cost;            // optional per task: SM cycles spent on the task
    uint64_t ntasks;
    const unsigned long long *ntasks_dev;  // optional: task count read from device memory
    unsigned long long *head;
    uint32_t chunk;
    uint32_t *scratch;
    uint64_t words_per_warp;
    unsigned long long *out;        // [0] count
    unsigned long long *work;       // optional: work model W in bytes (metrics kernel)
    uint32_t *deferred;
    unsigned long long *ndeferred;
    uint64_t deferred_cap;
    uint64_t *root_nodes;           // optional: embeddings counted per task
    int *status;
    // hand-off of pending plan-walk work to idle warps (g2_handoff.cuh); record:
    // [task, level, kind, ncand, M[0..7], window pos (2), end (2), candidates (16)]
    uint32_t *records;
    uint32_t *ready;
    unsigned long long *nrec;
    uint64_t rec_cap;
    uint32_t rec_stride;
    unsigned long long *qctl;
    uint32_t epoch;                 // ready word of records published in this run (read from epoch_dev)
    const uint32_t *epoch_dev;      // the run's epoch, bumped on the device at the run's start
    uint64_t wait_cycles;
    uint64_t spill_cycles;          // 0: no hand-off
    uint32_t p0_words;              // shared words per warp for P0 (see match_p0_words)
    const unsigned long long *deadline;  // optional: %globaltimer (ns) past which roots are dropped
};

// Shared-memory words per warp the clique path needs besides its row buffer:
// P0 staged for the symmetric-row walk (k > 5 or the metrics build), or the
// P0 filter and hit queue of the lane-parallel counting (k <= 5); none for
// plan walks (non-clique plans).
uint32_t match_p0_words(int wpl, bool clique_path, uint32_t k, bool metrics);
size_t match_smem_bytes(int wpl, int warps_per_block, uint32_t p0_words);
cudaError_t match_launch(const DevPlan &plan, const MatchArgs &a, int blocks, int warps_per_block,
                         cudaStream_t st, bool clique_path, int wpl, int ctas_per_sm);

// Counting of 3-, 4- and 5-cliques on core bit rows (clique.cu).
struct CliqueArgs {
    const uint64_t *rp;
    const uint32_t *ci;
    const uint32_t *fo;
    const uint32_t *tasks;
    const uint32_t *task_part;      // optional per task: (nparts << 16) | part of a split root
    uint64_t ntasks;
    const unsigned long long *ntasks_dev;  // optional: task count read from device memory
    CoreBits core;
    uint32_t *bits_out;             // the matrix, written by the preparation kernel
    uint32_t in_order;              // one list in task order (else lists by root size)
    uint32_t cta_min;               // lists by size: roots with larger |P0| are shared by a CTA
    uint32_t p_fit;                 // roots with larger |P0| go to the rest list
    uint32_t by_cost;               // so do those whose forward lists are cheaper than their tiles
    uint32_t *lists;                // four lists of list_cap task ids: by size (or [0] in order), [3] rest
    uint32_t *pieces;               // 5-cliques, lists by size: (pieces << 16) | piece of list 0's entries
    uint64_t list_cap, extra_cap;   // list_cap >= ntasks + extra_cap; extra_cap = pieces beyond one per root
    unsigned long long *counts;     // list lengths; [4] extra pieces, [5] roots whose lists are cheaper (about)
    unsigned long long *heads;      // list heads
    uint32_t chunk;                 // in-order runs: tasks per queue atomic
    uint32_t *scratch;              // per-warp slabs
    uint64_t words_per_warp;
    uint32_t smem_words;            // dynamic shared memory of a CTA
    uint32_t q_words;               // words of a candidate-set row (5-cliques), else 0
    unsigned long long *out;
    uint64_t *root_nodes;           // optional: embeddings counted per task
    uint64_t *root_cost;            // optional: SM cycles per task
    int *status;
    const unsigned long long *deadline;
};
// Largest |P0| that one warp walks in runs by size.
uint32_t clique_cta_min(uint32_t k);
// Largest |P0| a launch of this geometry counts itself.
uint32_t clique_p_fit(uint32_t k, bool in_order, uint64_t words_per_warp, int warps_per_block);
// Can a root's forward lists be cheaper than its tiles?  (whole: every id has a bit row)
bool clique_by_cost(uint32_t max_fwd, bool whole);
// Dynamic shared memory (words) for roots up to max_fwd, and a row's word count for 5-cliques.
uint32_t clique_smem_words(uint32_t k, bool in_order, uint32_t max_fwd, int warps_per_block, uint32_t *q_words);
int clique_blocks_per_sm(uint32_t k, bool in_order, int warps_per_block, uint32_t smem_words);
// The core's bit rows alone (core.bits), in stream order.
cudaError_t core_rows_launch(const CoreBits &core, uint32_t *bits, const uint64_t *rp, const uint32_t *ci,
                             const uint32_t *fo, int sms, cudaStream_t st);
// *count += roots of a graph that may be cheaper by their forward lists than by tiles
// over the block `core` (legacy stream).
cudaError_t sparse_roots_launch(const uint64_t *rp, const uint32_t *ci, const uint32_t *fo, uint64_t n,
                                const CoreBlock &core, int sms, unsigned int *count);
cudaError_t clique_prepare_launch(const CliqueArgs &a, uint32_t k, int sms, cudaStream_t st);
cudaError_t clique_launch(const CliqueArgs &a, uint32_t k, int blocks, int warps_per_block, cudaStream_t st);

// Sort each row of `in` (device CSR rows given by rp) into `out`, in calls of at
// most max_chunk entries (kcore.cu); synchronous.
cudaError_t sort_rows_device(const uint64_t *rp, uint64_t n, uint64_t m, const uint32_t *in, uint32_t *out,
                             uint64_t max_chunk, int sms, uint64_t big_min = ~0ull);
// Degeneracy order of a CSR on the device (kcore.cu); synchronous.
cudaError_t degeneracy_order_device(const uint64_t *rp, const uint32_t *ci, uint64_t n, uint64_t m, uint32_t *perm,
                                    uint32_t *core, int sms, uint64_t *launches);
// The CSR with vertex v renamed perm[v], rows sorted (kcore.cu); synchronous.
// new_rp (n+1) and new_ci (m) are allocated here (cudaMalloc); rows are sorted
// in calls of at most max_chunk entries (a row longer than that: NotSupported).
cudaError_t recode_device(const uint64_t *rp, const uint32_t *ci, uint64_t n, uint64_t m, const uint32_t *perm,
                          uint64_t max_chunk, int sms, uint64_t **new_rp, uint32_t **new_ci);

// Learned root-cost model (costmodel.cu).
size_t model_smem_bytes();
cudaError_t features_launch(const uint64_t *rp, const uint32_t *ci, const uint32_t *fo, const uint32_t *core,
                            const uint32_t *src, uint64_t n, float *out, int sms, cudaStream_t st);
cudaError_t train_step_launch(const float *X, const float *Y, const uint32_t *idx, uint32_t n, const float *params,
                              const float *norm, float *grad, float *loss, cudaStream_t st);
cudaError_t adam_launch(float *params, float *mom, float *vel, const float *grad, float lr, int step,
                        cudaStream_t st);
cudaError_t score_launch(const uint32_t *src, uint64_t n, const float *X, const float *params, const float *norm,
                         float *pred, float *cost, float *total, int sms, cudaStream_t st);

}  // namespace g2
