// pb_fold_leaf.cuh - the fused two-ply leaf on folded counting (pb_fold.cuh),
// leaf kernel 6 and the default leaf of every path without tables.
//
// Two kernels per chunk of edges: k_fold makes each edge's child, sums its
// simple moves (fold_child) and appends its other moves to a queue in device
// memory; k_fold_count makes the queued moves and counts each of them in full,
// one per thread.  Both are bound by integer issue.  The queue between them
// costs 16 B of traffic per queued move (0.7 per child on the benchmark's
// leaves, 3.6 on middle-game playouts) and buys full warps in both halves, no
// barriers, and 55 + 20 KB of code instead of one kernel whose warps fetch from
// both at once (one kernel with a shared-memory queue and a barrier between the
// halves: 10.9 ms against 8.15 ms for the first form of these two on the
// benchmark's leaves).
//
// Measured on B200 against the leaf that makes and counts every move
// (children balanced across warps, listed pieces; the benchmark's 27.2 M edges, 774 M moves):
// 20.09 -> 6.78 ms (k_fold 6.09, k_fold_count 0.69); 5.2 M edges of 6-40 ply
// playouts 5.33 -> 2.10 ms; 4.2 M edges of 60-140 ply playouts 4.26 -> 1.90 ms.
// The test for a side left in check and the defined square of a missing king
// cost 0.3 to 0.9 % of that.
#pragma once
#include "pb_fold.cuh"
#include "pb_kernels.cuh"

namespace pb {

// k_fold's CTA: 80 registers a thread, 24 warps per SM, with the values read
// seldom on a shelf in shared memory (120 B a thread).  On the benchmark's leaves
// 20 warps (96 registers) without the shelf ran 6.49 ms and with it 6.40, 24 warps
// with it 6.07, 32 warps (64 registers, spills) 6.47; without the shelf 24 and 32
// warps had lost to 20.  The code is long and straight, so warps that start
// together share its instruction fetches: at the same 24 warps CTAs of 256
// threads ran 9 % slower (barriers between the stages gained nothing more).
// Warps of a CTA in multiples of four, one for each scheduler: 22 warps in CTAs
// of 11 ran 6.73 ms.  Small launches use 64 threads so that they reach every SM.
constexpr int FOLD_THREADS = 384;
constexpr int FOLD_SMALL_THREADS = 64;
constexpr int FOLD_THREADS_PER_SM = 768;
// Staged moves per thread of a warp: with the shelf a CTA's 64.6 KB fill the 132 KB
// shared-memory split twice.  9 lose 5 to 17 % on playouts (the queue's atomics),
// 16 take 32 KB from the L1 cache and lose 1.5 % on the benchmark's leaves.
constexpr int FOLD_STAGE = 12;
constexpr int FOLD_SHELF_BYTES = SHELF_SLOTS * 8;  // dynamic shared memory per thread

enum : u32 { DEVERR_QUEUE = 8u };  // a queue was too short for its chunk: the leaf runs again

// The edges of a leaf.  With n_dev the sizes are in device memory (captured
// graphs): n and nparents are then the planned capacities.
struct LeafEdges {
    const Board *boards;  // positions the edges leave from
    const uint8_t *states;
    const u32 *root;  // root index of each position (rooted leaves)
    const u32 *pidx;
    const uint16_t *moves;
    u64 n, nparents;
    const u64 *n_dev, *nparents_dev;
    // FOLD_EACH: the edges to count (the table leaf's misses) and how many, the
    // count of each edge
    const u32 *list;
    const unsigned long long *list_len;
    u32 *each;
};

// Where the counts go: one sum, each root's counter, each listed edge's word.
enum FoldOut { FOLD_SUM, FOLD_ROOTED, FOLD_EACH };

// Queued moves of one chunk: edge << 16 | move.
struct FoldQueue {
    u64 *items;
    unsigned long long *cursor;
    u64 cap;
};

// A warp's sink: moves are staged in shared memory (lane << 16 | move) and
// flushed to the queue when the warp is done, so its queue entries are
// contiguous and take one atomic.  A set that does not fit the stage takes
// queue slots at once; every later set then does not fit either (the stage's
// cursor only grows), so the stage holds the entries below the smallest cursor
// of a set that did not fit, without holes.
struct StagedSink {
    u32 *stage;
    u32 *used;  // [0] slots taken, [1] the stage's length
    u32 lane_tag;
    u64 edge;
    FoldQueue q;
    static constexpr u32 CAP = FOLD_STAGE * 32;
    __device__ __forceinline__ void set(int from, u64 t)
    {
        if (!t) return;
        const u32 n = (u32)popc(t);
        u32 slot = atomicAdd(used, n);
        if (slot + n <= CAP) {
            const u32 w = lane_tag | (u32)from;
            for (; t; t &= t - 1) stage[slot++] = w | ((u32)lsb(t) << 6);
        } else {
            if (slot < CAP) atomicMin(used + 1, slot);
            u64 g = atomicAdd(q.cursor, (unsigned long long)n);
            for (; t; t &= t - 1, g++)
                if (g < q.cap) q.items[g] = (edge << 16) | (u32)from | ((u32)lsb(t) << 6);
        }
    }
    __device__ __forceinline__ void one(uint16_t m, bool promotes)
    {
        const u32 n = promotes ? 4 : 1;
        u32 w = m | (promotes ? (u32)MF_PROMO << 12 : 0u);
        const u32 slot = atomicAdd(used, n);
        if (slot + n <= CAP) {
            w |= lane_tag;
            stage[slot] = w;
            if (promotes)
                for (u32 k = 1; k < 4; k++) stage[slot + k] = w + (k << 12);
        } else {
            if (slot < CAP) atomicMin(used + 1, slot);
            const u64 g = atomicAdd(q.cursor, (unsigned long long)n);
            for (u32 k = 0; k < n; k++)
                if (g + k < q.cap) q.items[g + k] = (edge << 16) | (w + (k << 12));
        }
    }
};

// Edges [first, first + count) of the leaf, cut to its size.  counter[0] +=
// counts of the simple moves (or as OUT says), counter[1] += their number.
template <int C, bool STRICT, int T, FoldOut OUT>
__global__ void __launch_bounds__(T, FOLD_THREADS_PER_SM / T)
    k_fold(const __grid_constant__ LeafEdges e, u64 first, u64 count, const __grid_constant__ FoldQueue queue,
           unsigned long long *__restrict__ root_counts, unsigned long long *__restrict__ counter,
           u32 *__restrict__ err)
{
    constexpr int W = T / 32;
    __shared__ u32 s_stage[W][FOLD_STAGE * 32];
    __shared__ u32 s_used[W][2];
    extern __shared__ u64 s_shelf[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    u64 n = e.n, nparents = e.nparents;
    if (e.n_dev) {
        if (plan_overflowed(err)) return;
        n = dev_size(e.n_dev, n, err);
        nparents = min(*e.nparents_dev, nparents);
    }
    n = OUT == FOLD_EACH ? (u64)*e.list_len : min(n, first + count);
    const u64 at = first + (u64)blockIdx.x * T + threadIdx.x;
    if (at - lane >= n) return;
    if (lane == 0) s_used[warp][0] = 0, s_used[warp][1] = FOLD_STAGE * 32;
    __syncwarp();
    u32 total = 0, simple = 0, root = 0;
    const u64 i = OUT == FOLD_EACH && at < n ? e.list[at] : at;
    const u32 p = at < n ? e.pidx[i] : 0xFFFFFFFFu;
    const bool valid = at < n && p < nparents;
    if (valid) {
        if (OUT == FOLD_ROOTED) root = e.root[p];
        Board b = load_board(e.boards + p);
        u32 st = e.states[p];
        make_move<C>(b, st, e.moves[i]);
        StagedSink sink{s_stage[warp], s_used[warp], (u32)lane << 16, i, queue};
        total = fold_child<1 - C, STRICT>(b, st, sink, &simple, Shelf{s_shelf + threadIdx.x, T});
    }
    __syncwarp();
    const u32 used = min(s_used[warp][0], s_used[warp][1]);
    u64 base = 0;
    if (lane == 0 && used) base = atomicAdd(queue.cursor, (unsigned long long)used);
    base = __shfl_sync(0xffffffffu, base, 0);
    for (u32 k = lane; k < used; k += 32) {
        const u32 w = s_stage[warp][k];
        const u64 from = at - lane + (w >> 16);
        if (base + k < queue.cap)
            queue.items[base + k] = ((OUT == FOLD_EACH ? (u64)e.list[from] : from) << 16) | (w & 0xFFFFu);
    }
    if (OUT == FOLD_ROOTED) add_by_key(root_counts, root, total, valid);
    if (OUT == FOLD_EACH && at < n) e.each[i] = total;
    if (OUT == FOLD_SUM) total = __reduce_add_sync(0xffffffffu, total);
    simple = __reduce_add_sync(0xffffffffu, simple);
    if (lane == 0 && simple) {
        if (OUT == FOLD_SUM) atomicAdd(counter, (unsigned long long)total);
        atomicAdd(counter + 1, (unsigned long long)simple);
    }
}

// Counts the queued moves (the grid strides over them; their number is on the
// device).  A queue that was too short sets `overflow` in the error word.  Bound
// by integer issue behind the table loads: 40 warps per SM (48 registers, a few
// spills) against 32, and 64 CTAs per SM that come and go against 4 that stay,
// took 24.2 M moves of middle-game playouts from 0.99 to 0.85 ms.
template <int C, bool STRICT, FoldOut OUT>
__global__ void __launch_bounds__(256, 5)
    k_fold_count(const __grid_constant__ LeafEdges e, const __grid_constant__ FoldQueue queue,
                 unsigned long long *__restrict__ root_counts, unsigned long long *__restrict__ counter,
                 u32 overflow, u32 *__restrict__ err)
{
    const u64 len = *queue.cursor;
    if (len > queue.cap) {
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(err, overflow);
        return;
    }
    u64 total = 0;
    const u64 stride = (u64)gridDim.x * 256;
    for (u64 k0 = (u64)blockIdx.x * 256 + (threadIdx.x & ~31u); k0 < len; k0 += stride) {
        const u64 k = k0 + (threadIdx.x & 31);
        u32 c = 0, root = 0;
        const bool valid = k < len;
        if (valid) {
            const u64 w = queue.items[k], i = w >> 16;
            const u32 p = e.pidx[i];
            if (OUT == FOLD_ROOTED) root = e.root[p];
            Board b = load_board(e.boards + p);
            u32 st = e.states[p];
            make_move<C>(b, st, e.moves[i]);
            make_move<1 - C>(b, st, (uint16_t)w);
            c = count_moves<C, STRICT>(b, st);
            if (OUT == FOLD_EACH) atomicAdd(e.each + i, c);
        }
        if (OUT == FOLD_ROOTED) add_by_key(root_counts, root, c, valid);
        if (OUT == FOLD_SUM) total += c;
    }
    if (OUT == FOLD_SUM) {
#pragma unroll
        for (int o = 16; o; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
        if ((threadIdx.x & 31) == 0 && total) atomicAdd(counter, (unsigned long long)total);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0 && len) atomicAdd(counter + 1, (unsigned long long)len);
}

}  // namespace pb
