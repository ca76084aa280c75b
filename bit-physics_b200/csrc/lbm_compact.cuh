// lbm_compact.cuh -- ordered lists of the items a predicate picks.
//
// The per-lattice lists (special cells of the adjoint, rule quads, face
// items) are wanted in lattice order: neighbouring list entries then step
// neighbouring cells, whose gathers share cache lines.  Counted per block,
// scanned, then written at each item's rank, so the order comes out of the
// listing itself and nothing goes to the host but the counts.  (Atomics and a
// host sort in its place: the 65,000 special cells of a 128^3 channel took
// a copy each way and a sort of some milliseconds for every tape.)
#pragma once

#include <cuda_runtime.h>

namespace lbm {

constexpr int COMPACT_THREADS = 256, COMPACT_ROUNDS = 4, COMPACT_ITEMS = COMPACT_THREADS * COMPACT_ROUNDS;

inline int compact_blocks(int items) { return (items + COMPACT_ITEMS - 1) / COMPACT_ITEMS; }
// Scratch ints of a listing of `items` items into `kinds` lists.
inline size_t compact_scratch(int items, int kinds) { return (size_t)kinds * compact_blocks(items); }

// Block b's number of items of each kind: counts[k * gridDim.x + b].  KIND(i)
// is the list of item i, or a negative number.
template <int KINDS, class KIND>
__global__ void __launch_bounds__(COMPACT_THREADS) k_compact_count(KIND kind, int items, int* __restrict__ counts)
{
    int mine[KINDS] = {};
    for (int r = 0; r < COMPACT_ROUNDS; ++r) {
        const int i = blockIdx.x * COMPACT_ITEMS + r * COMPACT_THREADS + threadIdx.x;
        const int k = i < items ? kind(i) : -1;
#pragma unroll
        for (int q = 0; q < KINDS; ++q) mine[q] += __syncthreads_count(k == q);
    }
    if (threadIdx.x == 0)
#pragma unroll
        for (int q = 0; q < KINDS; ++q) counts[q * gridDim.x + blockIdx.x] = mine[q];
}

// Exclusive scan of each kind's block counts in place; totals[k] its sum.
// One block of 1024 threads.
template <int KINDS>
__global__ void __launch_bounds__(1024) k_compact_scan(int* __restrict__ counts, int nblocks, int* __restrict__ totals)
{
    __shared__ int warp_sum[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int q = 0; q < KINDS; ++q) {
        int* c = counts + (size_t)q * nblocks;
        int carry = 0;
        for (int b0 = 0; b0 < nblocks; b0 += 1024) {
            const int b = b0 + (int)threadIdx.x;
            const int v = b < nblocks ? c[b] : 0;
            int s = v;
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, s, o);
                if (lane >= o) s += t;
            }
            if (lane == 31) warp_sum[warp] = s;
            __syncthreads();
            int before = 0, all = 0;
            for (int w = 0; w < 32; ++w) {
                if (w < warp) before += warp_sum[w];
                all += warp_sum[w];
            }
            if (b < nblocks) c[b] = carry + before + s - v;
            carry += all;
            __syncthreads();  // warp_sum is reused
        }
        if (threadIdx.x == 0) totals[q] = carry;
    }
}

// Item i of kind k goes to lists[k * cap + its rank among the kind's items].
template <int KINDS, class KIND>
__global__ void __launch_bounds__(COMPACT_THREADS)
    k_compact_write(KIND kind, int items, const int* __restrict__ starts, int* __restrict__ lists, size_t cap)
{
    __shared__ int warp_count[KINDS][COMPACT_THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int base[KINDS];
#pragma unroll
    for (int q = 0; q < KINDS; ++q) base[q] = starts[q * gridDim.x + blockIdx.x];
    for (int r = 0; r < COMPACT_ROUNDS; ++r) {
        const int i = blockIdx.x * COMPACT_ITEMS + r * COMPACT_THREADS + threadIdx.x;
        const int k = i < items ? kind(i) : -1;
        unsigned own[KINDS];
#pragma unroll
        for (int q = 0; q < KINDS; ++q) {
            own[q] = __ballot_sync(0xffffffffu, k == q);
            if (lane == 0) warp_count[q][warp] = __popc(own[q]);
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < KINDS; ++q) {
            int before = 0, all = 0;
            for (int w = 0; w < COMPACT_THREADS / 32; ++w) {
                if (w < warp) before += warp_count[q][w];
                all += warp_count[q][w];
            }
            if (k == q) lists[q * cap + base[q] + before + __popc(own[q] & ((1u << lane) - 1u))] = i;
            base[q] += all;
        }
        __syncthreads();  // warp_count is reused
    }
}

// The items 0 .. items - 1 by kind, each list in increasing order, their
// numbers in totals[KINDS] (device).  scratch: compact_scratch() ints.
template <int KINDS, class KIND>
inline cudaError_t compact(KIND kind, int items, int* lists, size_t cap, int* totals, int* scratch, cudaStream_t s)
{
    const int blocks = compact_blocks(items);
    k_compact_count<KINDS><<<blocks, COMPACT_THREADS, 0, s>>>(kind, items, scratch);
    k_compact_scan<KINDS><<<1, 1024, 0, s>>>(scratch, blocks, totals);
    k_compact_write<KINDS><<<blocks, COMPACT_THREADS, 0, s>>>(kind, items, scratch, lists, cap);
    return cudaGetLastError();
}

}  // namespace lbm
