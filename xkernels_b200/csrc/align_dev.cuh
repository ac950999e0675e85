// The single-CTA form of the routing sort as a device function (align.cu has the contract), for the kernels
// that start with it: align_small_kernel, and the activation gathers of decode batches.
#pragma once
#include "common.cuh"

namespace xkb {
namespace align {

constexpr int kThreads = 1024;
constexpr int kWarps = kThreads / 32;
constexpr int kChunk = kThreads;       // slots per round (one per thread)
constexpr int64_t kSmallMax = kChunk;  // single-CTA path up to this many slots
constexpr int kMaxExperts = 1024;

__device__ __forceinline__ int map_expert(int id, int E, const int32_t* expert_map, int num_map) {
  if (expert_map != nullptr) {
    if (id < 0 || id >= num_map) return E;
    id = expert_map[id];
  }
  return (id < 0 || id >= E) ? E : id;  // E = ghost expert (dropped)
}

// Exclusive scan of padded per-expert counts; one CTA, any E <= kMaxExperts.
// hist[e] (e < E) -> off[e], off[E] = total.  scratch: kWarps ints.
__device__ inline void padded_offsets(const int* hist, int* off, int* warp_tot, int E, int block) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // E <= 1024 = kThreads: one expert per thread.
  int padded = 0;
  if (tid < E) padded = (hist[tid] + block - 1) / block * block;
  int incl = padded;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    int v = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += v;
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int t = warp_tot[lane];
    int ti = t;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      int v = __shfl_up_sync(0xffffffffu, ti, d);
      if (lane >= d) ti += v;
    }
    warp_tot[lane] = ti - t;  // exclusive
  }
  __syncthreads();
  const int excl = incl - padded + warp_tot[warp];
  if (tid < E) off[tid] = excl;
  if (tid == E - 1) off[E] = excl + padded;
  if (E == 0 && tid == 0) off[0] = 0;
  __syncthreads();
}

// expert_ids[b] for every block b < max_blocks: the expert whose padded run
// holds position b*block, 0 past the used blocks.  block_live (may be nullptr): the block's slots that are not padding.
__device__ inline void write_expert_ids(const int* off, const int* count, int E, int block, int32_t* expert_ids,
                                 int32_t* block_live, int64_t max_blocks, int tid0, int stride) {
  const int total = off[E];
  for (int64_t b = tid0; b < max_blocks; b += stride) {
    const int64_t pos = b * block;
    int e = 0, live = 0;
    if (pos < total) {
      // largest e with off[e] <= pos and off[e+1] > pos (runs of zero length skipped)
      int lo = 0, hi = E;  // invariant: off[lo] <= pos < off[hi]
      while (hi - lo > 1) {
        int mid = (lo + hi) >> 1;
        if (off[mid] <= pos) lo = mid; else hi = mid;
      }
      e = lo;
      const int left = off[e] + count[e] - (int)pos;   // a run's padding is at its end
      live = left < block ? left : block;
    }
    expert_ids[b] = e;
    if (block_live != nullptr) block_live[b] = live;
  }
}

// Rank of this thread's slot among the slots of its expert in one 1024-slot round (0 if inactive), and the
// round's slots per expert in tot[0 .. E].  wcnt: [kWarps][E+1] uint16.
__device__ inline int round_rank(int my_e, bool active, int E, uint16_t* wcnt, int* tot) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int EP = E + 1;
  uint32_t* wcnt2 = reinterpret_cast<uint32_t*>(wcnt);
  for (int i = tid; i < kWarps * EP / 2; i += kThreads) wcnt2[i] = 0;   // kWarps is even
  __syncthreads();
  // inactive lanes vote with a key no expert uses so they never match
  const int key = active ? my_e : (EP + lane);
  const unsigned peers = __match_any_sync(0xffffffffu, key);
  const int rank = __popc(peers & ((1u << lane) - 1u));
  if (active && rank == 0) wcnt[warp * EP + my_e] = (uint16_t)__popc(peers);
  __syncthreads();
  // exclusive scan over warps, one expert per scanning warp per step
  for (int e = warp; e < EP; e += kWarps) {
    int v = wcnt[lane * EP + e];
    int incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      int u = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += u;
    }
    wcnt[lane * EP + e] = (uint16_t)(incl - v);
    if (lane == 31) tot[e] = incl;
  }
  __syncthreads();
  return active ? (int)wcnt[warp * EP + my_e] + rank : 0;
}

// What one sort reads and writes.  zero / zero_n: ints the caller wants cleared; expert_off and block_live may be nullptr.
struct Job {
  const int32_t* topk_ids;
  const int32_t* expert_map;
  int32_t* sorted_ids;
  int32_t* expert_ids;
  int32_t* num_post;
  int32_t* expert_off;
  int32_t* block_live;
  int32_t* zero;
  int64_t zero_n, numel, max_pad, max_blocks;
  int num_map, E, block;
};

// Sorted positions that a gather may go through, read after its wait (0 if the count is none the sort wrote: recorded).
constexpr int kErrGatherPositions = 3 + (3 << 8);   // kErrBadRouting, site 3
__device__ __forceinline__ int positions_to_gather(const int32_t* num_post, int64_t max_pad, int* status) {
  const int total = __ldcg(num_post);
  if (total >= 0 && total <= max_pad) return total;
  if (threadIdx.x == 0 && blockIdx.x == 0) atomicCAS(status, 0, kErrGatherPositions);
  return 0;
}

// shared memory of align_in_block; the first kThreads ints are free again when it returns
inline size_t small_smem(int E) {
  const size_t EP = E + 1;
  const size_t n = kWarps * EP * sizeof(uint16_t) + 2 * EP * sizeof(int) + kWarps * sizeof(int);
  return n < kThreads * sizeof(int) ? kThreads * sizeof(int) : n;
}

// The whole sort of numel <= 1024 slots by one block of 1024 threads; returns the position of slot
// threadIdx.x (-1: none or dropped).  write: also write the routing (one block of a grid does).
__device__ __forceinline__ int align_in_block(const Job& j, unsigned char* smem, bool write) {
  const int E = j.E, EP = E + 1, tid = threadIdx.x;
  uint16_t* wcnt = reinterpret_cast<uint16_t*>(smem);                             // [kWarps][EP]
  int* off = reinterpret_cast<int*>(smem + kWarps * EP * sizeof(uint16_t));       // [EP]   off[E] = total
  int* tot = off + EP;                                                            // [EP]
  int* warp_tot = tot + EP;                                                       // [kWarps]
  const bool active = tid < j.numel;
  const int e = active ? map_expert(j.topk_ids[tid], E, j.expert_map, j.num_map) : E;
  if (write) {
    for (int64_t i = tid; i < j.zero_n; i += kThreads) j.zero[i] = 0;
    for (int64_t i = tid; i < j.max_pad; i += kThreads) j.sorted_ids[i] = (int32_t)j.numel;
  }
  const int rank = round_rank(e, active, E, wcnt, tot);
  padded_offsets(tot, off, warp_tot, E, j.block);
  const int pos = active && e < E ? off[e] + rank : -1;
  if (write) {
    // (the barriers in between order the fill above before these stores of other threads)
    if (pos >= 0) j.sorted_ids[pos] = tid;
    if (tid == 0) j.num_post[0] = off[E];
    if (j.expert_off != nullptr)
      for (int i = tid; i < EP; i += kThreads) j.expert_off[i] = off[i];
    write_expert_ids(off, tot, E, j.block, j.expert_ids, j.block_live, j.max_blocks, tid, kThreads);
  }
  __syncthreads();
  return pos;
}

// The same at the head of an activation gather, whose blocks each take a piece of one token: every block sorts
// for itself (a few microseconds on one SM, as one block would take) instead of waiting for a kernel in front.
// Returns the position of the block's token's slot of index `lane` (< top_k <= 32), -1 if there is none.
__device__ __forceinline__ int positions_of_token(const Job& j, unsigned char* smem, unsigned token, int top_k, bool write) {
  const int pos = align_in_block(j, smem, write);
  int* all = reinterpret_cast<int*>(smem);
  all[threadIdx.x] = pos;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  return lane < top_k ? all[token * top_k + lane] : -1;
}

}  // namespace align
}  // namespace xkb
