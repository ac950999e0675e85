// moe_align_block_size for sm_100a: sort/pad routed token-slots into per-expert
// blocks, bit-exact with the reference (src/xkernels/ops/moe/w4a16.py:53-101):
// stable order inside an expert, every run padded to a multiple of block_size,
// unused entries of sorted_ids = numel, unused entries of expert_ids = 0.
//
// Stability without sorting: a slot's rank inside its expert is the number of same-expert slots before it, which is
// counted in pieces (earlier chunks or blocks, earlier warps, lower lanes by a __match_any_sync ballot).
// Counters only ever count, so atomics never decide an output position.
//
// Latency-bound: a call moves about a megabyte at most, so what counts is the number of dependent steps.
//   numel <= kSmallMax (a decode batch): ONE single-CTA kernel with one pass over the ids; the ranks
//     of the slots and the expert counts come out of the same warp x expert matrix.
//   numel <= kClusterMax: one cluster of eight CTAs.  Every warp counts a contiguous segment of 32 or 64 slots, the CTAs
//     read one another's expert counts through distributed shared memory, and every warp then walks its segment
//     again with running positions: two cluster barriers and no launch between counting and placing.
//   larger inputs: two launches over at most kMaxChunks chunks of whole 1024-slot rounds, count, then place.  Every CTA of
//     the second adds up the chunk x expert matrix for itself and is launched while the first still runs.
// A call: 1040 to 6000 slots 9.6 -> 8.2 us with the cluster; M=16384, top_k=8, E=48, block 16 (two launches) 10.4.
#include "align_dev.cuh"
#include "common.cuh"

namespace xkb {
namespace {

using namespace align;

constexpr int kMaxChunks = 148;        // CTAs of the two-launch path: one wave
constexpr int64_t kNoWorkspaceMax = 8192;   // slots that need no workspace (callers may pass none)
constexpr int kCluster = 8;            // CTAs of the cluster path: the portable cluster size
constexpr int kRounds = 2;             // rounds of 32 slots a warp of the cluster takes at most
// Walking longer segments takes longer than the second launch: 8.2 us a call against 9.6 at 6000 slots and E=64, 12.3 / 12.3 at
// 24000 and 256, 22.6 / 11.3 at 131072 and 48.
constexpr int64_t kClusterMax = (int64_t)kCluster * kWarps * 32 * kRounds;   // 16384

// ---------------------------------------------------------------------------
// Single-CTA path: numel <= 1024.  zero / zero_n: ints the caller wants cleared (nullptr, 0: none).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads)
align_small_kernel(const int32_t* __restrict__ topk_ids, int64_t numel, int E, int block,
                   const int32_t* __restrict__ expert_map, int num_map,
                   int32_t* __restrict__ sorted_ids, int64_t max_pad,
                   int32_t* __restrict__ expert_ids, int64_t max_blocks,
                   int32_t* __restrict__ num_post, int32_t* __restrict__ expert_off_out,
                   int32_t* __restrict__ slot_pos, int32_t* __restrict__ block_live, int32_t* __restrict__ zero, int64_t zero_n) {
  chain_trigger();   // a kernel chained behind this one may be launched; it waits for completion itself
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const Job j{topk_ids, expert_map, sorted_ids, expert_ids, num_post, expert_off_out, block_live, zero, zero_n, numel, max_pad,
              max_blocks, num_map, E, block};
  const int pos = align_in_block(j, smem_raw, true);
  if (threadIdx.x < numel && slot_pos != nullptr) slot_pos[threadIdx.x] = pos;
}

// ---------------------------------------------------------------------------
// Cluster path: warp g of the cluster (kCluster * kWarps of them) takes the slots [g * segment, (g + 1) * segment)
// ---------------------------------------------------------------------------
// (.aligned: every lane of the warp executes it together)
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// the int at the same shared-memory address in CTA `rank` of the cluster
__device__ __forceinline__ int load_remote(const int* p, int rank) {
  uint32_t at;
  int v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(at) : "memory");
  return v;
}

__global__ void __cluster_dims__(kCluster, 1, 1) __launch_bounds__(kThreads)
align_cluster_kernel(const int32_t* __restrict__ topk_ids, int64_t numel, int64_t segment, int E, int block,
                     const int32_t* __restrict__ expert_map, int num_map,
                     int32_t* __restrict__ sorted_ids, int64_t max_pad, int32_t* __restrict__ expert_ids, int64_t max_blocks,
                     int32_t* __restrict__ num_post, int32_t* __restrict__ expert_off_out, int32_t* __restrict__ slot_pos,
                     int32_t* __restrict__ block_live, int32_t* __restrict__ zero, int64_t zero_n) {
  chain_trigger();   // a kernel chained behind this one may be launched; it waits for completion itself
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int EP = E + 1, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = (int)blockIdx.x;   // (one cluster)
  int* wcnt = reinterpret_cast<int*>(smem_raw);   // [kWarps][EP] a warp's slots per expert, then their next place in the CTA
  int* own = wcnt + kWarps * EP;                  // [EP] this CTA's slots per expert
  int* tot = own + EP;                            // [EP] all slots per expert
  int* off = tot + EP;                            // [EP] off[E] = total
  int* base = off + EP;                           // [EP] first position of this CTA's slots
  int* warp_tot = base + EP;                      // [kWarps]
  const int64_t first = ((int64_t)rank * kWarps + warp) * segment;
  const int64_t last = first + segment < numel ? first + segment : numel;
  int e[kRounds];   // the slots' experts (E: dropped); no slot: a number of the lane's own, which matches nobody
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    const int64_t slot = first + r * 32 + lane;
    e[r] = slot < last ? map_expert(topk_ids[slot], E, expert_map, num_map) : EP + lane;
  }
  for (int i = tid; i < kWarps * EP; i += kThreads) wcnt[i] = 0;
  for (int64_t i = (int64_t)rank * kThreads + tid; i < zero_n; i += (int64_t)kCluster * kThreads) zero[i] = 0;
  __syncthreads();
  int* mine = wcnt + warp * EP;
#pragma unroll
  for (int r = 0; r < kRounds; ++r)
    if (e[r] < EP) atomicAdd(&mine[e[r]], 1);
  __syncthreads();
  // exclusive scan over the warps, one expert per scanning warp per step
  for (int x = warp; x < EP; x += kWarps) {
    const int v = wcnt[lane * EP + x];
    int incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += u;
    }
    wcnt[lane * EP + x] = incl - v;
    if (lane == 31) own[x] = incl;
  }
  __syncthreads();
  cluster_arrive();
  cluster_wait();
  int before = 0;
  if (tid < E) {   // E <= kThreads
    int all = 0;
#pragma unroll
    for (int r = 0; r < kCluster; ++r) {
      const int v = load_remote(own + tid, r);
      all += v;
      before += r < rank ? v : 0;
    }
    tot[tid] = all;
  }
  __syncthreads();
  cluster_arrive();   // this CTA has read the others' counts; the wait for theirs is at the end
  padded_offsets(tot, off, warp_tot, E, block);
  if (tid < E) base[tid] = off[tid] + before;
  if (rank == 0) {
    if (tid == 0) num_post[0] = off[E];
    if (expert_off_out != nullptr)
      for (int i = tid; i < EP; i += kThreads) expert_off_out[i] = off[i];
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    const int x = e[r];
    const int64_t slot = first + r * 32 + lane;
    const unsigned peers = __match_any_sync(0xffffffffu, x);
    const int below = __popc(peers & ((1u << lane) - 1u));
    const int at = x < EP ? mine[x] : 0;
    __syncwarp();
    if (x < EP && below == 0) mine[x] = at + __popc(peers);
    __syncwarp();
    if (x < E) sorted_ids[base[x] + at + below] = (int32_t)slot;
    if (x < EP && slot_pos != nullptr) slot_pos[slot] = x < E ? base[x] + at + below : -1;
  }
  // the positions that hold no slot: the ends of the experts' runs, and what lies behind the last
  for (int x = rank * kWarps + warp; x < E; x += kCluster * kWarps)
    for (int i = off[x] + tot[x] + lane; i < off[x + 1]; i += 32) sorted_ids[i] = (int32_t)numel;
  for (int64_t i = off[E] + (int64_t)rank * kThreads + tid; i < max_pad; i += (int64_t)kCluster * kThreads) sorted_ids[i] = (int32_t)numel;
  write_expert_ids(off, tot, E, block, expert_ids, block_live, max_blocks, rank * kThreads + tid, kCluster * kThreads);
  __syncwarp();       // the loops above end lane by lane, and the barrier takes whole warps
  cluster_wait();     // no CTA leaves while another may read its counts
}

size_t cluster_smem(int E) {
  const size_t EP = E + 1;
  return (kWarps * EP + 4 * EP + kWarps) * sizeof(int);
}

// ---------------------------------------------------------------------------
// Two-launch path: count -> place, chunk c = slots [c * span, (c + 1) * span), span a multiple of 1024
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads)
align_count_kernel(const int32_t* __restrict__ topk_ids, int64_t numel, int64_t span, int E,
                   const int32_t* __restrict__ expert_map, int num_map,
                   int32_t* __restrict__ chunk_cnt /*[C][E+1]*/,
                   int32_t* __restrict__ sorted_ids, int64_t max_pad, int32_t* __restrict__ zero, int64_t zero_n) {
  chain_trigger();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int* hist = reinterpret_cast<int*>(smem_raw);
  const int EP = E + 1, tid = threadIdx.x;
  for (int i = tid; i < EP; i += kThreads) hist[i] = 0;
  __syncthreads();
  const int64_t first = (int64_t)blockIdx.x * span;
  const int64_t last = first + span < numel ? first + span : numel;
  for (int64_t slot = first + tid; slot < last; slot += kThreads)
    atomicAdd(&hist[map_expert(topk_ids[slot], E, expert_map, num_map)], 1);
  // pre-fill this CTA's slice of sorted_ids with the padding id
  const int64_t per = (max_pad + gridDim.x - 1) / gridDim.x;
  const int64_t lo = (int64_t)blockIdx.x * per;
  const int64_t hi = (lo + per < max_pad) ? lo + per : max_pad;
  for (int64_t i = lo + tid; i < hi; i += kThreads) sorted_ids[i] = (int32_t)numel;
  for (int64_t i = (int64_t)blockIdx.x * kThreads + tid; i < zero_n; i += (int64_t)gridDim.x * kThreads) zero[i] = 0;
  __syncthreads();
  for (int i = tid; i < EP; i += kThreads) chunk_cnt[(int64_t)blockIdx.x * EP + i] = hist[i];
}

__global__ void __launch_bounds__(kThreads)
align_place_kernel(const int32_t* __restrict__ topk_ids, int64_t numel, int64_t span, int E, int block,
                   const int32_t* __restrict__ expert_map, int num_map,
                   const int32_t* chunk_cnt /*[C][E+1]: written by the kernel this one overlaps*/,
                   int32_t* sorted_ids, int64_t max_pad, int32_t* __restrict__ expert_ids, int64_t max_blocks,
                   int32_t* __restrict__ num_post, int32_t* __restrict__ expert_off_out,
                   int32_t* __restrict__ slot_pos, int32_t* __restrict__ block_live) {
  chain_trigger();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int EP = E + 1, tid = threadIdx.x, C = (int)gridDim.x;
  uint16_t* wcnt = reinterpret_cast<uint16_t*>(smem_raw);                 // [kWarps][EP]
  int* off = reinterpret_cast<int*>(smem_raw + kWarps * EP * sizeof(uint16_t));   // [EP]   off[E] = total
  int* base = off + EP;                                                   // [EP]   next position per expert
  int* tot = base + EP;                                                   // [EP]
  int* warp_tot = tot + EP;                                               // [kWarps]
  for (int i = tid; i < EP; i += kThreads) base[i] = tot[i] = 0;
  __syncthreads();
  const int64_t first = (int64_t)blockIdx.x * span;
  const int64_t last = first + span < numel ? first + span : numel;
  int64_t slot = first + tid;
  bool active = slot < last;
  int e = active ? map_expert(topk_ids[slot], E, expert_map, num_map) : E;   // an input of the call, not of the kernel before
  chain_wait();
  // slots per expert in all chunks (tot) and in the chunks before this one (base): threads side by side
  // take neighbouring experts, the groups of threads share the chunks out
  const int width = E < kThreads ? (E > 0 ? E : 1) : kThreads;
  const int groups = kThreads / width, grp = tid / width;
  if (grp < groups) {
    for (int x = tid - grp * width; x < E; x += width) {
      int all = 0, before = 0;
#pragma unroll 8
      for (int c = grp; c < C; c += groups) {
        const int v = __ldcg(chunk_cnt + (int64_t)c * EP + x);
        all += v;
        if (c < (int)blockIdx.x) before += v;
      }
      if (all != 0) atomicAdd(&tot[x], all);
      if (before != 0) atomicAdd(&base[x], before);
    }
  }
  __syncthreads();
  padded_offsets(tot, off, warp_tot, E, block);
  for (int i = tid; i < E; i += kThreads) base[i] += off[i];
  if (blockIdx.x == 0) {
    if (tid == 0) num_post[0] = off[E];
    if (expert_off_out != nullptr)
      for (int i = tid; i < EP; i += kThreads) expert_off_out[i] = off[i];
  }
  write_expert_ids(off, tot, E, block, expert_ids, block_live, max_blocks, (int)blockIdx.x * kThreads + tid, C * kThreads);
  __syncthreads();
  for (int64_t s0 = first; s0 < last; s0 += kThreads) {
    if (s0 != first) {
      slot = s0 + tid;
      active = slot < last;
      e = active ? map_expert(topk_ids[slot], E, expert_map, num_map) : E;
    }
    const int rank = round_rank(e, active, E, wcnt, tot);
    if (active && e < E) sorted_ids[base[e] + rank] = (int32_t)slot;
    if (active && slot_pos != nullptr) slot_pos[slot] = e < E ? base[e] + rank : -1;
    if (s0 + kThreads < last) {
      __syncthreads();
      for (int i = tid; i < E; i += kThreads) base[i] += tot[i];
      __syncthreads();
    }
  }
}

size_t place_smem(int E) {
  const size_t EP = E + 1;
  return kWarps * EP * sizeof(uint16_t) + 3 * EP * sizeof(int) + kWarps * sizeof(int);
}

template <typename K>
cudaError_t allow_smem(K kernel, size_t bytes) {
  if (bytes <= 48 * 1024) return cudaSuccess;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

}  // namespace

int64_t align_workspace_bytes(int64_t numel, int num_experts) {
  const int64_t C = ceil_div(numel > 0 ? numel : 1, kChunk);
  // at least the chunk x expert matrix (callers size buffers by this formula: it stays as it is)
  return align_up(C * (num_experts + 1) * 4, 256) + align_up((int64_t)(num_experts + 1) * 4, 256);
}

int launch_align(const int32_t* topk_ids, int64_t numel, int E, int block,
                 const int32_t* expert_map, int num_map, int32_t* sorted_ids,
                 int32_t* expert_ids, int32_t* num_post, int32_t* expert_off,
                 void* workspace, int64_t workspace_bytes, cudaStream_t stream, int32_t* zero, int64_t zero_n,
                 int32_t* slot_pos, int32_t* block_live) {
  XKB_REQUIRE(numel >= 0 && numel < (1ll << 30), "moe_align: numel=%lld out of range", (long long)numel);
  XKB_REQUIRE(block > 0, "moe_align: block_size must be > 0 (got %d)", block);
  XKB_REQUIRE(E >= 0 && E <= kMaxExperts, "moe_align: num_experts=%d outside [0,%d]", E, kMaxExperts);
  XKB_REQUIRE(sorted_ids && expert_ids && num_post, "moe_align: null output pointer");
  XKB_REQUIRE(numel == 0 || topk_ids, "moe_align: null topk_ids");
  const int64_t max_pad = numel + (int64_t)(E + 1) * (block - 1);
  const int64_t max_blocks = ceil_div(max_pad, block);
  if (numel <= kSmallMax) {
    const size_t smem = small_smem(E);
    XKB_CHECK_CUDA(allow_smem(align_small_kernel, smem));
    align_small_kernel<<<1, kThreads, smem, stream>>>(topk_ids, numel, E, block, expert_map, num_map,
                                                      sorted_ids, max_pad, expert_ids, max_blocks,
                                                      num_post, expert_off, slot_pos, block_live, zero, zero_n);
    XKB_CHECK_LAUNCH("align_small_kernel");
    return XKB_OK;
  }
  const int64_t need = align_workspace_bytes(numel, E);
  if ((workspace == nullptr || workspace_bytes < need) && (numel > kNoWorkspaceMax || zero_n != 0))
    return fail(XKB_ERR_WORKSPACE, "moe_align: workspace of %lld bytes needed, %lld given",
                (long long)need, (long long)workspace_bytes);
  if (numel <= kClusterMax) {
    const int64_t segment = align_up(ceil_div(numel, (int64_t)kCluster * kWarps), 32);
    const size_t smem = cluster_smem(E);
    XKB_CHECK_CUDA(allow_smem(align_cluster_kernel, smem));
    align_cluster_kernel<<<kCluster, kThreads, smem, stream>>>(topk_ids, numel, segment, E, block, expert_map, num_map, sorted_ids,
                                                               max_pad, expert_ids, max_blocks, num_post, expert_off, slot_pos,
                                                               block_live, zero, zero_n);
    XKB_CHECK_LAUNCH("align_cluster_kernel");
    return XKB_OK;
  }
  const int64_t span = ceil_div(numel, (int64_t)kMaxChunks * kChunk) * kChunk;
  const int C = (int)ceil_div(numel, span);
  int32_t* chunk_cnt = static_cast<int32_t*>(workspace);
  const size_t smem1 = (size_t)(E + 1) * sizeof(int);
  const size_t smem2 = place_smem(E);
  XKB_CHECK_CUDA(allow_smem(align_place_kernel, smem2));
  align_count_kernel<<<C, kThreads, smem1, stream>>>(topk_ids, numel, span, E, expert_map, num_map,
                                                     chunk_cnt, sorted_ids, max_pad, zero, zero_n);
  XKB_CHECK_LAUNCH("align_count_kernel");
  XKB_CHECK_CUDA(launch_chained(align_place_kernel, dim3((unsigned)C), dim3(kThreads), smem2, stream, topk_ids, numel,
                                span, E, block, expert_map, num_map, chunk_cnt, sorted_ids, max_pad, expert_ids, max_blocks,
                                num_post, expert_off, slot_pos, block_live));
  XKB_CHECK_LAUNCH("align_place_kernel");
  return XKB_OK;
}

}  // namespace xkb

extern "C" int64_t xkb_moe_align_workspace_bytes(int64_t numel, int num_experts) {
  return xkb::align_workspace_bytes(numel, num_experts);
}

extern "C" int xkb_moe_align_block_size(const int32_t* topk_ids, int64_t numel, int num_experts,
                                        int block_size, const int32_t* expert_map, int num_map,
                                        int32_t* sorted_ids, int32_t* expert_ids,
                                        int32_t* num_post_pad, int32_t* expert_offsets,
                                        void* workspace, int64_t workspace_bytes, void* stream) {
  return xkb::launch_align(topk_ids, numel, num_experts, block_size, expert_map, num_map, sorted_ids,
                           expert_ids, num_post_pad, expert_offsets, workspace, workspace_bytes,
                           static_cast<cudaStream_t>(stream));
}

// ---------------------------------------------------------------------------
// Allocation-free variant.
//
// Some hosts of this library may not create device memory at all: a plug-in that runs inside
// another runtime's memory pool, code that executes while that runtime forbids allocation (for
// example between the points where its allocator may be entered), or a C caller that simply has
// no allocator for scratch buffers.  For them the chunk x expert count matrix of the multi-launch
// align path lives in a fixed array inside the library image instead of a caller workspace.
// The price is a size limit and the loss of re-entrancy (see the header comment).
// ---------------------------------------------------------------------------
namespace xkb {
namespace {

constexpr int64_t kStaticMaxSlots = 262144;   // numel limit: 256 chunks of 1024 slots
constexpr int kStaticMaxExperts = 256;        // num_experts limit
constexpr int64_t kStaticChunks = kStaticMaxSlots / kChunk;
constexpr int64_t kStaticInts = kStaticChunks * (kStaticMaxExperts + 1) + (kStaticMaxExperts + 1) + 256;

// 265 220 bytes (259 KiB) per GPU that loads the library, held until the process exits.
static __device__ __align__(256) int32_t g_align_static_scratch[kStaticInts];

constexpr int kMaxDevices = 64;
std::atomic<void*> g_static_ptr[kMaxDevices];   // device address of the array, per device (zero-initialised)

// The array's name is only a host-side handle; the device address has to be asked for, once per
// device, with that device current.  The address is looked up for the device that is CURRENT at
// the call, so the stream passed in must belong to the current device (as for any launch).
// Threads that race on a device's first call all store the same value.
int static_scratch_address(void** out) {
  int dev = -1;
  XKB_CHECK_CUDA(cudaGetDevice(&dev));
  XKB_REQUIRE(dev >= 0 && dev < kMaxDevices, "moe_align (static): device index %d not supported", dev);
  void* p = g_static_ptr[dev].load(std::memory_order_acquire);
  if (p == nullptr) {
    XKB_CHECK_CUDA(cudaGetSymbolAddress(&p, g_align_static_scratch));
    XKB_REQUIRE(p != nullptr, "moe_align (static): cudaGetSymbolAddress returned a null address");
    g_static_ptr[dev].store(p, std::memory_order_release);
  }
  *out = p;
  return XKB_OK;
}

}  // namespace
}  // namespace xkb

extern "C" int xkb_moe_align_block_size_static(const int32_t* topk_ids, int64_t numel, int num_experts,
                                               int block_size, const int32_t* expert_map, int num_map,
                                               int32_t* sorted_ids, int32_t* expert_ids,
                                               int32_t* num_post_pad, int32_t* expert_offsets,
                                               void* stream) {
  using namespace xkb;
  XKB_REQUIRE(numel >= 0 && numel <= kStaticMaxSlots,
              "moe_align (static): numel=%lld exceeds the built-in scratch limit of %lld token-slots; "
              "use xkb_moe_align_block_size with a caller workspace",
              (long long)numel, (long long)kStaticMaxSlots);
  XKB_REQUIRE(num_experts >= 0 && num_experts <= kStaticMaxExperts,
              "moe_align (static): num_experts=%d exceeds the built-in scratch limit of %d; "
              "use xkb_moe_align_block_size with a caller workspace",
              num_experts, kStaticMaxExperts);
  void* scratch = nullptr;
  const int rc = static_scratch_address(&scratch);
  if (rc != XKB_OK) return rc;
  // Nothing in the scratch has to start at zero: the count kernel writes every entry of the
  // chunk x expert matrix that the place kernel reads.
  return launch_align(topk_ids, numel, num_experts, block_size, expert_map, num_map, sorted_ids,
                      expert_ids, num_post_pad, expert_offsets, scratch,
                      kStaticInts * (int64_t)sizeof(int32_t), static_cast<cudaStream_t>(stream));
}
