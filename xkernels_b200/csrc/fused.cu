// Host side of the fused ops: workspace carving, kernel-path choice and the
// launch sequence  align -> grouped GEMM(s) -> fixed-order fp32 combine.
// Everything is enqueued on the caller's stream; no host synchronisation and no
// allocation happens here.
#include "align_dev.cuh"
#include "common.cuh"
#include "moe_kernels.h"

#include <vector>

namespace xkb {

std::atomic<int64_t> g_launches{0};

char* last_error_buf() {
  static thread_local char buf[512] = {0};
  return buf;
}

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(last_error_buf(), 512, fmt, ap);
  va_end(ap);
  return code;
}

// ---- optional per-call timing of the grouped-GEMM kernel(s) -----------------
// A ring of event pairs; when enabled, every fused call records one pair around
// its expert GEMM launch(es) on the caller's stream.
struct GemmTimer {
  std::vector<cudaEvent_t> start, stop;
  int used = 0;
  bool enabled = false;
};
static GemmTimer g_timer;

// Scopes nest: only the outermost one records (two GEMMs that overlap are timed as one span, and no
// event lands between them, which would serialise them).
static thread_local int g_timer_depth = 0;
GemmTimerScope::GemmTimerScope(cudaStream_t s) : stream(s), slot(-1) {
  if (g_timer_depth++ == 0 && g_timer.enabled && g_timer.used < (int)g_timer.start.size()) {
    slot = g_timer.used++;
    cudaEventRecord(g_timer.start[slot], stream);
  }
}
GemmTimerScope::~GemmTimerScope() {
  --g_timer_depth;
  if (slot >= 0) cudaEventRecord(g_timer.stop[slot], stream);
}

namespace {

struct RoutingBuffers {
  int* status;
  int64_t num_blocks;       // token blocks that the arrays with one entry per block hold
  int64_t num_positions;    // length of sorted_ids
  int32_t* counters;        // one per block, directly behind the status header: cleared as one span
  int32_t* sorted_ids;
  int32_t* expert_ids;
  int32_t* num_post;
  int32_t* expert_off;
  int32_t* slot_pos;
  int32_t* block_live;
  void* align_ws;
  int64_t align_ws_bytes;
};

// Routing buffers are sized for the worst case over the block sizes any path may pick: the longest
// sorted_ids (largest block) and the most blocks.  The sort writes ceil((numel + (E + 1) (B - 1)) / B) entries
// per block array at block size B, which is below numel / B + E + 2 - (E + 1) / B, so numel / kMinBlock + E + 2 holds them
// at every B >= kMinBlock.  (The count at the smallest block is no such bound: with fewer slots than experts wider
// blocks have more entries, 257 at B = 16 and 240 at B = 8 for 8 slots and 272 experts.)
constexpr int kMaxBlock = 256;
constexpr int kMinBlock = 8;

int64_t routing_max_pad(int64_t numel, int E, int block) {
  return numel + (int64_t)(E + 1) * (block - 1);
}
int64_t routing_max_blocks(int64_t numel, int E) { return numel / kMinBlock + E + 2; }

RoutingBuffers carve_routing(Carver& c, int64_t numel, int E) {
  RoutingBuffers r;
  r.status = c.take<int>(64);  // workspace header: word 0 = device status of the last call
  r.num_blocks = routing_max_blocks(numel, E);
  r.num_positions = routing_max_pad(numel, E, kMaxBlock);
  r.counters = c.take<int32_t>(r.num_blocks);
  r.sorted_ids = c.take<int32_t>(r.num_positions);
  r.expert_ids = c.take<int32_t>(r.num_blocks);
  r.num_post = c.take<int32_t>(1);
  r.expert_off = c.take<int32_t>(E + 1);
  r.slot_pos = c.take<int32_t>(numel);
  r.block_live = c.take<int32_t>(r.num_blocks);
  r.align_ws_bytes = align_workspace_bytes(numel, E);
  r.align_ws = c.take<char>(r.align_ws_bytes);
  return r;
}

// status header and the block counters behind it, as one span
int64_t header_ints(const RoutingBuffers& r) { return r.counters + r.num_blocks - r.status; }

int64_t routing_bytes(int64_t numel, int E) {
  Carver c(nullptr);
  carve_routing(c, numel, E);
  return c.off;
}

int make_routing(const RoutingBuffers& b, int64_t numel, int E, int block, Routing* out) {
  Routing r;
  r.sorted_ids = b.sorted_ids;
  r.expert_ids = b.expert_ids;
  r.num_post = b.num_post;
  r.expert_off = b.expert_off;
  r.slot_pos = b.slot_pos;
  r.block_live = b.block_live;
  r.numel = numel;
  r.block = block;
  r.max_pad = routing_max_pad(numel, E, block);
  r.max_blocks = ceil_div(r.max_pad, block);
  r.block_counters = b.counters;
  r.job = nullptr;
  XKB_REQUIRE(r.max_pad <= b.num_positions && r.max_blocks <= b.num_blocks,
              "routing: blocks of %d do not fit the routing buffers (%lld of %lld positions, %lld of %lld blocks)", block,
              (long long)r.max_pad, (long long)b.num_positions, (long long)r.max_blocks, (long long)b.num_blocks);
  *out = r;
  return XKB_OK;
}

// The align stage of a fused call: clears the status word and the block counters on its way.  A decode batch on
// a tensor-core path is sorted by the activation gather itself (r->job = *job): one launch less, and the gather
// does not wait for another kernel's completion.  Larger batches take the sort's own kernels.
// Whole calls: K=2048, N=7168, E=48, top_k=8 at M=1 39.8 -> 32.7 us, M=64 110.0 -> 108.1; K=7168, N=4096 at M=1 46.0 -> 44.0 us
// (M=64: 1 %, within its runs' spread).  At M=128 (1024 slots: nearly every SM sorts) nothing is left of it: 132.4 / 132.0
// us, and the two-GEMM layer 448 / 451, so the line lies at M=64's 512 slots.  Every block of the gather sorts, so they
// have to fit the SMs side by side as well: K=2048, N=512, E=48, the sort's own kernels against this, 128 blocks 20.5 /
// 19.1 us (top_k 1) and 21.4 / 20.0 (2), 256 blocks 21.1 / 22.7 and 22.4 / 23.9, 512 blocks 21.9 / 29.6; E=1024, N=256
// 27.9 / 26.6, 36.9 / 43.1 and 49.4 / 73.3.
constexpr int64_t kSortInGatherMax = 512;
constexpr unsigned kSortInGatherBlocks = 148;
static_assert(kSortInGatherMax <= align::kSmallMax, "the sort takes one slot per thread");
// A map that leaves a token two kept slots or fewer on average (top_k * local experts / all experts: a rank's share)
// has the gather of a large batch go through the kept slots' positions: going through the tokens starts a block for each
// of them, most of which only find out that they have nothing to do.  K=2048, N=2048, top_k=8, whole calls, tokens against
// positions: M=16384 with 1 of 256 experts 104 / 84 us, 8 of 256 130 / 115, 32 of 256 248 / 242; M=2048 (2048 blocks)
// 36.0 / 36.4, 38.3 / 39.5 and 58.7 / 60.7, so the line lies at two rounds of sixteen blocks per SM.
constexpr int64_t kPositionsPerToken = 2;
constexpr unsigned kPositionsMinBlocks = 2 * 16 * 148;
int route(const RoutingBuffers& rb, const int32_t* topk_ids, const int32_t* expert_map, int num_map, int E, int top_k,
          int64_t gather_units, Routing* r, align::Job* job, cudaStream_t stream) {   // gather_units: of a row, 0 = no gather
  GatherGrid g{};
  r->by_position = gather_units > 0 && expert_map != nullptr && (int64_t)top_k * E <= kPositionsPerToken * num_map &&
                   gather_grid(r->numel / top_k, gather_units, false, &g) == XKB_OK && g.blocks > kPositionsMinBlocks;
  if (gather_units > 0 && r->numel >= 1 && r->numel <= kSortInGatherMax && top_k <= 32 && E >= 1 && E <= align::kMaxExperts &&
      gather_grid(r->numel / top_k, gather_units, true, &g) == XKB_OK && g.blocks <= kSortInGatherBlocks) {
    *job = align::Job{topk_ids, expert_map, rb.sorted_ids, rb.expert_ids, rb.num_post, rb.expert_off, rb.block_live, rb.status,
                      header_ints(rb), r->numel, r->max_pad, r->max_blocks, num_map, E, r->block};
    r->job = job;
    return XKB_OK;
  }
  return launch_align(topk_ids, r->numel, E, r->block, expert_map, num_map, rb.sorted_ids, rb.expert_ids, rb.num_post,
                      rb.expert_off, rb.align_ws, rb.align_ws_bytes, stream, rb.status, header_ints(rb), rb.slot_pos, rb.block_live);
}

bool tma_base_ok(const void* a, const void* b) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15) == 0;
}

}  // namespace
}  // namespace xkb

using namespace xkb;

extern "C" const char* xkb_version(void) { return "xkb200 0.1 (sm_100a)"; }
extern "C" const char* xkb_last_error(void) { return last_error_buf(); }
extern "C" int64_t xkb_launch_count(void) { return g_launches.load(); }

extern "C" int xkb_int4_token_tile(int64_t numel, int E, int top_k) { return int4_tc_block(numel, E, top_k); }
extern "C" int xkb_mxfp4_token_tile(int64_t numel, int E) {
  const int block = mxfp4_bs_block(numel, E);
  return block > 0 ? block : mxfp4_tc_block(numel, E);
}
extern "C" int64_t xkb_routing_blocks(int64_t numel, int E) { return numel < 0 || E < 0 ? -1 : routing_max_blocks(numel, E); }

// ---------------------------------------------------------------------------
// INT4 W4A16
// ---------------------------------------------------------------------------
extern "C" int64_t xkb_fused_moe_int4_w4a16_workspace_bytes(int64_t M, int64_t N, int64_t K, int E,
                                                            int top_k, int a_dtype) {
  (void)a_dtype;
  if (M < 0 || N < 0 || K < 0 || E < 0 || top_k < 0) return -1;
  const int64_t numel = M * top_k;
  int64_t total = routing_bytes(numel, E);
  total += align_up(numel * N * 4, 256);           // fp32 slot-indexed rows
  total += int4_tc_workspace_bytes(numel, N, K, E);  // gathered activations etc.
  return total + 256;
}

// rows_out == nullptr: combine into `out` ([M,N], a_dtype).  rows_out != nullptr: leave the fp32
// per-slot rows ([M*top_k, N], row = token*top_k + j) there and skip the combine.
static int int4_impl(const void* A, int a_dtype, const int32_t* packed, const void* scale,
                     const int32_t* topk_ids, const float* topk_w, const int32_t* expert_map,
                     int num_map, void* out, float* rows_out, int64_t M, int64_t N, int64_t K, int E,
                     int top_k, int group_size, int mul_routed_weight, int path, void* workspace,
                     int64_t workspace_bytes, cudaStream_t stream, int out_dtype = -1) {
  if (out_dtype < 0) out_dtype = a_dtype;
  XKB_REQUIRE(a_dtype == XKB_BF16 || a_dtype == XKB_F32, "fused_moe_int4_w4a16: bad a_dtype %d", a_dtype);
  XKB_REQUIRE(M >= 0 && N >= 0 && K >= 0 && E >= 0 && top_k >= 0, "fused_moe_int4_w4a16: negative dim");
  XKB_REQUIRE(group_size > 0 && group_size % 8 == 0 && K % group_size == 0 && K % 8 == 0,
              "fused_moe_int4_w4a16: need K %% 8 == 0, group_size %% 8 == 0, K %% group_size == 0 "
              "(K=%lld group_size=%d)", (long long)K, group_size);
  XKB_REQUIRE(path == XKB_PATH_AUTO || path == XKB_PATH_SIMT || path == XKB_PATH_TC,
              "fused_moe_int4_w4a16: bad path %d", path);
  if (M == 0 || N == 0) return XKB_OK;
  XKB_REQUIRE(A && packed && scale && topk_ids && (out || rows_out),
              "fused_moe_int4_w4a16: null pointer argument");
  XKB_REQUIRE(topk_w || !mul_routed_weight, "fused_moe_int4_w4a16: topk_w is null");
  const int64_t need = xkb_fused_moe_int4_w4a16_workspace_bytes(M, N, K, E, top_k, a_dtype);
  if (workspace == nullptr || workspace_bytes < need)
    return fail(XKB_ERR_WORKSPACE, "fused_moe_int4_w4a16: workspace of %lld bytes needed, %lld given",
                (long long)need, (long long)workspace_bytes);
  XKB_REQUIRE(reinterpret_cast<uintptr_t>(workspace) % 256 == 0, "workspace must be 256-byte aligned");

  const int64_t numel = M * top_k;
  Carver carve(workspace);
  RoutingBuffers rb = carve_routing(carve, numel, E);
  float* scratch = carve.take<float>(numel * N);
  if (rows_out != nullptr) scratch = rows_out;
  void* tc_ws = carve.take<char>(int4_tc_workspace_bytes(numel, N, K, E));

  // (the other groups came to the tcgen05 path later: weights that TMA cannot read keep the generic kernel there)
  const bool tc_fit = int4_tc_supported(a_dtype, M, N, K, E, top_k, group_size) &&
                      (group_size == 32 || tma_base_ok(packed, scale));
  if (path == XKB_PATH_TC && !(tc_fit && group_size == 32))
    return fail(XKB_ERR_ARG,
                "fused_moe_int4_w4a16: shape not supported by the tcgen05 path (needs bf16 A, "
                "N %% 128 == 0, K %% 256 == 0, group_size 32)");
  const bool use_tc = (path == XKB_PATH_TC) || (path == XKB_PATH_AUTO && tc_fit);
  const int block = use_tc ? int4_tc_block(numel, E, top_k) : kSimtBlock;

  Routing r;
  align::Job job;
  int rc = make_routing(rb, numel, E, block, &r);
  if (rc != XKB_OK) return rc;
  rc = route(rb, topk_ids, expert_map, num_map, E, top_k, use_tc ? K / 8 : 0, &r, &job, stream);
  if (rc != XKB_OK) return rc;
  if (use_tc)
    rc = launch_int4_tc(A, packed, scale, r, topk_w, scratch, N, K, E, top_k, group_size,
                        mul_routed_weight, tc_ws, rb.status, stream);
  else
    rc = launch_int4_simt(A, a_dtype, packed, scale, r, topk_w, scratch, N, K, top_k, group_size,
                          mul_routed_weight, stream);
  if (rc != XKB_OK) return rc;
  if (rows_out != nullptr) return XKB_OK;
  return launch_combine(scratch, topk_ids, expert_map, num_map, E, out, out_dtype, M, top_k, N, stream);
}

extern "C" int xkb_fused_moe_int4_w4a16(const void* A, int a_dtype, const int32_t* packed,
                                        const void* scale, const int32_t* topk_ids,
                                        const float* topk_w, const int32_t* expert_map, int num_map,
                                        void* out, int64_t M, int64_t N, int64_t K, int E, int top_k,
                                        int group_size, int mul_routed_weight, int path,
                                        void* workspace, int64_t workspace_bytes, void* stream) {
  XKB_REQUIRE(out != nullptr || M == 0 || N == 0, "fused_moe_int4_w4a16: null out");
  return int4_impl(A, a_dtype, packed, scale, topk_ids, topk_w, expert_map, num_map, out, nullptr, M, N,
                   K, E, top_k, group_size, mul_routed_weight, path, workspace, workspace_bytes,
                   static_cast<cudaStream_t>(stream));
}

extern "C" int xkb_moe_int4_w4a16_rows(const void* A, int a_dtype, const int32_t* packed,
                                       const void* scale, const int32_t* topk_ids, const float* topk_w,
                                       float* rows_out, int64_t M, int64_t N, int64_t K, int E,
                                       int top_k, int group_size, int mul_routed_weight, int path,
                                       void* workspace, int64_t workspace_bytes, void* stream) {
  XKB_REQUIRE(rows_out != nullptr || M == 0 || N == 0, "moe_int4_w4a16_rows: null rows_out");
  return int4_impl(A, a_dtype, packed, scale, topk_ids, topk_w, nullptr, 0, nullptr, rows_out, M, N, K,
                   E, top_k, group_size, mul_routed_weight, path, workspace, workspace_bytes,
                   static_cast<cudaStream_t>(stream));
}

// ---------------------------------------------------------------------------
// Expert side of the all-to-all mode in one call: received rows whose routing travels with them as
// [M, 2*top_k] int32 (top_k local expert ids, -1 = slot served elsewhere, then the top_k routing
// weights' bit patterns) -> one fp32 partial row per received row (the weighted sum over its local
// experts, ascending slot order).  The routing is split into the two contiguous arrays the align
// stage and the combine read by a small kernel, so that the host makes ONE call per chunk.
// ---------------------------------------------------------------------------
namespace xkb {
namespace {
__global__ void __launch_bounds__(256)
split_routing_kernel(const int32_t* __restrict__ routing, int64_t numel, int top_k, int32_t* __restrict__ ids,
                     float* __restrict__ w) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= numel) return;
  const int64_t m = i / top_k;
  const int j = (int)(i - m * top_k);
  ids[i] = routing[m * 2 * top_k + j];
  w[i] = __int_as_float(routing[m * 2 * top_k + top_k + j]);
}
}  // namespace
}  // namespace xkb

extern "C" int64_t xkb_moe_int4_w4a16_partial_workspace_bytes(int64_t M, int64_t N, int64_t K, int E, int top_k,
                                                              int a_dtype) {
  const int64_t base = xkb_fused_moe_int4_w4a16_workspace_bytes(M, N, K, E, top_k, a_dtype);
  if (base < 0) return base;
  return base + 2 * align_up(M * top_k * 4, 256);
}

extern "C" int xkb_moe_int4_w4a16_partial(const void* A, int a_dtype, const int32_t* packed, const void* scale,
                                          const int32_t* routing, float* out, int64_t M, int64_t N, int64_t K,
                                          int E, int top_k, int group_size, int path, void* workspace,
                                          int64_t workspace_bytes, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  XKB_REQUIRE(M >= 0 && N >= 0 && K >= 0 && E >= 0 && top_k >= 1, "moe_int4_w4a16_partial: bad dimension");
  if (M == 0 || N == 0) return XKB_OK;
  XKB_REQUIRE(routing != nullptr && out != nullptr, "moe_int4_w4a16_partial: null routing/out");
  const int64_t need = xkb_moe_int4_w4a16_partial_workspace_bytes(M, N, K, E, top_k, a_dtype);
  if (workspace == nullptr || workspace_bytes < need)
    return fail(XKB_ERR_WORKSPACE, "moe_int4_w4a16_partial: workspace of %lld bytes needed, %lld given",
                (long long)need, (long long)workspace_bytes);
  XKB_REQUIRE(reinterpret_cast<uintptr_t>(workspace) % 256 == 0, "workspace must be 256-byte aligned");
  // the two routing arrays sit behind the fused op's own workspace
  const int64_t base = xkb_fused_moe_int4_w4a16_workspace_bytes(M, N, K, E, top_k, a_dtype);
  const int64_t numel = M * top_k;
  int32_t* ids = reinterpret_cast<int32_t*>(static_cast<char*>(workspace) + align_up(base, 256));
  float* w = reinterpret_cast<float*>(reinterpret_cast<char*>(ids) + align_up(numel * 4, 256));
  split_routing_kernel<<<(unsigned)ceil_div(numel, 256), 256, 0, stream>>>(routing, numel, top_k, ids, w);
  XKB_CHECK_LAUNCH("split_routing_kernel");
  return int4_impl(A, a_dtype, packed, scale, ids, w, nullptr, 0, out, nullptr, M, N, K, E, top_k, group_size, 1,
                   path, workspace, base, stream, XKB_F32);
}

// ---------------------------------------------------------------------------
// INT4 two-GEMM expert layer
// ---------------------------------------------------------------------------
extern "C" int64_t xkb_fused_moe_int4_ffn_workspace_bytes(int64_t M, int64_t hidden, int64_t inter, int E, int top_k,
                                                          int a_dtype) {
  (void)a_dtype;
  if (M < 0 || hidden < 0 || inter < 0 || E < 0 || top_k < 0) return -1;
  const int64_t numel = M * top_k;
  int64_t total = routing_bytes(numel, E);
  total += align_up(numel * hidden * 4, 256);                                   // fp32 slot rows of the down GEMM
  total += align_up(numel * 2 * inter * 4, 256);                                // fp32 gate_up slot rows (generic path)
  total += align_up(routing_max_pad(numel, E, kMaxBlock) * inter * 4, 256);     // activations (bf16 by position, or by slot)
  total += int4_tc_workspace_bytes(numel, hidden, hidden, E);                   // gathered input activations
  return total + 256;
}

extern "C" int xkb_fused_moe_int4_ffn(const void* A, int a_dtype, const int32_t* w13_packed, const void* w13_scale,
                                      const int32_t* w2_packed, const void* w2_scale, const int32_t* topk_ids,
                                      const float* topk_w, const int32_t* expert_map, int num_map, void* out,
                                      int64_t M, int64_t hidden, int64_t inter, int E, int top_k, int group_size,
                                      float swiglu_limit, int path, void* workspace, int64_t workspace_bytes,
                                      void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  XKB_REQUIRE(a_dtype == XKB_BF16 || a_dtype == XKB_F32, "fused_moe_int4_ffn: bad a_dtype %d", a_dtype);
  XKB_REQUIRE(M >= 0 && hidden >= 0 && inter >= 0 && E >= 0 && top_k >= 0, "fused_moe_int4_ffn: negative dim");
  XKB_REQUIRE(group_size > 0 && group_size % 8 == 0 && hidden % group_size == 0 && inter % group_size == 0,
              "fused_moe_int4_ffn: hidden and inter must be multiples of group_size, group_size of 8 "
              "(hidden=%lld inter=%lld group_size=%d)", (long long)hidden, (long long)inter, group_size);
  XKB_REQUIRE(path == XKB_PATH_AUTO || path == XKB_PATH_SIMT || path == XKB_PATH_TC, "fused_moe_int4_ffn: bad path %d", path);
  if (M == 0 || hidden == 0) return XKB_OK;
  XKB_REQUIRE(A && w13_packed && w13_scale && w2_packed && w2_scale && topk_ids && topk_w && out,
              "fused_moe_int4_ffn: null pointer argument");
  const int64_t need = xkb_fused_moe_int4_ffn_workspace_bytes(M, hidden, inter, E, top_k, a_dtype);
  if (workspace == nullptr || workspace_bytes < need)
    return fail(XKB_ERR_WORKSPACE, "fused_moe_int4_ffn: workspace of %lld bytes needed, %lld given", (long long)need,
                (long long)workspace_bytes);
  XKB_REQUIRE(reinterpret_cast<uintptr_t>(workspace) % 256 == 0, "workspace must be 256-byte aligned");

  const int64_t numel = M * top_k;
  Carver carve(workspace);
  RoutingBuffers rb = carve_routing(carve, numel, E);
  float* scratch = carve.take<float>(numel * hidden);
  float* rows1 = carve.take<float>(numel * 2 * inter);
  void* act = carve.take<float>(routing_max_pad(numel, E, kMaxBlock) * inter);
  void* tc_ws = carve.take<char>(int4_tc_workspace_bytes(numel, hidden, hidden, E));

  const bool tc_fit = int4_ffn_tc_supported(a_dtype, M, hidden, inter, E, top_k, group_size) &&
                      (group_size == 32 || (tma_base_ok(w13_packed, w13_scale) && tma_base_ok(w2_packed, w2_scale)));
  if (path == XKB_PATH_TC && !(tc_fit && group_size == 32))
    return fail(XKB_ERR_ARG, "fused_moe_int4_ffn: shape not supported by the tcgen05 path (needs bf16 A, "
                             "hidden %% 256 == 0, inter %% 256 == 0, group_size 32)");
  const bool use_tc = (path == XKB_PATH_TC) || (path == XKB_PATH_AUTO && tc_fit);
  const int block = use_tc ? int4_tc_block(numel, E, top_k) : kSimtBlock;
  Routing r;
  align::Job job;
  int rc = make_routing(rb, numel, E, block, &r);
  if (rc != XKB_OK) return rc;
  rc = route(rb, topk_ids, expert_map, num_map, E, top_k, use_tc ? hidden / 8 : 0, &r, &job, stream);
  if (rc != XKB_OK) return rc;
  if (use_tc) {
    __nv_bfloat16* rows16 = reinterpret_cast<__nv_bfloat16*>(scratch);
    rc = launch_int4_ffn_tc(A, w13_packed, w13_scale, w2_packed, w2_scale, r, topk_w, static_cast<__nv_bfloat16*>(act),
                            rows16, hidden, inter, E, top_k, group_size, swiglu_limit, tc_ws, rb.status, stream);
    if (rc != XKB_OK) return rc;
    return launch_combine_bf16(rows16, nullptr, topk_ids, expert_map, num_map, E, out, a_dtype, M, top_k, hidden, stream);
  }
  rc = launch_int4_ffn_simt(A, a_dtype, w13_packed, w13_scale, w2_packed, w2_scale, r, topk_ids, expert_map, num_map,
                            E, topk_w, rows1, act, scratch, hidden, inter, top_k, group_size, swiglu_limit, stream);
  if (rc != XKB_OK) return rc;
  return launch_combine(scratch, topk_ids, expert_map, num_map, E, out, a_dtype, M, top_k, hidden, stream);
}

// ---------------------------------------------------------------------------
// MXFP4
// ---------------------------------------------------------------------------
extern "C" int64_t xkb_fused_moe_mxfp4_workspace_bytes(int64_t M, int64_t hidden, int64_t ispp, int E,
                                                       int top_k) {
  if (M < 0 || hidden < 0 || ispp < 0 || E < 0 || top_k < 0) return -1;
  const int64_t numel = M * top_k;
  int64_t total = routing_bytes(numel, E);
  int64_t own = align_up(numel * hidden * 4, 256);                          // fp32 partial rows
  own += align_up(routing_max_pad(numel, E, kMaxBlock) * ispp * 2, 256);    // bf16 activations
  own += mxfp4_tc_workspace_bytes(numel, hidden, ispp, E);
  const int64_t bs = mxfp4_bs_workspace_bytes(numel, hidden, ispp, E);      // the block-scaled path's, in the same place
  return total + (own > bs ? own : bs) + 256;
}

extern "C" int xkb_fused_moe_mxfp4(const void* A, int a_dtype, const uint8_t* w13,
                                   const uint8_t* w13_scale, const uint8_t* w2,
                                   const uint8_t* w2_scale, const int32_t* topk_ids,
                                   const float* topk_w, const void* b13, const void* b2,
                                   const int32_t* expert_map, int num_map, void* out, int64_t M,
                                   int64_t hidden, int64_t ispp, int E, int top_k, float swiglu_limit,
                                   int mul_routed_weight, int path, void* workspace,
                                   int64_t workspace_bytes, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  XKB_REQUIRE(a_dtype == XKB_BF16 || a_dtype == XKB_F32, "fused_moe_mxfp4: bad a_dtype %d", a_dtype);
  XKB_REQUIRE(M >= 0 && hidden >= 0 && ispp >= 0 && E >= 0 && top_k >= 0, "fused_moe_mxfp4: negative dim");
  XKB_REQUIRE(hidden % 32 == 0 && ispp % 32 == 0,
              "fused_moe_mxfp4: hidden and ispp must be multiples of the MX block 32 (got %lld, %lld)",
              (long long)hidden, (long long)ispp);
  XKB_REQUIRE(path == XKB_PATH_AUTO || path == XKB_PATH_SIMT || path == XKB_PATH_TC,
              "fused_moe_mxfp4: bad path %d", path);
  if (M == 0 || hidden == 0) return XKB_OK;
  XKB_REQUIRE(A && w13 && w13_scale && w2 && w2_scale && topk_ids && out,
              "fused_moe_mxfp4: null pointer argument");
  XKB_REQUIRE(topk_w || !mul_routed_weight, "fused_moe_mxfp4: topk_w is null");
  const int64_t need = xkb_fused_moe_mxfp4_workspace_bytes(M, hidden, ispp, E, top_k);
  if (workspace == nullptr || workspace_bytes < need)
    return fail(XKB_ERR_WORKSPACE, "fused_moe_mxfp4: workspace of %lld bytes needed, %lld given",
                (long long)need, (long long)workspace_bytes);
  XKB_REQUIRE(reinterpret_cast<uintptr_t>(workspace) % 256 == 0, "workspace must be 256-byte aligned");

  const int64_t numel = M * top_k;
  Carver carve(workspace);
  RoutingBuffers rb = carve_routing(carve, numel, E);
  void* bs_ws = carve.take<char>(0);
  float* scratch = carve.take<float>(numel * hidden);
  __nv_bfloat16* act = carve.take<__nv_bfloat16>(routing_max_pad(numel, E, kMaxBlock) * ispp);
  void* tc_ws = carve.take<char>(mxfp4_tc_workspace_bytes(numel, hidden, ispp, E));

  const bool tc_fit = mxfp4_tc_supported(a_dtype, M, hidden, ispp, E, top_k);
  if (path == XKB_PATH_TC && !tc_fit)
    return fail(XKB_ERR_ARG,
                "fused_moe_mxfp4: shape not supported by the tcgen05 path (needs bf16 A, "
                "hidden %% 512 == 0, ispp %% 512 == 0)");
  const bool use_tc = (path == XKB_PATH_TC) || (path == XKB_PATH_AUTO && tc_fit);
  const int bs_block = use_tc && mxfp4_bs_supported(w13, w2, w13_scale, w2_scale) ? mxfp4_bs_block(numel, E) : 0;
  const bool use_bs = bs_block > 0;
  const int block = use_bs ? bs_block : use_tc ? mxfp4_tc_block(numel, E) : kSimtBlock;

  Routing r;
  align::Job job;
  int rc = make_routing(rb, numel, E, block, &r);
  if (rc != XKB_OK) return rc;
  rc = route(rb, topk_ids, expert_map, num_map, E, top_k, use_tc ? hidden / 8 : 0, &r, &job, stream);
  if (rc != XKB_OK) return rc;
  if (use_bs) {
    const __nv_bfloat16* rows = nullptr;
    rc = launch_mxfp4_bs(A, w13, w13_scale, w2, w2_scale, b13, b2, r, hidden, ispp, E, top_k, swiglu_limit, bs_ws, rb.status,
                         &rows, stream);
    if (rc != XKB_OK) return rc;
    return launch_combine_bf16(rows, mul_routed_weight ? topk_w : nullptr, topk_ids, expert_map, num_map, E, out,
                               a_dtype, M, top_k, hidden, stream);
  }
  if (use_tc) {
    __nv_bfloat16* rows = reinterpret_cast<__nv_bfloat16*>(scratch);
    const int check_scale = numel > 48 * (int64_t)E;   // these batches report scale bytes 191..254, as they always have
    rc = launch_mxfp4_tc(A, w13, w13_scale, w2, w2_scale, b13, b2, r, act, rows, hidden, ispp, E, top_k, swiglu_limit,
                         check_scale, tc_ws, rb.status, stream);
    if (rc != XKB_OK) return rc;
    return launch_combine_bf16(rows, mul_routed_weight ? topk_w : nullptr, topk_ids, expert_map, num_map, E, out,
                               a_dtype, M, top_k, hidden, stream);
  }
  rc = launch_mxfp4_simt(A, a_dtype, w13, w13_scale, w2, w2_scale, b13, b2, r, topk_w, act, scratch,
                         hidden, ispp, top_k, swiglu_limit, mul_routed_weight, stream);
  if (rc != XKB_OK) return rc;
  return launch_combine(scratch, topk_ids, expert_map, num_map, E, out, a_dtype, M, top_k, hidden, stream);
}

// ---------------------------------------------------------------------------
extern "C" int xkb_workspace_status(const void* workspace, void* stream_) {
  XKB_REQUIRE(workspace != nullptr, "xkb_workspace_status: null workspace");
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  int host = 0;
  XKB_CHECK_CUDA(cudaMemcpyAsync(&host, workspace, sizeof(int), cudaMemcpyDeviceToHost, stream));
  XKB_CHECK_CUDA(cudaStreamSynchronize(stream));
  if (host == 2)
    return fail(XKB_ERR_DEVICE, "an MXFP4 scale byte in 191..254 (weights of 2^64 and more), which batches of more than 48 "
                                "slots per expert do not take: status 0x2");
  if ((host & 0xFF) == 3)
    return fail(XKB_ERR_DEVICE, "a kernel read a routing value outside what the routing buffers hold and skipped the "
                                "work: status 0x%x (site %d)", host, host >> 8);
  if (host != 0)
    return fail(XKB_ERR_DEVICE, "a kernel gave up a bounded wait: status 0x%x (wait site %d)", host, host >> 8);
  return XKB_OK;
}

// ---------------------------------------------------------------------------
extern "C" int xkb_gemm_timer_enable(int max_calls) {
  XKB_REQUIRE(max_calls >= 0 && max_calls <= (1 << 16), "xkb_gemm_timer_enable: max_calls out of range");
  for (auto e : g_timer.start) cudaEventDestroy(e);
  for (auto e : g_timer.stop) cudaEventDestroy(e);
  g_timer.start.clear();
  g_timer.stop.clear();
  g_timer.used = 0;
  g_timer.enabled = max_calls > 0;
  for (int i = 0; i < max_calls; ++i) {
    cudaEvent_t a, b;
    XKB_CHECK_CUDA(cudaEventCreate(&a));
    XKB_CHECK_CUDA(cudaEventCreate(&b));
    g_timer.start.push_back(a);
    g_timer.stop.push_back(b);
  }
  return XKB_OK;
}

extern "C" int xkb_gemm_timer_read(float* ms_host, int capacity, int* count_host) {
  XKB_REQUIRE(ms_host != nullptr && count_host != nullptr, "xkb_gemm_timer_read: null output");
  const int n = g_timer.used < capacity ? g_timer.used : capacity;
  for (int i = 0; i < n; ++i) {
    XKB_CHECK_CUDA(cudaEventSynchronize(g_timer.stop[i]));
    XKB_CHECK_CUDA(cudaEventElapsedTime(&ms_host[i], g_timer.start[i], g_timer.stop[i]));
  }
  *count_host = n;
  g_timer.used = 0;
  return XKB_OK;
}
