// Launchers of the grouped expert GEMM kernels (SIMT and tcgen05 paths).
#pragma once
#include "common.cuh"

namespace xkb {

constexpr int kSimtBlock = 16;  // align block the SIMT kernels consume

// ---- activation gathers: one thread per 8 elements, blocks of one token or a piece of one ----
constexpr int kGatherThreads = 256;
struct GatherGrid { unsigned pieces, units, threads, blocks; };   // pieces of `units` 8-element units per token
// sorting: blocks of 1024 threads that sort the routing first; few tokens are cut finer, over sixteen SMs
inline int gather_grid(int64_t M, int64_t units, bool sorting, GatherGrid* g) {
  int64_t p = ceil_div(units, sorting ? 1024 : kGatherThreads);
  if (sorting && p * M < 16) p = ceil_div(16, M) < ceil_div(units, 32) ? ceil_div(16, M) : ceil_div(units, 32);
  XKB_REQUIRE(p * M <= 0x7fffffff, "activation gather: %lld blocks do not fit a grid", (long long)(p * M));
  g->pieces = (unsigned)p;
  g->units = (unsigned)align_up(ceil_div(units, p), 32);
  g->threads = sorting ? 1024u : g->units;
  g->blocks = (unsigned)(p * M);
  return XKB_OK;
}

// going through the sorted positions instead: sixteen blocks per SM at most, each takes positions in turn
inline unsigned position_blocks(int64_t max_pad) { return (unsigned)(max_pad < 148 * 16 ? max_pad : 148 * 16); }

// ---- generic SIMT path (moe_simt.cu) ---------------------------------------
int launch_int4_simt(const void* A, int a_dtype, const int32_t* packed, const void* scale,
                     const Routing& r, const float* topk_w, float* scratch, int64_t N, int64_t K,
                     int top_k, int group, int mul_w, cudaStream_t stream, int round_out = 0);
int launch_mxfp4_simt(const void* A, int a_dtype, const uint8_t* w13, const uint8_t* w13_scale,
                      const uint8_t* w2, const uint8_t* w2_scale, const void* b13, const void* b2,
                      const Routing& r, const float* topk_w, __nv_bfloat16* act, float* scratch,
                      int64_t hidden, int64_t ispp, int top_k, float limit, int mul_w,
                      cudaStream_t stream);

constexpr int kErrBadRouting = 3;   // status code: a routing value read by a kernel was outside what the buffers can hold

// ---- tcgen05 path (moe_tc.cu) ----------------------------------------------
bool int4_tc_supported(int a_dtype, int64_t M, int64_t N, int64_t K, int E, int top_k, int group);
int int4_tc_block(int64_t numel, int E, int top_k);
int64_t int4_tc_workspace_bytes(int64_t numel, int64_t N, int64_t K, int E);
int launch_int4_tc(const void* A, const int32_t* packed, const void* scale, const Routing& r,
                   const float* topk_w, float* scratch, int64_t N, int64_t K, int E, int top_k, int group,
                   int mul_w, void* tc_ws, int* status, cudaStream_t stream);

// INT4 two-GEMM expert layer (gate_up + SwiGLU, then down with bf16-rounded weighted slot rows)
bool int4_ffn_tc_supported(int a_dtype, int64_t M, int64_t hidden, int64_t inter, int E, int top_k, int group);
int launch_int4_ffn_tc(const void* A, const int32_t* w13, const void* s13, const int32_t* w2, const void* s2,
                       const Routing& r, const float* topk_w, __nv_bfloat16* act, __nv_bfloat16* rows16, int64_t hidden,
                       int64_t inter, int E, int top_k, int group, float limit, void* tc_ws, int* status,
                       cudaStream_t stream);
int launch_int4_ffn_simt(const void* A, int a_dtype, const int32_t* w13, const void* s13, const int32_t* w2,
                         const void* s2, const Routing& r, const int32_t* topk_ids, const int32_t* expert_map,
                         int num_map, int E, const float* topk_w, float* rows1, void* act, float* scratch,
                         int64_t hidden, int64_t inter, int top_k, int group, float limit, cudaStream_t stream);

// MXFP4 on the block-scaled instructions (moe_mx.cu): the shapes of mxfp4_tc_supported, 32-byte aligned weights, and
// batches for which mxfp4_bs_block gives a token tile (0: too many slots per expert).
// Leaves the bf16 rows of the slots, before the routing weight, in the workspace (*rows).
bool mxfp4_bs_supported(const void* w13, const void* w2, const void* s13, const void* s2);
int mxfp4_bs_block(int64_t numel, int E);
int64_t mxfp4_bs_workspace_bytes(int64_t numel, int64_t hidden, int64_t ispp, int E);
int launch_mxfp4_bs(const void* A, const uint8_t* w13, const uint8_t* w13_scale, const uint8_t* w2,
                    const uint8_t* w2_scale, const void* b13, const void* b2, const Routing& r, int64_t hidden,
                    int64_t ispp, int E, int top_k, float limit, void* ws, int* status, const __nv_bfloat16** rows,
                    cudaStream_t stream);

bool mxfp4_tc_supported(int a_dtype, int64_t M, int64_t hidden, int64_t ispp, int E, int top_k);
int mxfp4_tc_block(int64_t numel, int E);
int64_t mxfp4_tc_workspace_bytes(int64_t numel, int64_t hidden, int64_t ispp, int E);
int launch_mxfp4_tc(const void* A, const uint8_t* w13, const uint8_t* w13_scale, const uint8_t* w2,
                    const uint8_t* w2_scale, const void* b13, const void* b2, const Routing& r,
                    __nv_bfloat16* act, __nv_bfloat16* rows16, int64_t hidden, int64_t ispp, int E, int top_k,
                    float limit, int check_scale, void* tc_ws, int* status, cudaStream_t stream);   // rows before the routing weight, in bf16

}  // namespace xkb
