// MoE router: softmax over the experts, top-k, optional renormalisation (sm_100a).
//
// Contract (src/xkernels/ops/moe/topk_softmax.py:33-95 in the reference): logits are upcast to
// fp32, softmax runs over ALL experts, then the k largest probabilities are taken in DESCENDING
// probability with ties broken by ASCENDING expert id (a stable descending argsort), then the
// selected weights are optionally divided by their sum.  Equal logits give equal probabilities
// here as there, so the tie rule decides the same way.
//
// One warp per token row: lane l holds experts l, l + 32, ...; row maximum and sum by shuffles.
//
// Bound by the warp's instructions, not by memory (a row of 256 bf16 logits is 512 bytes).  k rounds of
// "best of my lane, then best of the warp" over all experts cost about 900 instructions per row, so the
// selection first cuts the row down to a handful of candidates: the k-th largest of the 32 lane maxima
// bounds the k-th largest element from below, usually 8 to 16 of the experts reach it, and only those
// are divided by the sum (one per lane), ranked against each other and written.  Rows that leave more
// than 32 candidates (long runs of equal logits, a k-th probability near the subnormals), a top-k above 32
// or a sum that is not finite take the rounds (select_by_rounds), which order every probability of the row.  They
// pay for the candidates first, and make that good with two warp reductions a round instead of ten shuffles (all
// logits equal, E=256, top 8, fp32, M=16384: 28.1 us before there were candidates, 32.1 with shuffles, 25.9 now).
// M=16384, E=256, bf16, top 8, renormalised: 28.7 -> 11.8 us on the device, 12.3 us a call.
#include <cuda_fp16.h>

#include "common.cuh"

namespace xkb {
namespace {

constexpr int kMaxPerLane = 32;               // experts per lane -> at most 1024 experts
constexpr int kWarpsPerBlock = 8;
// Up to this top-k the candidates of rows of independent logits fit 32 lanes (74-100 % of the rows at 20, E = 48 to
// 1024; 31-99 % at 22; 5-85 % at 24); above, looking for them mostly comes on top of the rounds (top 32 of 1024
// experts, M=16384: 227 us without, 231 with).  Up to 32 experts they fit in any case.
constexpr int kShortTopk = 20;

template <typename T> __device__ __forceinline__ float load_logit(const T* p);
template <> __device__ __forceinline__ float load_logit<float>(const float* p) { return *p; }
template <> __device__ __forceinline__ float load_logit<__nv_bfloat16>(const __nv_bfloat16* p) {
  return __bfloat162float(*p);
}
template <> __device__ __forceinline__ float load_logit<__half>(const __half* p) { return __half2float(*p); }

// (probability, id) ordering of the contract: larger probability first, then smaller id
__device__ __forceinline__ bool better(float pa, int ia, float pb, int ib) {
  return pa > pb || (pa == pb && ia < ib);
}

// k rounds over the whole row: p[t] = probability of expert lane + 32 t, or -1 where there is none.
template <int PER_LANE>
__device__ __forceinline__ void select_by_rounds(float (&p)[PER_LANE], int64_t row, int lane, int topk, int renormalize,
                                              float* __restrict__ topk_w, int32_t* __restrict__ topk_ids) {
  float wsum = 0.f;
  float my_w = 0.f;     // lane j keeps the j-th selected weight (j < 32), further ones go out directly
  for (int j = 0; j < topk; ++j) {
    float bp = -1.f;
    int bi = 0x7fffffff;
#pragma unroll
    for (int t = 0; t < PER_LANE; ++t) {
      const int e = lane + 32 * t;
      if (better(p[t], e, bp, bi)) { bp = p[t]; bi = e; }
    }
    // best of the warp: bp is -1 or >= 0 and never NaN (better() is false for one), so its bits order as signed integers
    const int top = __reduce_max_sync(0xffffffffu, __float_as_int(bp));
    bi = __reduce_min_sync(0xffffffffu, __float_as_int(bp) == top ? bi : 0x7fffffff);
    bp = __int_as_float(top);
    // every lane now holds the same winner; its owner retires it
    if ((bi & 31) == lane) {
#pragma unroll
      for (int t = 0; t < PER_LANE; ++t)
        if (t == (bi >> 5)) p[t] = -1.f;
    }
    wsum += bp;
    if (lane == 0) topk_ids[row * topk + j] = bi;
    if (renormalize) {
      if (j < 32) { if (lane == j) my_w = bp; }
      else if (lane == 0) topk_w[row * topk + j] = bp;   // divided below
    } else if (lane == 0) {
      topk_w[row * topk + j] = bp;
    }
  }
  if (renormalize) {
    if (lane < topk) topk_w[row * topk + lane] = my_w / wsum;
    if (lane == 0)
      for (int j = 32; j < topk; ++j) topk_w[row * topk + j] = topk_w[row * topk + j] / wsum;
  }
}

template <typename T, int PER_LANE>
__global__ void __launch_bounds__(32 * kWarpsPerBlock)
topk_softmax_kernel(const T* __restrict__ gating, float* __restrict__ topk_w, int32_t* __restrict__ topk_ids,
                    int64_t M, int E, int topk, int renormalize) {
  __shared__ uint64_t s_cand[kWarpsPerBlock][32];   // candidates, then their sort keys
  __shared__ float s_w[kWarpsPerBlock][32];         // the selected weights in order
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t row = (int64_t)blockIdx.x * kWarpsPerBlock + warp;
  if (row >= M) return;
  const T* x = gating + row * E;

  float p[PER_LANE];
  float mx = -INFINITY;
#pragma unroll
  for (int t = 0; t < PER_LANE; ++t) {
    const int e = lane + 32 * t;
    p[t] = e < E ? load_logit<T>(x + e) : -INFINITY;
    mx = fmaxf(mx, p[t]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  float sum = 0.f;
  float lane_max = -1.f;
#pragma unroll
  for (int t = 0; t < PER_LANE; ++t) {
    const int e = lane + 32 * t;
    p[t] = e < E ? expf(p[t] - mx) : 0.f;
    sum += p[t];
    p[t] = e < E ? p[t] : -1.f;    // -1 marks "not a candidate" (exponentials are >= 0)
    lane_max = fmaxf(lane_max, p[t]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);

  // The k-th largest lane maximum (equal ones leave together, so it may be a smaller one: still a bound).
  // The floats are >= 0 or -1, and as signed integers they order the same way.
  int tau = -1, lm = __float_as_int(lane_max);
  const bool short_way = topk <= (PER_LANE == 1 ? 32 : kShortTopk) && sum < INFINITY;   // (a NaN sum fails the comparison)
  if (short_way) {
    for (int j = 0; j < topk; ++j) {
      tau = __reduce_max_sync(0xffffffffu, lm);
      if (lm == tau) lm = __float_as_int(-1.f);
    }
  }
  // Division by the sum is monotone but may round neighbours to one probability, and then the smaller id
  // wins: exponentials a few units in the last place below the bound are candidates as well.  That slack
  // covers the rounding of normal quotients only.  Subnormal ones merge exponentials that lie far apart (at
  // 27 and 28 * 2^-149 and a sum of 2 both are 14 * 2^-149, and below half a unit everything is 0), so with
  // a bound whose quotient comes near the subnormals every expert is a candidate.
  float bound = -1.f;
  if (short_way && tau >= 0 && __int_as_float(tau) >= sum * 7.8886090522101181e-31f)   // 2^-100
    bound = __int_as_float(tau) * (1.f - 9.5367431640625e-7f);
  int n = 0;
  uint64_t* cand = s_cand[warp];
#pragma unroll
  for (int t = 0; t < PER_LANE; ++t) {
    const bool c = p[t] >= bound && p[t] >= 0.f;
    const unsigned who = __ballot_sync(0xffffffffu, c);
    const int at = n + __popc(who & ((1u << lane) - 1u));
    if (c && at < 32) cand[at] = ((uint64_t)__float_as_uint(p[t]) << 32) | (uint32_t)(lane + 32 * t);
    n += __popc(who);
  }
  if (!short_way || n > 32) {
#pragma unroll
    for (int t = 0; t < PER_LANE; ++t) p[t] = lane + 32 * t < E ? p[t] / sum : -1.f;
    select_by_rounds<PER_LANE>(p, row, lane, topk, renormalize, topk_w, topk_ids);
    return;
  }
  // one candidate per lane: probability, then a key whose larger value is the better one
  __syncwarp();
  float prob = -1.f;
  uint64_t key = 0;
  if (lane < n) {
    const uint64_t v = cand[lane];
    prob = __uint_as_float((uint32_t)(v >> 32)) / sum;
    key = ((uint64_t)__float_as_uint(prob) << 32) | (uint32_t)~(uint32_t)v;
  }
  __syncwarp();
  cand[lane] = key;
  __syncwarp();
  int rank = 0;
  for (int j = 0; j < n; ++j) rank += cand[j] > key ? 1 : 0;
  const bool selected = lane < n && rank < topk;   // keys differ in the id: ranks 0 .. topk - 1 are all taken
  float wsum = 1.f;
  if (renormalize) {
    if (selected) s_w[warp][rank] = prob;
    __syncwarp();
    wsum = 0.f;
    for (int j = 0; j < topk; ++j) wsum += s_w[warp][j];
  }
  if (selected) {
    topk_ids[row * topk + rank] = (int32_t)~(uint32_t)key;
    topk_w[row * topk + rank] = renormalize ? prob / wsum : prob;
  }
}

template <typename T>
int launch_for_type(const void* gating, float* w, int32_t* ids, int64_t M, int E, int topk, int renorm,
                    cudaStream_t s) {
  const unsigned blocks = (unsigned)ceil_div(M, (int64_t)kWarpsPerBlock);
  const T* g = static_cast<const T*>(gating);
  const int per_lane = (E + 31) / 32;
#define XKB_TS_CASE(PL)                                                                                  \
  if (per_lane <= PL) {                                                                                  \
    topk_softmax_kernel<T, PL><<<blocks, 32 * kWarpsPerBlock, 0, s>>>(g, w, ids, M, E, topk, renorm);  \
    XKB_CHECK_LAUNCH("topk_softmax_kernel");                                                             \
    return XKB_OK;                                                                                       \
  }
  XKB_TS_CASE(1)
  XKB_TS_CASE(2)
  XKB_TS_CASE(4)
  XKB_TS_CASE(8)
  XKB_TS_CASE(16)
  XKB_TS_CASE(32)
#undef XKB_TS_CASE
  return fail(XKB_ERR_ARG, "topk_softmax: E=%d exceeds %d experts", E, 32 * kMaxPerLane);
}

}  // namespace
}  // namespace xkb

extern "C" int xkb_topk_softmax(const void* gating_output, int dtype, float* topk_weights, int32_t* topk_ids,
                                int64_t M, int E, int topk, int renormalize, void* stream) {
  using namespace xkb;
  XKB_REQUIRE(M >= 0 && E >= 1, "topk_softmax: bad shape M=%lld E=%d", (long long)M, E);
  XKB_REQUIRE(topk >= 1 && topk <= E, "topk_softmax: topk must satisfy 1 <= topk <= E (got topk=%d, E=%d)", topk, E);
  XKB_REQUIRE(E <= 32 * kMaxPerLane, "topk_softmax: E=%d exceeds %d experts", E, 32 * kMaxPerLane);
  if (M == 0) return XKB_OK;
  XKB_REQUIRE(gating_output != nullptr && topk_weights != nullptr && topk_ids != nullptr,
              "topk_softmax: null pointer");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case XKB_BF16: return launch_for_type<__nv_bfloat16>(gating_output, topk_weights, topk_ids, M, E, topk, renormalize, s);
    case XKB_F32: return launch_for_type<float>(gating_output, topk_weights, topk_ids, M, E, topk, renormalize, s);
    case XKB_F16: return launch_for_type<__half>(gating_output, topk_weights, topk_ids, M, E, topk, renormalize, s);
    default: return fail(XKB_ERR_ARG, "topk_softmax: unsupported logits dtype code %d", dtype);
  }
}
