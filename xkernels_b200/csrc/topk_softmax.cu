// MoE router: softmax over the experts, top-k, optional renormalisation (sm_100a).
//
// Contract (src/xkernels/ops/moe/topk_softmax.py:33-95 in the reference): logits are upcast to
// fp32, softmax runs over ALL experts, then the k largest probabilities are taken in DESCENDING
// probability with ties broken by ASCENDING expert id (a stable descending argsort), then the
// selected weights are optionally divided by their sum.  Equal logits give equal probabilities
// here as there, so the tie rule decides the same way.
//
// One warp per token row: lane l holds the PER_LANE experts from l * PER_LANE on, read with as few loads as their
// alignment allows; row maximum by one warp reduction, sum by shuffles.
//
// Bound by the warp's instructions, not by memory (a row of 256 bf16 logits is 512 bytes).  k rounds of
// "best of my lane, then best of the warp" over all experts cost about 900 instructions per row, so the
// selection first cuts the row down to a handful of candidates: the k-th largest of the 32 lane maxima
// bounds the k-th largest element from below, usually 8 to 16 of the experts reach it, and only those
// are divided by the sum (one per lane), ranked against each other and written.  They are collected by ascending id
// (a lane's experts are neighbours), so a rank is a count of larger probabilities and of equal ones in lower lanes.
// Rows that leave more than 32 candidates (long runs of equal logits, a k-th probability near the subnormals), a top-k
// above 32 or a sum that is not finite take the rounds (select_by_rounds), which order every probability of the row.
// They pay for the candidates first, and make that good with two warp reductions a round instead of ten shuffles.
// M=16384, E=256, bf16, top 8, renormalised: 28.7 us with the rounds, 10.8 with strided loads of one
// logit, branches around the candidates' stores and a loop over all of them, 9.2 now (460 instructions a row).
#include <cuda_fp16.h>

#include "common.cuh"

namespace xkb {
namespace {

constexpr int kMaxPerLane = 32;               // experts per lane -> at most 1024 experts
constexpr int kWarpsPerBlock = 8;
// Up to this top-k the candidates of rows of independent logits fit 32 lanes (74-100 % of the rows at 20, E = 48 to
// 1024; 31-99 % at 22; 5-85 % at 24); above, looking for them mostly comes on top of the rounds (top 32 of 1024
// experts, M=16384: 227 us without, 231 with, in the form with strided logits).  Up to 32 experts they fit in any case.
constexpr int kShortTopk = 20;

template <typename T> __device__ __forceinline__ float load_logit(const T* p);
template <> __device__ __forceinline__ float load_logit<float>(const float* p) { return *p; }
template <> __device__ __forceinline__ float load_logit<__nv_bfloat16>(const __nv_bfloat16* p) {
  return __bfloat162float(*p);
}
template <> __device__ __forceinline__ float load_logit<__half>(const __half* p) { return __half2float(*p); }

// k rounds over the whole row: p[t] = probability of expert lane * PER_LANE + t, or -1 where there is none.
template <int PER_LANE>
__device__ __forceinline__ void select_by_rounds(float (&p)[PER_LANE], int64_t row, int lane, int topk, int renormalize,
                                              float* __restrict__ topk_w, int32_t* __restrict__ topk_ids) {
  float wsum = 0.f;
  float my_w = 0.f;     // lane j keeps the j-th selected weight (j < 32), further ones go out directly
  for (int j = 0; j < topk; ++j) {
    float bp = -1.f;
    int bt = 0;
#pragma unroll
    for (int t = 0; t < PER_LANE; ++t)   // a lane's ids ascend: the first of equal ones stays
      if (p[t] > bp) { bp = p[t]; bt = t; }
    int bi = bp >= 0.f ? lane * PER_LANE + bt : 0x7fffffff;
    // best of the warp: bp is -1 or >= 0 and never NaN (no comparison with one holds), so its bits order as signed integers
    const int top = __reduce_max_sync(0xffffffffu, __float_as_int(bp));
    bi = __reduce_min_sync(0xffffffffu, __float_as_int(bp) == top ? bi : 0x7fffffff);
    bp = __int_as_float(top);
    // every lane now holds the same winner; its owner retires it
    // (bi of no expert: every remaining probability is NaN, and nothing is retired)
#pragma unroll
    for (int t = 0; t < PER_LANE; ++t)
      if (t == bi - lane * PER_LANE) p[t] = -1.f;
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

// The largest of the warp's values that are not NaN (-inf if all are).
__device__ __forceinline__ float warp_max(float v) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// PER_LANE neighbouring logits.  VEC: E is a multiple of PER_LANE and every lane's first one lies on a VEC-byte boundary.
template <typename T, int PER_LANE, int VEC>
__device__ __forceinline__ void load_lane(const T* row, int lane, int E, float (&v)[PER_LANE]) {
  if constexpr (VEC == 0) {
#pragma unroll
    for (int t = 0; t < PER_LANE; ++t) v[t] = lane * PER_LANE + t < E ? load_logit<T>(row + lane * PER_LANE + t) : -INFINITY;
  } else {
    constexpr int kPer = VEC / (int)sizeof(T);
    struct alignas(VEC) Chunk { T x[kPer]; };
#pragma unroll
    for (int c = 0; c < PER_LANE / kPer; ++c) {
      Chunk q;
      if (lane * PER_LANE < E) q = reinterpret_cast<const Chunk*>(row + lane * PER_LANE)[c];
#pragma unroll
      for (int i = 0; i < kPer; ++i) v[c * kPer + i] = lane * PER_LANE < E ? load_logit<T>(&q.x[i]) : -INFINITY;
    }
  }
}

template <typename T, int PER_LANE, int VEC>
__global__ void __launch_bounds__(32 * kWarpsPerBlock)
topk_softmax_kernel(const T* __restrict__ gating, float* __restrict__ topk_w, int32_t* __restrict__ topk_ids,
                    int64_t M, int E, int topk, int renormalize) {
  __shared__ uint2 s_cand[kWarpsPerBlock][32];   // candidates by ascending id: exponential, id
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t row = (int64_t)blockIdx.x * kWarpsPerBlock + warp;
  if (row >= M) return;

  float p[PER_LANE];
  load_lane<T, PER_LANE, VEC>(gating + row * E, lane, E, p);
  // a lane's experts are all in the row or none is (VEC), or one by one
  const bool in_row = VEC == 0 || lane * PER_LANE < E;
  auto valid = [&](int t) -> bool { return VEC != 0 || lane * PER_LANE + t < E; };
  float mx = p[0];
#pragma unroll
  for (int t = 1; t < PER_LANE; ++t) mx = fmaxf(mx, p[t]);
  mx = warp_max(mx);
  float sum = 0.f, lane_max = -1.f;
#pragma unroll
  for (int t = 0; t < PER_LANE; ++t) {
    p[t] = valid(t) ? expf(p[t] - mx) : -1.f;    // -1 marks "not a candidate" (exponentials are >= 0)
    sum += valid(t) ? p[t] : 0.f;
    lane_max = fmaxf(lane_max, p[t]);
  }
  sum = warp_sum(in_row ? sum : 0.f);

  // The k-th largest lane maximum (equal ones leave together, so it may be a smaller one: still a bound).
  float tau = -1.f, lm = in_row ? lane_max : -1.f;
  const bool short_way = topk <= (PER_LANE == 1 ? 32 : kShortTopk) && sum < INFINITY;   // (a NaN sum fails the comparison)
  if (short_way) {
    int j = topk;
    for (; j >= 4; j -= 4) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        tau = warp_max(lm);
        if (lm == tau) lm = -1.f;
      }
    }
    for (; j > 0; --j) {
      tau = warp_max(lm);
      if (lm == tau) lm = -1.f;
    }
  }
  // Division by the sum is monotone but may round neighbours to one probability, and then the smaller id
  // wins: exponentials a few units in the last place below the bound are candidates as well.  That slack
  // covers the rounding of normal quotients only.  Subnormal ones merge exponentials that lie far apart (at
  // 27 and 28 * 2^-149 and a sum of 2 both are 14 * 2^-149, and below half a unit everything is 0), so with
  // a bound whose quotient comes near the subnormals every expert is a candidate.
  float bound = 0.f;
  if (short_way && tau >= 0.f && tau >= sum * 7.8886090522101181e-31f)   // 2^-100
    bound = tau * (1.f - 9.5367431640625e-7f);
  int mine = 0;
#pragma unroll
  for (int t = 0; t < PER_LANE; ++t) mine += p[t] >= bound ? 1 : 0;
  if (!in_row) mine = 0;
  int at = mine;   // inclusive sum over the lanes
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int below = __shfl_up_sync(0xffffffffu, at, d);
    if (lane >= d) at += below;
  }
  const int n = __shfl_sync(0xffffffffu, at, 31);
  if (!short_way || n > 32) {
#pragma unroll
    for (int t = 0; t < PER_LANE; ++t) p[t] = in_row && valid(t) ? p[t] / sum : -1.f;
    select_by_rounds<PER_LANE>(p, row, lane, topk, renormalize, topk_w, topk_ids);
    return;
  }
  uint2* cand = s_cand[warp];
  uint32_t to = (uint32_t)__cvta_generic_to_shared(cand + (at - mine));
  const float low = in_row ? bound : INFINITY;
#pragma unroll
  for (int t = 0; t < PER_LANE; ++t)   // predicated: a branch each took twice as many instructions
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ge.f32 q, %1, %2;\n\t@q st.shared.v2.b32 [%0], {%3, %4};\n\t@q add.u32 %0, %0, 8;\n\t}"
                 : "+r"(to) : "f"(p[t]), "f"(low), "r"(__float_as_uint(p[t])), "r"(lane * PER_LANE + t) : "memory");
  __syncwarp();
  // one candidate per lane
  float prob = -1.f;
  int id = 0;
  if (lane < n) {
    const uint2 c = cand[lane];
    prob = __uint_as_float(c.x) / sum;
    id = (int)c.y;
  }
  int rank = __popc(__match_any_sync(0xffffffffu, __float_as_uint(prob)) & ((1u << lane) - 1u));
#pragma unroll
  for (int j = 0; j < 16; ++j) rank += __shfl_sync(0xffffffffu, prob, j) > prob ? 1 : 0;   // (lanes from n on hold -1)
  if (n > 16) {
#pragma unroll
    for (int j = 16; j < 32; ++j) rank += __shfl_sync(0xffffffffu, prob, j) > prob ? 1 : 0;
  }
  const bool selected = lane < n && rank < topk;   // the ranks are all different: 0 .. topk - 1 are taken
  float wsum = 1.f;
  if (renormalize) wsum = warp_sum(selected ? prob : 0.f);
  if (selected) {
    topk_ids[row * topk + rank] = id;
    topk_w[row * topk + rank] = renormalize ? prob / wsum : prob;
  }
}

// the widest load of 16 bytes or less that a lane's `bytes` are a multiple of (at least two logits), 0: one by one
constexpr int lane_vec(int bytes) { return bytes % 16 == 0 ? 16 : bytes % 8 == 0 ? 8 : bytes == 4 ? 4 : 0; }

template <typename T>
int launch_for_type(const void* gating, float* w, int32_t* ids, int64_t M, int E, int topk, int renorm,
                    cudaStream_t s) {
  const unsigned blocks = (unsigned)ceil_div(M, (int64_t)kWarpsPerBlock);
  const T* g = static_cast<const T*>(gating);
  // neighbours per lane: the fewest that cover the row.  Loads of up to 16 bytes where every lane's first logit lies
  // on them, of one logit otherwise.
  const int per_lane = (E + 31) / 32;
  const uintptr_t odd = reinterpret_cast<uintptr_t>(gating) | (uintptr_t)(E * (int64_t)sizeof(T));
#define XKB_TS_CASE(PL)                                                                                  \
  if (per_lane <= PL) {                                                                                  \
    constexpr int kVec = lane_vec(PL * (int)sizeof(T));                                                  \
    const bool vec = kVec > 0 && E % PL == 0 && odd % (kVec > 0 ? kVec : 1) == 0;                                     \
    (vec ? topk_softmax_kernel<T, PL, kVec> : topk_softmax_kernel<T, PL, 0>)<<<blocks, 32 * kWarpsPerBlock, 0, s>>>( \
        g, w, ids, M, E, topk, renorm);                                                                  \
    XKB_CHECK_LAUNCH("topk_softmax_kernel");                                                             \
    return XKB_OK;                                                                                       \
  }
  XKB_TS_CASE(1)
  XKB_TS_CASE(2)
  XKB_TS_CASE(4)
  XKB_TS_CASE(8)
  XKB_TS_CASE(12)
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
