// MoE router: softmax over the experts, top-k, optional renormalisation (sm_100a).
//
// Contract (src/xkernels/ops/moe/topk_softmax.py:33-95 in the reference): logits are upcast to
// fp32, softmax runs over ALL experts, then the k largest probabilities are taken in DESCENDING
// probability with ties broken by ASCENDING expert id (a stable descending argsort), then the
// selected weights are optionally divided by their sum.  Equal logits give equal probabilities
// here as there, so the tie rule decides the same way.
//
// One warp per token row.  A row is dealt to the lanes in pieces of P neighbouring experts, piece i to lane i % 32, one
// load a piece; row maximum by one warp reduction, sum by shuffles.
//
// Bound by the warp's instructions, not by memory (a row of 256 bf16 logits is 512 bytes).  k rounds of
// "best of my lane, then best of the warp" over all experts cost about 900 instructions per row, so the
// selection first cuts the row down to a handful of candidates: the k-th largest of the 32 lane maxima
// bounds the k-th largest element from below, usually 8 to 16 of the experts reach it, and only those
// are divided by the sum (one per lane), ranked against each other and written.  They are collected by ascending id
// (piece by piece), so a rank is a count of larger probabilities and of equal ones in lower lanes.
// Rows that leave more than 32 candidates (long runs of equal logits, a k-th probability near the subnormals), a top-k
// above 32 or a sum that is not finite take the rounds (select_by_rounds), which order every probability of the row.
// They pay for the candidates first, and make that good with two warp reductions a round instead of ten shuffles.
// Why small pieces in turn: rows whose live logits are neighbours (routers that mask all groups of experts but a few) have
// to spread them over the lanes, or few lanes carry maxima, the bound gets loose and the row takes the rounds.
// M=16384, E=256, bf16, top 8, renormalised, on the device: 28.7 us with the rounds; 10.9 with single logits dealt to the lanes
// and a loop over all candidates; 9.3 with eight neighbours a lane, but 28.3, 17.1 and 9.6 where one, two and four groups of 32
// are live, 22.1 for sorted rows; 9.2 with pieces of two, and 9.3, 9.4, 9.5 and 9.5 for those rows.  (E=1024, where the
// rounds are common, a call in a loop: top 8 34.4 / 22.9 / 20.8, top 20 158 / 106 / 109, top 32 227 / 166 / 168; all logits
// equal, top 8 - / 55.4 / 57.5.)
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

// The id of a lane's t-th expert is lane * P plus this; a lane's ids ascend with t.
template <int P> struct Deal { static __device__ __forceinline__ constexpr int at(int t) { return t / P * 32 * P + t % P; } };

// k rounds over the whole row: p[t] = probability of the lane's t-th expert, 0 behind the row.
template <int PER_LANE, int P>
__device__ __forceinline__ void select_by_rounds(float (&p)[PER_LANE], int64_t row, int lane, int topk, int renormalize,
                                              float* __restrict__ topk_w, int32_t* __restrict__ topk_ids) {
  float rest = 0.f;     // every lane's share of the sum of further ones (600 weights added one by one were off by 2.2e-6 of it)
  float my_w = 0.f;     // lane j keeps the j-th selected weight (j < 32), further ones go out directly
  for (int j = 0; j < topk; ++j) {
    float bp = -1.f;
    int bt = 0;
    // a lane's ids ascend: the first of equal ones stays.  (Many experts: the maximum first, which takes half the instructions of
    // carrying the id along.  M=16384, top 32 of 1024: 178 -> 168 us; top 24 of 128: 35 -> 40, so not there.)
    if constexpr (PER_LANE >= 8) {
#pragma unroll
      for (int t = 0; t < PER_LANE; ++t) bp = fmaxf(bp, p[t]);
#pragma unroll
      for (int t = PER_LANE - 1; t >= 0; --t)
        if (p[t] == bp) bt = Deal<P>::at(t);
    } else {
#pragma unroll
      for (int t = 0; t < PER_LANE; ++t)
        if (p[t] > bp) { bp = p[t]; bt = Deal<P>::at(t); }
    }
    const int mine = bp >= 0.f ? lane * P + bt : 0x7fffffff;
    // best of the warp: bp is -1 or >= 0 and never NaN (no comparison with one holds), so its bits order as signed integers
    const int top = __reduce_max_sync(0xffffffffu, __float_as_int(bp));
    const int bi = __reduce_min_sync(0xffffffffu, __float_as_int(bp) == top ? mine : 0x7fffffff);
    bp = __int_as_float(top);
    // every lane now holds the same winner; its owner retires it
    // (bi of no expert: every remaining probability is NaN, and nothing is retired)
#pragma unroll
    for (int t = 0; t < PER_LANE; ++t)
      if (Deal<P>::at(t) == bi - lane * P) p[t] = -1.f;
    if (lane == 0) topk_ids[row * topk + j] = bi;
    if (renormalize) {
      if (j < 32) {
        if (lane == j) my_w = bp;
      } else {
        if (lane == (j & 31)) rest += bp;
        if (lane == 0) topk_w[row * topk + j] = bp;   // divided below
      }
    } else if (lane == 0) {
      topk_w[row * topk + j] = bp;
    }
  }
  if (renormalize) {
    const float wsum = warp_sum(my_w + rest);
    if (lane < topk) topk_w[row * topk + lane] = my_w / wsum;
    if (lane == 0)
      for (int j = 32; j < topk; ++j) topk_w[row * topk + j] = topk_w[row * topk + j] / wsum;
  }
}

// Experts per lane, in the order of the instances: an instance takes the rows that the one before it does not hold.
template <int PER_LANE> constexpr int kPerLaneBefore = PER_LANE == 16 ? 12 : PER_LANE == 12 ? 8 : PER_LANE / 2;

// P > 1: E is a multiple of P and every row lies on a boundary of P logits, so that a piece is in the row or not.
template <typename T, int PER_LANE, int P>
__global__ void __launch_bounds__(32 * kWarpsPerBlock, PER_LANE == 32 ? 0 : 1)   // (1 against 0, which leaves it open: E=256 9.2 / 9.4 us; E=1024, all logits equal, 58.6 / 57.5)
topk_softmax_kernel(const T* __restrict__ gating, float* __restrict__ topk_w, int32_t* __restrict__ topk_ids,
                    int64_t M, int E, int topk, int renormalize) {
  __shared__ uint2 s_cand[kWarpsPerBlock][32];   // candidates by ascending id: exponential, id
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t row = (int64_t)blockIdx.x * kWarpsPerBlock + warp;
  if (row >= M) return;

  constexpr int kPieces = PER_LANE / P;
  constexpr int kSure = kPerLaneBefore<PER_LANE>;   // the lane's first experts are in every row of this instance
  auto valid = [&](int t) -> bool { return t < kSure || (t / P * 32 + lane) * P < E; };
  struct alignas(P * sizeof(T)) Piece { T x[P]; };
  const Piece* x = reinterpret_cast<const Piece*>(gating + row * E);
  float p[PER_LANE];
#pragma unroll
  for (int c = 0; c < kPieces; ++c) {
    Piece q;
#pragma unroll
    for (int i = 0; i < P; ++i) q.x[i] = T(-INFINITY);
    if (valid(c * P)) q = x[c * 32 + lane];
#pragma unroll
    for (int i = 0; i < P; ++i) p[c * P + i] = load_logit<T>(&q.x[i]);
  }
  float mx = p[0];
#pragma unroll
  for (int t = 1; t < PER_LANE; ++t) mx = fmaxf(mx, p[t]);
  mx = warp_max(mx);
  // (experts behind the row: -inf, which is 0 here unless the whole row is -inf or NaN, and then the sum is NaN)
  float sum = 0.f, lane_max = 0.f;
#pragma unroll
  for (int t = 0; t < PER_LANE; ++t) {
    p[t] = expf(p[t] - mx);
    sum += p[t];
    lane_max = fmaxf(lane_max, p[t]);
  }
  sum = warp_sum(sum);

  // The k-th largest lane maximum (equal ones leave together, so it may be a smaller one: still a bound).
  float tau = -1.f, lm = lane_max;
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
  // An exponential is a candidate from here on.  Places behind the row hold 0: with a bound of 0 the row's own experts,
  // more than 32 from two a lane on, are candidates too, and the row takes the rounds.
  auto low = [&](int t) -> float { return PER_LANE > 1 || valid(t) ? bound : INFINITY; };
  // Candidates are counted piece by piece.  P > 1: a lane's counts are fields of eight bits (a piece has at most 128
  // candidates in the warp), so that one sum over the lanes serves four pieces.
  constexpr int kWords = (kPieces + 3) / 4;
  uint32_t mine[kWords] = {}, upto[kWords] = {}, all[kWords] = {};   // this lane's, the lanes' up to it, the warp's
  int n = 33;
  if (PER_LANE > 8 && !short_way) {   // (a branch for up to eight costs the short way more than it gives: E=256 10.4 / 10.9 us)
  } else if constexpr (P > 1) {
    n = 0;
#pragma unroll
    for (int t = 0; t < PER_LANE; ++t) mine[t / P / 4] += p[t] >= low(t) ? 1u << (8 * (t / P % 4)) : 0u;
#pragma unroll
    for (int i = 0; i < kWords; ++i) upto[i] = mine[i];
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
#pragma unroll
      for (int i = 0; i < kWords; ++i) {
        const uint32_t below = __shfl_up_sync(0xffffffffu, upto[i], d);
        if (lane >= d) upto[i] += below;
      }
    }
#pragma unroll
    for (int i = 0; i < kWords; ++i) {
      all[i] = __shfl_sync(0xffffffffu, upto[i], 31);
      n = (int)__dp4a(all[i], 0x01010101u, (uint32_t)n);
    }
  } else {
    n = 0;
#pragma unroll
    for (int t = 0; t < PER_LANE; ++t) n += __popc(__ballot_sync(0xffffffffu, p[t] >= low(t)));
  }
  if (!short_way || n > 32) {
#pragma unroll
    for (int t = 0; t < PER_LANE; ++t) p[t] = p[t] / sum;   // (behind the row: 0, or NaN if all are, and higher ids than topk needs)
    select_by_rounds<PER_LANE, P>(p, row, lane, topk, renormalize, topk_w, topk_ids);
    return;
  }
  uint2* cand = s_cand[warp];
  const uint32_t cand_u32 = (uint32_t)__cvta_generic_to_shared(cand);
  if constexpr (P > 1) {
    uint32_t first[kWords], before = 0;   // the fields before it, and the lanes before
#pragma unroll
    for (int i = 0; i < kWords; ++i) {
      first[i] = upto[i] - mine[i] + all[i] * 0x01010100u + before * 0x01010101u;
      before = __dp4a(all[i], 0x01010101u, before);
    }
#pragma unroll
    for (int c = 0; c < kPieces; ++c) {
      uint32_t to = cand_u32 + (first[c / 4] >> (8 * (c % 4)) & 0xFFu) * 8u;
#pragma unroll
      for (int i = 0; i < P; ++i)   // predicated: a branch each took twice as many instructions
        asm volatile("{\n\t.reg .pred q;\n\tsetp.ge.f32 q, %1, %2;\n\t@q st.shared.v2.b32 [%0], {%3, %4};\n\t@q add.u32 %0, %0, 8;\n\t}"
                     : "+r"(to) : "f"(p[c * P + i]), "f"(low(c * P)), "r"(__float_as_uint(p[c * P + i])),
                       "r"(lane * P + Deal<P>::at(c * P + i))
                     : "memory");
    }
  } else {
    uint32_t to = cand_u32;
#pragma unroll
    for (int t = 0; t < PER_LANE; ++t) {
      const unsigned who = __ballot_sync(0xffffffffu, p[t] >= low(t));
      asm volatile("{\n\t.reg .pred q;\n\tsetp.ge.f32 q, %1, %2;\n\t@q st.shared.v2.b32 [%0], {%3, %4};\n\t}"
                   :: "r"(to + (uint32_t)__popc(who & ((1u << lane) - 1u)) * 8u), "f"(p[t]), "f"(low(t)), "r"(__float_as_uint(p[t])),
                      "r"(t * 32 + lane) : "memory");
      to += (uint32_t)__popc(who) * 8u;
    }
  }
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

// Experts of a piece.  Wider ones take fewer loads and spread less: E=256 with pieces of four 9.1 us for independent logits
// and 14.3, 12.4 for one and two live groups, of two 9.2 and 9.3, 9.4; E=128 with pieces of two 7.9 and 9.7 for two live
// groups of sixteen, of one 7.8 and 7.8.  From 257 experts on a live group is rarely that small.
constexpr int piece_of(int per_lane) { return per_lane <= 4 ? 1 : per_lane == 8 ? 2 : 4; }

template <typename T>
int launch_for_type(const void* gating, float* w, int32_t* ids, int64_t M, int E, int topk, int renorm,
                    cudaStream_t s) {
  const unsigned blocks = (unsigned)ceil_div(M, (int64_t)kWarpsPerBlock);
  const T* g = static_cast<const T*>(gating);
  // the fewest experts per lane that cover the row; single logits where pieces would straddle its ends or their alignment
  const int per_lane = (E + 31) / 32;
#define XKB_TS_CASE(PL)                                                                                  \
  if (per_lane <= PL) {                                                                                  \
    constexpr int kP = piece_of(PL);                                                                     \
    const bool whole = E % kP == 0 && reinterpret_cast<uintptr_t>(gating) % (kP * sizeof(T)) == 0;       \
    (whole ? topk_softmax_kernel<T, PL, kP> : topk_softmax_kernel<T, PL, 1>)<<<blocks, 32 * kWarpsPerBlock, 0, s>>>( \
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
