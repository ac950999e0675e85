// moe_sum_reduce and the fused ops' top-k combine for sm_100a.
//
//   out[m, h] = rsf * sum_k (w[m,k] or 1) * y[m,k,h]        fp32, ascending k
//
// HBM-bound.  A thread owns 8 consecutive columns of one token and requests up to kBatch of its top_k
// rows with 128-bit loads before it adds the first; a block is a piece of one token's columns, or several
// tokens of narrow rows, so that the token is found with one 32-bit division and not a 64-bit one.
// No atomics, fixed summation order: the result is bit-reproducible run to run.  Reference semantics:
// src/xkernels/ops/moe/sum_reduce.py:20-39.
// M=8192, top_k=8, H=7168, bf16 (1.06 GB): 232 -> 153 us, 6.9 TB/s.
#include "common.cuh"

namespace xkb {
namespace {

template <typename T> struct Vec8;
template <> struct Vec8<__nv_bfloat16> {
  uint4 r;
  __device__ __forceinline__ void load(const __nv_bfloat16* p) {
    r = *reinterpret_cast<const uint4*>(p);   // plain loads: the rows may come from a kernel this one overlaps
  }
  __device__ __forceinline__ float get(int i) const {   // constant i
    const uint32_t u = i < 2 ? r.x : i < 4 ? r.y : i < 6 ? r.z : r.w;
    return (i & 1) ? __uint_as_float(u & 0xffff0000u) : __uint_as_float(u << 16);
  }
  static __device__ __forceinline__ void store(__nv_bfloat16* p, const float (&v)[8]) {
    uint32_t u[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
      u[i] = *reinterpret_cast<uint32_t*>(&h);
    }
    *reinterpret_cast<uint4*>(p) = make_uint4(u[0], u[1], u[2], u[3]);
  }
  static constexpr int kBatch = 8;
};
template <> struct Vec8<float> {
  float4 a, b;
  __device__ __forceinline__ void load(const float* p) {
    a = *reinterpret_cast<const float4*>(p);
    b = *(reinterpret_cast<const float4*>(p) + 1);
  }
  __device__ __forceinline__ float get(int i) const {
    const float4 q = i < 4 ? a : b;
    return (i & 3) == 0 ? q.x : (i & 3) == 1 ? q.y : (i & 3) == 2 ? q.z : q.w;
  }
  static __device__ __forceinline__ void store(float* p, const float (&v)[8]) {
    reinterpret_cast<float4*>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<float4*>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
  }
  static constexpr int kBatch = 4;
};

__device__ __forceinline__ float to_f(float x) { return x; }
__device__ __forceinline__ float to_f(__nv_bfloat16 x) { return __bfloat162float(x); }
__device__ __forceinline__ void from_f(float& d, float x) { d = x; }
__device__ __forceinline__ void from_f(__nv_bfloat16& d, float x) { d = __float2bfloat16_rn(x); }

// Validity of slot (m,k): the same predicate as the align stage (align.cu:map_expert), which
// drops a slot whose (mapped) expert id falls outside [0, E) and therefore never has its fp32
// row written.  The reference skips those slots too (src/xkernels/ops/moe/reference.py:59-63,
// mxfp4_reference.py:82-83).  ids == nullptr means every slot contributes (moe_sum_reduce).
__device__ __forceinline__ bool slot_valid(const int32_t* ids, const int32_t* emap, int num_map,
                                           int E, int64_t slot) {
  if (ids == nullptr) return true;
  int g = ids[slot];
  if (emap != nullptr) {
    if (g < 0 || g >= num_map) return false;
    g = emap[g];
  }
  return g >= 0 && g < E;
}

// Which rows a token adds up.
//   kAll: row m * top_k + k;  kSlots: the same, without the slots the align stage dropped (ids, emap);
//   kIndexed: row ids[m * top_k + k], none where that is negative.
enum Rows { kAll, kSlots, kIndexed };

// NARROW: a block is `per` tokens instead of a piece of one.
template <typename TY, typename TW, typename TO, Rows ROWS, bool NARROW>
__global__ void __launch_bounds__(256)
sum_reduce_vec8_kernel(const TY* y, const TW* __restrict__ w, TO* __restrict__ out,
                       int64_t M, unsigned pieces, unsigned per, int top_k, int64_t H, float rsf,
                       const int32_t* __restrict__ ids, const int32_t* __restrict__ emap, int num_map, int E) {
  // As the combine of a fused call the slot rows come from the GEMM kernel before this one, which is
  // still running when this kernel starts: `y` is therefore not `const __restrict__` (no invariant /
  // non-coherent loads, which may deliver what was there before the wait).
  chain_wait();
  unsigned m = blockIdx.x / pieces;
  int64_t h = ((int64_t)(blockIdx.x - m * pieces) * blockDim.x + threadIdx.x) << 3;
  if (NARROW) {
    const unsigned hv = (unsigned)(H >> 3), t = threadIdx.x / hv;
    m = blockIdx.x * per + t;
    h = (int64_t)(threadIdx.x - t * hv) << 3;
    if (t >= per || m >= M) return;
  }
  if (h >= H) return;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  const int64_t slot0 = (int64_t)m * top_k;
  constexpr int kBatch = NARROW ? 4 : Vec8<TY>::kBatch;   // (there are enough tokens)
  for (int k0 = 0; k0 < top_k; k0 += kBatch) {
    Vec8<TY> v[kBatch];
    bool take[kBatch];
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      const int64_t slot = slot0 + k0 + j;
      int64_t row = slot;
      take[j] = k0 + j < top_k;
      if (ROWS == kSlots) take[j] = take[j] && slot_valid(ids, emap, num_map, E, slot);
      if (ROWS == kIndexed && take[j]) { row = ids[slot]; take[j] = row >= 0; }
      if (take[j]) v[j].load(y + row * H + h);
    }
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      if (!take[j]) continue;
      if (w != nullptr) {
        const float wk = to_f(w[slot0 + k0 + j]);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          // the combine's rows count as fp32 products: rounded before they are added, not fused
          if (ROWS == kSlots) acc[i] = __fadd_rn(acc[i], __fmul_rn(v[j].get(i), wk));
          else acc[i] += v[j].get(i) * wk;
        }
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] += v[j].get(i);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] *= rsf;
  Vec8<TO>::store(out + (int64_t)m * H + h, acc);
}

// The grid: as few pieces of a token of at most `most` threads as cover H / 8 columns, in whole warps; or, where
// a row fills half a block or less and the tokens are many, `per` tokens per block (a block of a few live threads
// per token costs more in launches than in loads: M=262144, H=8, top_k=2, bf16 137 us with a token per block,
// 3.3 with as many as fit; M=65536, H=64, top_k=8 36.3 and 8.2; M=16384, H=128, top_k=8 10.7 and 4.7).  At least kFullGrid blocks are left, below which the
// tokens are spread over the chip instead.  False if the grid would not fit.  The combine of a fused call takes
// 128: blocks of 256 threads need more registers than a GEMM block leaves free, so that they could not be resident
// yet when the GEMM ends (2 us a call).
struct Vec8Grid { unsigned pieces, per, threads, blocks; };
constexpr int64_t kFullGrid = 4 * 148;
bool vec8_grid(int64_t M, int64_t H, int64_t most, Vec8Grid* g) {
  const int64_t hv = H / 8, p = ceil_div(hv, most);
  int64_t per = most / hv < M / kFullGrid ? most / hv : M / kFullGrid;
  if (per < 1) per = 1;
  if (p * ceil_div(M, per) > 0x7fffffff || M > 0x7fffffff) return false;
  g->pieces = (unsigned)p;
  g->per = (unsigned)per;
  g->threads = (unsigned)align_up(per > 1 ? per * hv : ceil_div(hv, p), 32);
  g->blocks = (unsigned)(p * ceil_div(M, per));
  return true;
}

// Any H / any alignment.
template <typename TY, typename TW, typename TO>
__global__ void __launch_bounds__(256)
sum_reduce_scalar_kernel(const TY* __restrict__ y, const TW* __restrict__ w, TO* __restrict__ out,
                         int64_t M, int top_k, int64_t H, float rsf,
                         const int32_t* __restrict__ ids, const int32_t* __restrict__ emap,
                         int num_map, int E) {
  const int64_t total = M * H;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t m = idx / H, h = idx - m * H;
    float acc = 0.f;
    for (int k = 0; k < top_k; ++k) {
      if (!slot_valid(ids, emap, num_map, E, m * top_k + k)) continue;
      const float v = to_f(y[(m * top_k + k) * H + h]);
      if (w != nullptr && ids != nullptr) acc = __fadd_rn(acc, __fmul_rn(v, to_f(w[m * top_k + k])));   // as above
      else acc += (w != nullptr) ? v * to_f(w[m * top_k + k]) : v;
    }
    from_f(out[idx], acc * rsf);
  }
}

template <typename TY, typename TW, typename TO>
int launch_typed(const void* y, const void* w, void* out, int64_t M, int top_k, int64_t H, float rsf,
                 const int32_t* ids, const int32_t* emap, int num_map, int E, cudaStream_t stream) {
  if (M == 0 || H == 0) return XKB_OK;
  Vec8Grid g{};
  const bool vec_ok = (H % 8 == 0) && (reinterpret_cast<uintptr_t>(y) % 16 == 0) &&
                      (reinterpret_cast<uintptr_t>(out) % 16 == 0) && vec8_grid(M, H, ids != nullptr ? 128 : 256, &g);
  if (vec_ok) {
    const bool narrow = g.per > 1;
    auto kernel = ids != nullptr ? (narrow ? sum_reduce_vec8_kernel<TY, TW, TO, kSlots, true> : sum_reduce_vec8_kernel<TY, TW, TO, kSlots, false>)
                                 : (narrow ? sum_reduce_vec8_kernel<TY, TW, TO, kAll, true> : sum_reduce_vec8_kernel<TY, TW, TO, kAll, false>);
    XKB_CHECK_CUDA(launch_chained(kernel, dim3(g.blocks), dim3(g.threads), 0, stream,
                                  static_cast<const TY*>(y), static_cast<const TW*>(w), static_cast<TO*>(out), M, g.pieces,
                                  g.per, top_k, H, rsf, ids, emap, num_map, E));
    XKB_CHECK_LAUNCH("sum_reduce_vec8_kernel");
  } else {
    // 148 SMs x 8 resident 256-thread CTAs; grid-stride covers the rest
    int64_t blocks = ceil_div(M * H, 256);
    const int64_t cap = 148 * 8 * 4;
    if (blocks > cap) blocks = cap;
    sum_reduce_scalar_kernel<TY, TW, TO><<<(unsigned)blocks, 256, 0, stream>>>(
        static_cast<const TY*>(y), static_cast<const TW*>(w), static_cast<TO*>(out), M, top_k, H, rsf,
        ids, emap, num_map, E);
    XKB_CHECK_LAUNCH("sum_reduce_scalar_kernel");
  }
  return XKB_OK;
}

template <typename TY, typename TW>
int dispatch_out(int out_dtype, const void* y, const void* w, void* out, int64_t M, int top_k,
                 int64_t H, float rsf, const int32_t* ids, const int32_t* emap, int num_map,
                 int E, cudaStream_t s) {
  if (out_dtype == XKB_BF16)
    return launch_typed<TY, TW, __nv_bfloat16>(y, w, out, M, top_k, H, rsf, ids, emap, num_map, E, s);
  return launch_typed<TY, TW, float>(y, w, out, M, top_k, H, rsf, ids, emap, num_map, E, s);
}

// out[m, :] = sum_k w[m,k] * rows[row_index[m,k], :]   (fp32 rows, ascending k, fp32 sum).
// row_index < 0 skips the term.  H not a multiple of 8: one thread = 4 consecutive columns.
template <typename TO>
__global__ void __launch_bounds__(256)
gather_reduce_kernel(const float* __restrict__ rows, const int32_t* __restrict__ row_index,
                     const float* __restrict__ w, TO* __restrict__ out, int64_t M, int top_k, int64_t H) {
  const int64_t hv = H >> 2;
  const int64_t total = M * hv;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t m = idx / hv;
    const int64_t h = (idx - m * hv) << 2;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k = 0; k < top_k; ++k) {
      const int32_t r = row_index[m * top_k + k];
      if (r < 0) continue;
      const float4 v = __ldg(reinterpret_cast<const float4*>(rows + (int64_t)r * H + h));
      const float wk = (w != nullptr) ? w[m * top_k + k] : 1.f;
      acc.x += wk * v.x; acc.y += wk * v.y; acc.z += wk * v.z; acc.w += wk * v.w;
    }
    TO* o = out + m * H + h;
    from_f(o[0], acc.x); from_f(o[1], acc.y); from_f(o[2], acc.z); from_f(o[3], acc.w);
  }
}

template <bool NARROW>
void launch_indexed_as(const Vec8Grid& g, const float* rows, const int32_t* row_index, const float* w, void* out, int out_dtype,
                       int64_t M, int top_k, int64_t H, cudaStream_t s) {
  if (out_dtype == XKB_BF16)
    sum_reduce_vec8_kernel<float, float, __nv_bfloat16, kIndexed, NARROW><<<g.blocks, g.threads, 0, s>>>(
        rows, w, static_cast<__nv_bfloat16*>(out), M, g.pieces, g.per, top_k, H, 1.f, row_index, nullptr, 0, 0);
  else
    sum_reduce_vec8_kernel<float, float, float, kIndexed, NARROW><<<g.blocks, g.threads, 0, s>>>(
        rows, w, static_cast<float*>(out), M, g.pieces, g.per, top_k, H, 1.f, row_index, nullptr, 0, 0);
}

}  // namespace

int launch_combine(const float* scratch, const int32_t* topk_ids, const int32_t* expert_map,
                   int num_map, int E, void* out, int out_dtype, int64_t M, int top_k, int64_t N,
                   cudaStream_t stream) {
  return dispatch_out<float, float>(out_dtype, scratch, nullptr, out, M, top_k, N, 1.0f, topk_ids,
                                    expert_map, num_map, E, stream);
}

int launch_combine_bf16(const __nv_bfloat16* rows, const float* w, const int32_t* topk_ids, const int32_t* expert_map,
                        int num_map, int E, void* out, int out_dtype, int64_t M, int top_k, int64_t N,
                        cudaStream_t stream) {
  return dispatch_out<__nv_bfloat16, float>(out_dtype, rows, w, out, M, top_k, N, 1.0f, topk_ids, expert_map, num_map, E,
                                            stream);
}

}  // namespace xkb

extern "C" int xkb_moe_sum_reduce(const void* y, int y_dtype, const void* w, int w_dtype, void* out,
                                  int out_dtype, int64_t M, int top_k, int64_t H,
                                  float routed_scaling_factor, void* stream) {
  using namespace xkb;
  XKB_REQUIRE(M >= 0 && H >= 0 && top_k >= 0, "moe_sum_reduce: negative dimension");
  XKB_REQUIRE((y_dtype == XKB_BF16 || y_dtype == XKB_F32) &&
                  (out_dtype == XKB_BF16 || out_dtype == XKB_F32) &&
                  (w == nullptr || w_dtype == XKB_BF16 || w_dtype == XKB_F32),
              "moe_sum_reduce: dtype codes must be XKB_BF16 or XKB_F32");
  XKB_REQUIRE(M * H == 0 || (y != nullptr && out != nullptr) || top_k == 0,
              "moe_sum_reduce: null y/out pointer");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const float rsf = routed_scaling_factor;
  if (y_dtype == XKB_BF16) {
    if (w != nullptr && w_dtype == XKB_BF16)
      return dispatch_out<__nv_bfloat16, __nv_bfloat16>(out_dtype, y, w, out, M, top_k, H, rsf, nullptr, nullptr, 0, 0, s);
    return dispatch_out<__nv_bfloat16, float>(out_dtype, y, w, out, M, top_k, H, rsf, nullptr, nullptr, 0, 0, s);
  }
  if (w != nullptr && w_dtype == XKB_BF16)
    return dispatch_out<float, __nv_bfloat16>(out_dtype, y, w, out, M, top_k, H, rsf, nullptr, nullptr, 0, 0, s);
  return dispatch_out<float, float>(out_dtype, y, w, out, M, top_k, H, rsf, nullptr, nullptr, 0, 0, s);
}

extern "C" int xkb_moe_gather_sum_reduce(const float* rows, const int32_t* row_index, const float* w,
                                         void* out, int out_dtype, int64_t M, int top_k, int64_t H,
                                         void* stream) {
  using namespace xkb;
  XKB_REQUIRE(M >= 0 && H >= 0 && top_k >= 0, "moe_gather_sum_reduce: negative dimension");
  XKB_REQUIRE(H % 4 == 0, "moe_gather_sum_reduce: H must be a multiple of 4 (got %lld)", (long long)H);
  XKB_REQUIRE(out_dtype == XKB_BF16 || out_dtype == XKB_F32, "moe_gather_sum_reduce: bad out_dtype");
  if (M == 0 || H == 0) return XKB_OK;
  XKB_REQUIRE(rows && row_index && out, "moe_gather_sum_reduce: null pointer");
  XKB_REQUIRE(reinterpret_cast<uintptr_t>(rows) % 16 == 0, "moe_gather_sum_reduce: rows must be 16-byte aligned");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  Vec8Grid g{};
  if (H % 8 == 0 && reinterpret_cast<uintptr_t>(out) % 16 == 0 && vec8_grid(M, H, 256, &g)) {
    (g.per > 1 ? launch_indexed_as<true> : launch_indexed_as<false>)(g, rows, row_index, w, out, out_dtype, M, top_k, H, s);
    XKB_CHECK_LAUNCH("sum_reduce_vec8_kernel");
    return XKB_OK;
  }
  int64_t blocks = ceil_div(M * (H / 4), 256);
  if (blocks > 148 * 32) blocks = 148 * 32;
  if (out_dtype == XKB_BF16)
    gather_reduce_kernel<__nv_bfloat16><<<(unsigned)blocks, 256, 0, s>>>(
        rows, row_index, w, static_cast<__nv_bfloat16*>(out), M, top_k, H);
  else
    gather_reduce_kernel<float><<<(unsigned)blocks, 256, 0, s>>>(rows, row_index, w,
                                                                 static_cast<float*>(out), M, top_k, H);
  XKB_CHECK_LAUNCH("gather_reduce_kernel");
  return XKB_OK;
}
