// MXFP4 expert layer on the block-scaled tensor-core instructions (sm_100a), decode-sized batches.
//
// tcgen05.mma kind::mxf8f6f4 takes the E2M1 weights and their e8m0 scales as they are: TMA unpacks the
// nibbles into the byte containers the instruction reads, and nothing converts them.  The activations are
// bf16 and go in as three block-scaled 8-bit terms that hold every element down to 2^-31 of the largest of its
// 32 exactly (mx_split.cuh).  What bounds the kernel is the weight stream; there is no conversion beside it.
// Larger batches stay on the kernel that converts to bf16 (moe_tc.cu): three terms are half as many token
// bytes again as bf16 activations, and half as many multiplications at twice the rate (mxfp4_bs_block has the line).
//
// Swap-AB like the bf16 kernel: a tile is BT tokens of one expert block x two 128-row weight tiles (gate and
// up rows, or two neighbouring row tiles of the down projection).  One persistent CTA per SM, sixteen warps:
//   warp 0      weight producer: per 128-K stage two [128 x 128] tiles, per four stages their scales
//   warps 1, 2  MMA issuers, one per weight matrix.  One thread issues a narrow MMA per 45 cycles at best, so
//               the three terms are multiplied in one instruction of 3 BT tokens (four a stage): M=48 below
//               184 us with the terms on two issuers, 168 on three, 144 in one instruction (16-token tiles).
//   warp 3      token producer (the terms of the stage, per four stages their scales)
//   warps 4-7   scale movers: the scale tiles are row-major, the instruction wants row r of a 128-row tile in
//               lane r % 32, column r / 32 of tensor memory, the same in all four lane quarters.  Sixteen
//               bytes of a row are four stages' scales: every warp reads them once and writes one column
//               word per 32 rows and stage.
//   warps 8-15  read-out, a tile behind the MMAs (two to four accumulator sets)
//
// Measured at E=256, hidden 4096, ispp 512, top_k 6, whole call in a graph, against the kernel that converts to
// bf16: M=48 189 -> 139 us (0.58 GB of weights: 89 us at the copy rate), M=768 466 -> 259.
//
// Scale byte 0xFF means weight 0 here (it is NaN to the instruction): a mover that meets one clears the
// group's weights in shared memory and puts byte 0 in its place.
#include <cuda_fp16.h>
#include "align_dev.cuh"
#include "moe_kernels.h"
#include "mx_split.cuh"
#include "tc_common.cuh"
#include "tensor_map.h"

namespace xkb {
extern std::atomic<int> g_sm_margin;
namespace {

using namespace tc;

constexpr int kRows = 128;          // weight rows per matrix and tile (UMMA M)
constexpr int kStageK = 128;        // K per stage: one 128-byte swizzled row of byte containers
constexpr int kChunkStages = 4;     // stages per 16-byte scale row
constexpr int kWBytes = kRows * kStageK;
constexpr int kTerms = 3;             // of an activation: hi, mid, lo
constexpr int kThreads = 512;
constexpr int kTmemCols = 512;
constexpr uint32_t kProdSleepNs = 200;

template <int BT> struct MxCfg {
  static_assert(BT == 8 || BT == 16 || BT == 32, "token tile");
  // All three terms are multiplied in ONE instruction: the terms' tiles lie behind one another in shared
  // memory, which is a tile of 3 BT tokens, each term with accumulators of its own that the read-out adds up.  An
  // instruction costs its issuer 45 cycles up to 32 tokens or so, whatever its width.
  static constexpr int kTermRows = kTerms * BT;
  // UMMA N, a multiple of 16: 8-token tiles read eight rows more (of what lies behind the stage; columns that nobody reads)
  static constexpr int kMmaTokens = (kTermRows + 15) / 16 * 16;
  static constexpr int kTokRowGroups = (kMmaTokens + 31) / 32;
  static constexpr int kTokBytes = BT * kStageK;                      // one term
  static_assert(kTokBytes % 1024 == 0, "swizzle atoms");
  static constexpr int kStageBytes = 2 * kWBytes + kTerms * kTokBytes;
  static constexpr int kStages = BT == 8 ? 6 : BT == 16 ? 5 : 4;
  // Scale tiles are loaded with the first stage of their four and read with all four: a slot is free again
  // when the MMAs kStages before that first stage are done, if kStages <= 4 * slots - 3.
  static constexpr int kScSlots = kStages > 5 ? 3 : 2;
  static_assert(kStages <= 4 * kScSlots - 3, "scale slots");
  static constexpr int kScBytes = 2 * kRows * 16 + BT * 16;
  static_assert(kScSlots * kScBytes >= (kMmaTokens - kTermRows) * kStageK, "the rows read behind the last stage lie in the scale tiles");
  // columns: accumulator sets of two matrices, then per stage 4 gate + 4 up + 4 token scale columns
  static constexpr int kScStageCols = 12;
  static constexpr int kScCols = kScStageCols * kStages;
  static constexpr int kSetCols = 2 * kMmaTokens;                     // accumulators of matrix 1 behind those of matrix 0
  static constexpr int kDFit = (kTmemCols - kScCols) / kSetCols;
  static constexpr int kDBuf = kDFit > 4 ? 4 : kDFit;
  static_assert(kDBuf >= 2, "the read-out must overlap the next tile");
  // (with one column group the two warpgroups take alternate tiles: each must meet every use of its accumulator sets)
  static_assert(BT > 16 || kDBuf % 2 == 0, "accumulator sets alternate with the warpgroups");
  static constexpr int kScCol0 = kDBuf * kSetCols;
  static constexpr int kCols = BT < 16 ? BT : 16;                     // columns of a read-out step
  static constexpr int kColGroups = BT / kCols;
  static constexpr int kEpiWGs = kColGroups < 2 ? 1 : 2;              // read-out warpgroups per tile
  static constexpr int kNumBars = 3 * kStages + 2 * kDBuf;
  static constexpr size_t kSmemBytes = 1024 + (size_t)kStages * kStageBytes + (size_t)kScSlots * kScBytes + kNumBars * 8 + 64;
  static_assert(kSmemBytes <= 227 * 1024, "shared memory overcommitted");
};

struct MxParams {
  const int32_t* sorted_ids;
  const int32_t* expert_ids;
  const int32_t* num_post;
  const __nv_bfloat16* bias;    // [E, rows_per_expert] or nullptr
  uint8_t* act[kTerms];         // gate_up: the terms [positions, N] and hi's scales [positions, N / 32]
  uint8_t* act_scale;
  __nv_bfloat16* rows;          // down: [slots, N], the bf16-rounded rows before the routing weight
  int* status;
  int64_t numel;
  int N, K;                     // output columns (weight rows per matrix: N of gate and up each, N down), contraction
  int rows_per_expert;
  int mat_row;                  // rows between the two matrices of a tile
  int tile_step;                // output rows per tile: 128 gate_up, 256 down
  float limit;                  // SwiGLU clamp, <= 0 disables
  int max_blocks, num_experts;
  int32_t* done_signal;         // gate_up: finished read-outs per token block
  const int32_t* done_wait;     // down: the same, waited for
  int done_target;
};

// Instruction descriptor, kind::mxf8f6f4: b_sf_id [4,6), a type [7,10) (5 = e2m1), b type [10,13) (1 = e5m2),
// N >> 3 [17,23), scale type 23 (1 = ue8m0), M >> 7 [27,29), a_sf_id [29,31); fp32 accumulators,
// both operands K-major.
constexpr uint32_t mx_idesc(int n, int sf) {
  return ((uint32_t)sf << 4) | (5u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | (1u << 23) | (1u << 27) |
         ((uint32_t)sf << 29);
}
__device__ __forceinline__ void umma_mx(uint32_t d, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t sfa,
                                        uint32_t sfb, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %6, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%4], [%5], p;\n\t}"
      ::"r"(d), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(sfa), "r"(sfb), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_st_32x4(uint32_t taddr, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};"
               ::"r"(taddr), "r"(r0), "r"(r1), "r"(r2), "r"(r3) : "memory");
}
__device__ __forceinline__ void sts128_zero(uint32_t addr) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(addr), "r"(0) : "memory");
}
__device__ __forceinline__ uint32_t word_of(const uint4& v, int j) { return j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w; }

template <int BT, bool GATE_UP>
__global__ void __launch_bounds__(kThreads, 1)
moe_mx_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_ws,
              const __grid_constant__ CUtensorMap tm_hi, const __grid_constant__ CUtensorMap tm_mid,
              const __grid_constant__ CUtensorMap tm_lo, const __grid_constant__ CUtensorMap tm_xs, const MxParams p) {
  using Cfg = MxCfg<BT>;
  constexpr int kStages = Cfg::kStages, kDBuf = Cfg::kDBuf, kCols = Cfg::kCols;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* s_sc = smem + kStages * Cfg::kStageBytes;     // kScSlots x { gate, up [128 x 16], tokens [BT x 16] }
  uint64_t* full = reinterpret_cast<uint64_t*>(s_sc + Cfg::kScSlots * Cfg::kScBytes);
  uint64_t* sf_full = full + kStages;
  uint64_t* empty = sf_full + kStages;
  uint64_t* d_full = empty + kStages;
  uint64_t* d_empty = d_full + kDBuf;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(d_empty + kDBuf);
  int* abort_word = reinterpret_cast<int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  Guard guard{abort_word, p.status};
  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) { mbar_init(&full[i], 2); mbar_init(&sf_full[i], 4); mbar_init(&empty[i], 2); }
    for (int i = 0; i < kDBuf; ++i) { mbar_init(&d_full[i], 2); mbar_init(&d_empty[i], 4 * Cfg::kEpiWGs); }
    *abort_word = 0;
    mbar_fence_init();
  }
  if (warp == 3) tmem_alloc(tmem_slot, kTmemCols);
  if (warp == 0 && lane == 0) { prefetch_tensormap(&tm_w); prefetch_tensormap(&tm_ws); }
  if (warp == 3 && lane == 0) {
    prefetch_tensormap(&tm_hi); prefetch_tensormap(&tm_mid); prefetch_tensormap(&tm_lo); prefetch_tensormap(&tm_xs);
  }
  // Block hand-over between the two GEMMs: as in the bf16 kernel (moe_tc.cu).  The first lets its dependents
  // go after its own wait; the second does not wait for the first grid but per token block, on a counter.
  const bool first = GATE_UP && p.done_signal != nullptr, second = p.done_wait != nullptr;
  if (!first) chain_trigger();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  if (!second) chain_wait();
  if (first) chain_trigger();

  const int n_tiles = p.N / p.tile_step;
  const int n_post = __ldcg(p.num_post);   // written by kernels this one may overlap: L2 loads, after the wait
  const bool routing_ok = n_post >= 0 && n_post <= p.max_blocks * BT;
  if (!routing_ok && threadIdx.x == 0) atomicCAS(p.status, 0, kErrBadRouting + (1 << 8));
  const int total_tiles = routing_ok ? n_post / BT * n_tiles : 0;
  const int k_stages = p.K / kStageK;      // a multiple of kChunkStages: scale chunks never straddle tiles

  if (warp == 0) {
    // ---------------- weight producer ----------------
    if (lane == 0) {
      uint32_t st = 0, ph = 1, chunk = 0;
      bool ok = true;
      for (int t = (int)blockIdx.x; t < total_tiles && ok && !guard.aborted(); t += (int)gridDim.x) {
        const int b = t / n_tiles, nt = t - b * n_tiles;
        int e = __ldcg(p.expert_ids + b);
        if ((unsigned)e >= (unsigned)p.num_experts) { atomicCAS(p.status, 0, kErrBadRouting + (2 << 8)); e = 0; }
        const int row0 = e * p.rows_per_expert + nt * p.tile_step, row1 = row0 + p.mat_row;
        for (int ks = 0; ks < k_stages; ++ks) {
          if (!mbar_wait(&empty[st], ph, guard, 1, kProdSleepNs)) { ok = false; break; }
          unsigned char* s = smem + st * Cfg::kStageBytes;
          const bool head = (ks & (kChunkStages - 1)) == 0;
          mbar_expect_tx(&full[st], kWBytes + (head ? 2 * kRows * 16 : 0));   // the unpacking copies count the bytes read
          tma_load_2d(s, &tm_w, &full[st], ks * kStageK, row0);
          tma_load_2d(s + kWBytes, &tm_w, &full[st], ks * kStageK, row1);
          if (head) {
            unsigned char* sc = s_sc + (chunk % Cfg::kScSlots) * Cfg::kScBytes;
            tma_load_2d(sc, &tm_ws, &full[st], ks * (kStageK / 32), row0);
            tma_load_2d(sc + kRows * 16, &tm_ws, &full[st], ks * (kStageK / 32), row1);
            ++chunk;
          }
          if (++st == kStages) { st = 0; ph ^= 1; }
        }
      }
    }
  } else if (warp == 3) {
    // ---------------- token producer ----------------
    if (lane == 0) {
      uint32_t st = 0, ph = 1, chunk = 0;
      int ready_b = -1;
      bool ok = true;
      for (int t = (int)blockIdx.x; t < total_tiles && ok && !guard.aborted(); t += (int)gridDim.x) {
        const int b = t / n_tiles, pos0 = b * BT;
        if (second && b != ready_b) {
          uint64_t t0 = 0;
          bool ready = false;
          for (uint32_t i = 1; !ready; ++i) {
            int32_t seen;
            asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(seen) : "l"(p.done_wait + b) : "memory");
            if (seen >= p.done_target) { ready = true; break; }
            __nanosleep(100);
            if ((i & 15u) == 0u) {
              if (guard.aborted()) break;
              const uint64_t now = globaltimer_ns();
              if (t0 == 0) t0 = now;
              else if (now - t0 > kWaitBudgetNs) { guard.raise(kErrWaitTimeout + (9 << 8)); break; }
            }
          }
          if (!ready) { ok = false; break; }
          asm volatile("fence.proxy.async;" ::: "memory");   // the TMA loads below read what generic stores wrote
          ready_b = b;
        }
        for (int ks = 0; ks < k_stages; ++ks) {
          if (!mbar_wait(&empty[st], ph, guard, 2, kProdSleepNs)) { ok = false; break; }
          unsigned char* s = smem + st * Cfg::kStageBytes + 2 * kWBytes;
          const bool head = (ks & (kChunkStages - 1)) == 0;
          mbar_expect_tx(&full[st], kTerms * Cfg::kTokBytes + (head ? BT * 16 : 0));
          tma_load_2d(s, &tm_hi, &full[st], ks * kStageK, pos0);
          tma_load_2d(s + Cfg::kTokBytes, &tm_mid, &full[st], ks * kStageK, pos0);
          tma_load_2d(s + 2 * Cfg::kTokBytes, &tm_lo, &full[st], ks * kStageK, pos0);
          if (head) {
            unsigned char* sc = s_sc + (chunk % Cfg::kScSlots) * Cfg::kScBytes + 2 * kRows * 16;
            tma_load_2d(sc, &tm_xs, &full[st], ks * (kStageK / 32), pos0);
            ++chunk;
          }
          if (++st == kStages) { st = 0; ph ^= 1; }
        }
      }
    }
  } else if (warp < 3) {
    // ---------------- MMA issuers: warp 1 + matrix ----------------
    if (lane == 0) {
      const uint32_t mat = (uint32_t)warp - 1;
      uint32_t st = 0, ph = 0, dbuf = 0, dph = 1;
      bool ok = true;
      for (int t = (int)blockIdx.x; t < total_tiles && ok && !guard.aborted(); t += (int)gridDim.x) {
        if (!mbar_wait(&d_empty[dbuf], dph, guard, 8)) break;
        tc_fence_after();
        const uint32_t d = tmem_base + dbuf * Cfg::kSetCols + mat * Cfg::kMmaTokens;
        for (int ks = 0; ks < k_stages; ++ks) {
          if (!mbar_wait(&full[st], ph, guard, 3) || !mbar_wait(&sf_full[st], ph, guard, 4)) { ok = false; break; }
          tc_fence_after();
          const uint32_t s = smem_u32(smem + st * Cfg::kStageBytes);
          const uint64_t a = umma_desc_k_sw128(s + mat * kWBytes);
          const uint64_t bt = umma_desc_k_sw128(s + 2 * kWBytes);
          const uint32_t sc = tmem_base + Cfg::kScCol0 + st * Cfg::kScStageCols, sw = sc + mat * 4;
          // 32 K each: 32 bytes on in the swizzled rows, the next scale byte
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_mx(d, a + k * 2, bt + k * 2, mx_idesc(Cfg::kMmaTokens, k), sw, sc + 8, (ks | k) != 0);
          tc_commit(&empty[st]);
          if (++st == kStages) { st = 0; ph ^= 1; }
        }
        if (!ok) break;
        tc_commit(&d_full[dbuf]);
        if (++dbuf == kDBuf) { dbuf = 0; dph ^= 1; }
      }
    }
  } else if (warp < 8) {
    // ---------------- scale movers ----------------
    const int quarter = warp & 3;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    uint32_t st = 0, ph = 0, chunk = 0;
    bool ok = true;
    for (int t = (int)blockIdx.x; t < total_tiles && ok && !guard.aborted(); t += (int)gridDim.x) {
      for (int kc = 0; kc < k_stages && ok; kc += kChunkStages, ++chunk) {
        const uint32_t sc = smem_u32(s_sc + (chunk % Cfg::kScSlots) * Cfg::kScBytes);
        uint4 w[2][4], x[Cfg::kTokRowGroups];
#pragma unroll
        for (int j = 0; j < kChunkStages; ++j) {
          if (!mbar_wait(&full[st], ph, guard, 5)) { ok = false; break; }
          if (j == 0) {   // the chunk's scales came with this stage
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
              for (int c = 0; c < 4; ++c) w[m][c] = lds128(sc + (uint32_t)((m * kRows + c * 32 + lane) * 16));
#pragma unroll
            for (int c = 0; c < Cfg::kTokRowGroups; ++c)
              x[c] = (c * 32 + lane < Cfg::kTermRows) ? lds128(sc + 2 * kRows * 16 + (uint32_t)((c * 32 + lane) % BT * 16))
                                                       : make_uint4(0, 0, 0, 0);
          }
          const uint32_t dst = tmem_base + lane_base + Cfg::kScCol0 + st * Cfg::kScStageCols;
#pragma unroll
          for (int m = 0; m < 2; ++m) {
            uint32_t v[4], nan = 0;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              v[c] = word_of(w[m][c], j);
              nan |= __vcmpeq4(v[c], 0xFFFFFFFFu);
            }
            if (__any_sync(0xffffffffu, nan != 0)) {   // never for sane weights
#pragma unroll
              for (int c = 0; c < 4; ++c) {
                const uint32_t bad = __vcmpeq4(v[c], 0xFFFFFFFFu);
                if (c == quarter) {
                  const uint32_t row = (uint32_t)(c * 32 + lane);
                  const uint32_t base = smem_u32(smem + st * Cfg::kStageBytes) + m * kWBytes + row * 128;
                  for (uint32_t g = 0; g < 4; ++g)
                    if ((bad >> (8 * g)) & 0xFFu) {
                      sts128_zero(base + (((2 * g) ^ (row & 7)) << 4));
                      sts128_zero(base + (((2 * g + 1) ^ (row & 7)) << 4));
                    }
                }
                v[c] &= ~bad;
              }
              asm volatile("fence.proxy.async;" ::: "memory");   // the MMAs read the cleared weights
            }
            tmem_st_32x4(dst + m * 4, v[0], v[1], v[2], v[3]);
          }
          uint32_t v[4] = {0, 0, 0, 0};
#pragma unroll
          for (int c = 0; c < Cfg::kTokRowGroups; ++c) v[c] = word_of(x[c], j);
          // hi's bytes are kLoShift at least (padding positions hold anything: their columns are never read)
          constexpr uint32_t kMid4 = mx::kMidShift * 0x01010101u, kLo4 = mx::kLoShift * 0x01010101u;
#pragma unroll
          for (int c = 0; c < Cfg::kTokRowGroups; ++c) {
            const int term = (c * 32 + lane) / BT;
            v[c] = __vsub4(v[c], term == 0 ? 0u : term == 1 ? kMid4 : kLo4);
          }
          tmem_st_32x4(dst + 8, v[0], v[1], v[2], v[3]);
          tmem_wait_st();
          tc_fence_before();
          __syncwarp();
          mbar_arrive_if(&sf_full[st], lane == 0 ? 1u : 0u);
          if (++st == kStages) { st = 0; ph ^= 1; }
        }
      }
    }
  } else {
    // ---------------- read-out ----------------
    const int wg = (warp - 8) >> 2, quarter = warp & 3;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    uint32_t dbuf = 0, dph = 0, it = 0;
    for (int t = (int)blockIdx.x; t < total_tiles && !guard.aborted(); t += (int)gridDim.x, ++it) {
      const int b = t / n_tiles, nt = t - b * n_tiles;
      const int cg0 = Cfg::kEpiWGs == 2 ? wg : (int)((wg + it) & 1);   // one column group: the warpgroups take turns
      if (cg0 < Cfg::kColGroups) {
        const int n_glob = nt * p.tile_step + quarter * 32 + lane;
        float bias0 = 0.f, bias1 = 0.f;
        if (p.bias != nullptr) {
          int e = __ldcg(p.expert_ids + b);
          if ((unsigned)e >= (unsigned)p.num_experts) e = 0;   // recorded by the weight producer
          const __nv_bfloat16* eb = p.bias + (int64_t)e * p.rows_per_expert + n_glob;
          bias0 = __bfloat162float(eb[0]);
          bias1 = __bfloat162float(eb[p.mat_row]);
        }
        int32_t next = lane < kCols ? __ldcg(p.sorted_ids + (int64_t)b * BT + cg0 * kCols + lane) : -1;
        if (!mbar_wait(&d_full[dbuf], dph, guard, 7, 100)) break;
        tc_fence_after();
#pragma unroll 1
        for (int cg = cg0; cg < Cfg::kColGroups; cg += Cfg::kEpiWGs) {
          const int32_t my_slot = next;
          if (cg + Cfg::kEpiWGs < Cfg::kColGroups)
            next = lane < kCols ? __ldcg(p.sorted_ids + (int64_t)b * BT + (cg + Cfg::kEpiWGs) * kCols + lane) : -1;
          const uint32_t live = __ballot_sync(0xffffffffu, my_slot >= 0 && my_slot < p.numel) & ((1u << kCols) - 1u);
          if (live == 0u) continue;
          uint32_t a0[kCols], a1[kCols];
          const uint32_t d = tmem_base + lane_base + dbuf * Cfg::kSetCols + cg * kCols;
          tmem_ld(d, a0);
          tmem_ld(d + Cfg::kMmaTokens, a1);
          tmem_wait_ld();
#pragma unroll
          for (int i = 1; i < kTerms; ++i) {
            uint32_t b0[kCols], b1[kCols];
            tmem_ld(d + i * BT, b0);
            tmem_ld(d + Cfg::kMmaTokens + i * BT, b1);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < kCols; ++j) {
              a0[j] = __float_as_uint(__uint_as_float(a0[j]) + __uint_as_float(b0[j]));
              a1[j] = __float_as_uint(__uint_as_float(a1[j]) + __uint_as_float(b1[j]));
            }
          }
          // The columns are computed side by side whether they are live or padding (whose values are
          // never stored): their chains overlap, which branches between them would not allow.
          if (GATE_UP) {
            // rounding points of the reference (src/xkernels/ops/moe/mxfp4_reference.py:92-100)
            uint32_t top[kCols];
#pragma unroll
            for (int j = 0; j < kCols; ++j) {
              float v0 = __uint_as_float(a0[j]), v1 = __uint_as_float(a1[j]);
              round_pair_to_bf16(v0, v1);
              if (p.bias != nullptr) { v0 += bias0; v1 += bias1; round_pair_to_bf16(v0, v1); }
              if (p.limit > 0.f) { v0 = fminf(v0, p.limit); v1 = fminf(fmaxf(v1, -p.limit), p.limit); }
              const float silu = v0 / (1.f + expf(-v0));
              a0[j] = __float_as_uint(silu * v1);
              if (j & 1) {
                float x0 = __uint_as_float(a0[j - 1]), x1 = silu * v1;
                round_pair_to_bf16(x0, x1);
                a0[j - 1] = __float_as_uint(x0);
                a0[j] = __float_as_uint(x1);
              }
            }
            // this warp's 32 rows are one scale block of the next contraction
#pragma unroll
            for (int j = 0; j < kCols; ++j) top[j] = __reduce_max_sync(0xffffffffu, mx::finite_abs_bits(a0[j] >> 16));
            const int64_t pos = (int64_t)b * BT + cg * kCols;
            const int64_t at = pos * p.N + n_glob;
#pragma unroll
            for (int j = 0; j < kCols; j += 2) {
              const float x0 = __uint_as_float(a0[j]), x1 = __uint_as_float(a0[j + 1]);
              const uint32_t s0 = mx::hi_scale(top[j]), s1 = mx::hi_scale(top[j + 1]);
              uint32_t term[kTerms];
              mx::split_pair(x0, x1, mx::hi_factor(s0), mx::hi_factor(s1), term[0], term[1], term[2]);
#pragma unroll
              for (int i = 0; i < kTerms; ++i) {
                if ((live >> j) & 1u) p.act[i][at + (int64_t)j * p.N] = (uint8_t)term[i];
                if ((live >> (j + 1)) & 1u) p.act[i][at + (int64_t)(j + 1) * p.N] = (uint8_t)(term[i] >> 8);
              }
            }
            // lane j stores the scale byte of position j
            uint32_t sh = 0;
#pragma unroll
            for (int j = 0; j < kCols; ++j) sh = lane == j ? mx::hi_scale(top[j]) : sh;
            if ((live >> lane) & 1u)   // (live has kCols bits)
              p.act_scale[(pos + lane) * (p.N / 32) + (n_glob >> 5)] = (uint8_t)sh;
          } else {
#pragma unroll
            for (int j = 0; j < kCols; ++j) {
              float v0 = __uint_as_float(a0[j]), v1 = __uint_as_float(a1[j]);
              if (p.bias != nullptr) { round_pair_to_bf16(v0, v1); v0 += bias0; v1 += bias1; }
              const uint32_t two = pack_bf16(v0, v1);
              const int32_t slot = __shfl_sync(0xffffffffu, my_slot, j);
              if (!((live >> j) & 1u)) continue;        // warp-uniform
              __nv_bfloat16* out = p.rows + (int64_t)slot * p.N + n_glob;
              out[0] = low_bf16(two);
              out[kRows] = high_bf16(two);
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        mbar_arrive_if(&d_empty[dbuf], lane == 0 ? 1u : 0u);
        if (first && lane == 0) {   // the __syncwarp above orders the other lanes' stores before this release
          __threadfence();
          asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(p.done_signal + b) : "memory");
        }
      }
      if (++dbuf == kDBuf) { dbuf = 0; dph ^= 1; }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 3) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// Rows of A, split into the three terms, at the positions of all their slots (token by token, as
// gather_permute_kernel): 32 elements = one scale block = four threads.
struct SplitRows { uint8_t *hi, *mid, *lo, *scale; };   // [positions, K], scales of hi [positions, K / 32]
struct SplitUnit {
  uint32_t h[4], d[4], l[4], scale;
  // eight elements; the four threads of a scale block are neighbours
  __device__ __forceinline__ void load(const uint4* src) {
    const uint4 v = __ldg(src);   // an input of the call
    const uint32_t u[4] = {v.x, v.y, v.z, v.w};
    uint32_t top = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      top = max(top, max(mx::finite_abs_bits(u[q] & 0xFFFFu), mx::finite_abs_bits(u[q] >> 16)));
    top = max(top, __shfl_xor_sync(0xffffffffu, top, 1));
    top = max(top, __shfl_xor_sync(0xffffffffu, top, 2));
    scale = mx::hi_scale(top);
    const float f = mx::hi_factor(scale);
#pragma unroll
    for (int q = 0; q < 4; ++q)
      mx::split_pair(__uint_as_float(u[q] << 16), __uint_as_float(u[q] & 0xFFFF0000u), f, f, h[q], d[q], l[q]);
  }
  __device__ __forceinline__ void store(const SplitRows& x, int64_t pos, int K, int i) const {
    reinterpret_cast<uint2*>(x.hi + pos * K)[i] = make_uint2(h[0] | (h[1] << 16), h[2] | (h[3] << 16));
    reinterpret_cast<uint2*>(x.mid + pos * K)[i] = make_uint2(d[0] | (d[1] << 16), d[2] | (d[3] << 16));
    reinterpret_cast<uint2*>(x.lo + pos * K)[i] = make_uint2(l[0] | (l[1] << 16), l[2] | (l[3] << 16));
    if ((i & 3) == 0) x.scale[pos * (K / 32) + (i >> 2)] = (uint8_t)scale;
  }
};

template <bool SORT>
__global__ void __launch_bounds__(SORT ? 1024 : kGatherThreads)
gather_split_kernel(const __nv_bfloat16* __restrict__ A, const int32_t* slot_pos, const SplitRows x, int K, int top_k,
                    int64_t max_pad, unsigned pieces, unsigned units, int* __restrict__ status, const align::Job job) {
  if (SORT) chain_trigger();   // the first kernel of the call; the next one waits for its completion
  const unsigned m = blockIdx.x / pieces;
  const int i = (int)((blockIdx.x - m * pieces) * units + threadIdx.x);
  const bool mine = threadIdx.x < units && i < K / 8;   // both are multiples of 32: whole warps
  SplitUnit o = {};
  if (mine) o.load(reinterpret_cast<const uint4*>(A + (int64_t)m * K) + i);
  if (!SORT) {
    chain_wait();     // the routing is read with L2 loads after the wait (see gather_permute_kernel)
    chain_trigger();
  }
  const int lane = threadIdx.x & 31;
  for (int j0 = 0; j0 < top_k; j0 += 32) {   // the positions of up to 32 slots in one load
    int32_t mine_pos;
    if (SORT) {
      extern __shared__ __align__(16) unsigned char smem_raw[];
      mine_pos = align::positions_of_token(job, smem_raw, m, top_k, blockIdx.x == 0);   // top_k <= 32: one round
    } else {
      mine_pos = j0 + lane < top_k ? __ldcg(slot_pos + (int64_t)m * top_k + j0 + lane) : -1;
    }
    if (mine_pos >= max_pad) atomicCAS(status, 0, kErrBadRouting + (3 << 8));   // never with a routing the align stage wrote
    unsigned live = __ballot_sync(0xffffffffu, mine_pos >= 0 && mine_pos < max_pad);
    for (; live != 0; live &= live - 1) {
      const int64_t pos = __shfl_sync(0xffffffffu, mine_pos, __ffs(live) - 1);
      if (mine) o.store(x, pos, K, i);
    }
  }
}

// The same through the sorted positions, for calls whose tokens mostly have no slot here.
__global__ void __launch_bounds__(kGatherThreads)
gather_split_positions_kernel(const __nv_bfloat16* __restrict__ A, const int32_t* sorted_ids, const int32_t* num_post,
                              const SplitRows x, int64_t numel, int K, int top_k, int64_t max_pad, int* __restrict__ status) {
  chain_wait();
  chain_trigger();
  const int total = align::positions_to_gather(num_post, max_pad, status);
  for (int64_t pos = blockIdx.x; pos < total; pos += gridDim.x) {
    const int32_t slot = __ldcg(sorted_ids + pos);
    if (slot < 0 || slot >= numel) continue;
    const uint4* src = reinterpret_cast<const uint4*>(A + (int64_t)(slot / top_k) * K);
    for (int i = threadIdx.x; i < K / 8; i += kGatherThreads) {   // K / 8 is a multiple of 32: whole warps
      SplitUnit o;
      o.load(src + i);
      o.store(x, pos, K, i);
    }
  }
}

template <int BT, bool GATE_UP>
int launch_mx(const CUtensorMap (&tm)[6], const MxParams& prm, int64_t max_tiles, cudaStream_t stream) {
  int dev = 0;
  XKB_CHECK_CUDA(cudaGetDevice(&dev));
  static std::atomic<int> sm_count[64];   // 0: this kernel instance is not set up on that device yet
  int sms = dev < 64 ? sm_count[dev].load(std::memory_order_acquire) : 0;
  if (sms == 0) {
    XKB_CHECK_CUDA(cudaFuncSetAttribute(moe_mx_kernel<BT, GATE_UP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)MxCfg<BT>::kSmemBytes));
    XKB_CHECK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    if (dev < 64) sm_count[dev].store(sms, std::memory_order_release);
  }
  XKB_REQUIRE(max_tiles < (1ll << 31), "moe_mx_kernel: %lld tiles do not fit the kernel's 31-bit tile index", (long long)max_tiles);
  int64_t grid = (int64_t)sms - g_sm_margin.load(std::memory_order_relaxed);
  if (grid < 8) grid = 8;
  if (grid > max_tiles) grid = max_tiles;
  if (grid < 1) grid = 1;
  XKB_CHECK_CUDA(launch_chained(moe_mx_kernel<BT, GATE_UP>, dim3((unsigned)grid), dim3(kThreads), MxCfg<BT>::kSmemBytes,
                                stream, tm[0], tm[1], tm[2], tm[3], tm[4], tm[5], prm));
  XKB_CHECK_LAUNCH("moe_mx_kernel");
  return XKB_OK;
}

template <bool GATE_UP>
int launch_mx_by_block(int block, const CUtensorMap (&tm)[6], const MxParams& prm, int64_t max_tiles, cudaStream_t stream) {
  switch (block) {
    case 8: return launch_mx<8, GATE_UP>(tm, prm, max_tiles, stream);
    case 16: return launch_mx<16, GATE_UP>(tm, prm, max_tiles, stream);
    case 32: return launch_mx<32, GATE_UP>(tm, prm, max_tiles, stream);
    default: return fail(XKB_ERR_ARG, "mxfp4 block-scaled path: unsupported token tile %d", block);
  }
}

struct MxBuffers {
  __nv_bfloat16* rows;
  uint8_t *x[kTerms + 1], *act[kTerms + 1];   // hi, mid, lo, scales of hi
};
MxBuffers carve_mx(Carver& c, int64_t numel, int64_t max_pad, int64_t hidden, int64_t ispp) {
  MxBuffers b;
  b.rows = c.take<__nv_bfloat16>(numel * hidden);
  for (int i = 0; i <= kTerms; ++i) b.x[i] = c.take<uint8_t>(max_pad * (i < kTerms ? hidden : hidden / 32));
  for (int i = 0; i <= kTerms; ++i) b.act[i] = c.take<uint8_t>(max_pad * (i < kTerms ? ispp : ispp / 32));
  return b;
}

int token_maps(CUtensorMap* tm, uint8_t* const (&x)[kTerms + 1], int64_t max_pad, int64_t K, int block) {
  for (int i = 0; i <= kTerms; ++i) {
    const bool sc = i == kTerms;
    const int rc = make_map_2d(&tm[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, 8, x[i], (uint64_t)max_pad, (uint64_t)(sc ? K / 32 : K),
                               (uint32_t)block, sc ? 16 : kStageK, sc ? CU_TENSOR_MAP_SWIZZLE_NONE : CU_TENSOR_MAP_SWIZZLE_128B,
                               sc ? "activation scales" : "activation terms");
    if (rc != XKB_OK) return rc;
  }
  return XKB_OK;
}

int weight_maps(CUtensorMap* tm, const uint8_t* w, const uint8_t* scale, int64_t rows, int64_t K, const char* what) {
  // sixteen nibbles per 16-byte container: what the instruction reads
  int rc = make_map_2d(&tm[0], CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B, 4, w, (uint64_t)rows, (uint64_t)K, kRows, kStageK,
                       CU_TENSOR_MAP_SWIZZLE_128B, what);
  if (rc != XKB_OK) return rc;
  return make_map_2d(&tm[1], CU_TENSOR_MAP_DATA_TYPE_UINT8, 8, scale, (uint64_t)rows, (uint64_t)K / 32, kRows, 16,
                     CU_TENSOR_MAP_SWIZZLE_NONE, what);
}

}  // namespace

bool mxfp4_bs_supported(const void* w13, const void* w2, const void* s13, const void* s2) {
  // the unpacking TMA type wants 32-byte bases (row pitches are whole multiples of 256 bytes)
  return ((reinterpret_cast<uintptr_t>(w13) | reinterpret_cast<uintptr_t>(w2)) & 31) == 0 &&
         ((reinterpret_cast<uintptr_t>(s13) | reinterpret_cast<uintptr_t>(s2)) & 15) == 0;
}

// A narrower tile is taken while a block still holds nearly every expert's slots (an expert that needs a second block
// streams its weights twice); 0 = the bf16 kernel's 128-token tiles, whose tokens are 2 bytes and not 3 and which multiply
// a block's slots only.  Whole calls in a loop, us at 16 / 32 / bf16; E=256, hidden 4096, ispp 512: 232 / 261 / 331 at 7
// slots per expert, 261 / 276 / 333 at 12, 370 / 294 / 352 at 19, 447 / 334 / 370 at 26, 513 / 424 / 391 at 33; E=128, 4096,
// 1024: 389 / 302 / 346 at 25, 514 / 444 / 373 at 38; E=64, 2048, 1024: 82 / 84 / 104 at 14, 120 / 99 / 109 at 28.  (64-token
// tiles of this kernel took 10 to 20 % longer than the bf16 kernel from 26 slots on: 417 us at 26, 430 at 33, 449 / 411 at 40.)
// 8 against 16 tokens (half the token bytes, one more stage of weights in flight): 32.9 / 36.9 us at M=1, 81 / 87 at M=16,
// 139 / 145 at one slot per expert (M=48), 199 / 212 at 3.5, 212 / 220 at 4.7, 240 / 239 at 9.4; E=128: 167 / 182 at 1.9.
int mxfp4_bs_block(int64_t numel, int E) {
  const double avg = (double)numel / (E > 0 ? E : 1);
  return avg <= 5 ? 8 : avg <= 12 ? 16 : avg <= 28 ? 32 : 0;
}

int64_t mxfp4_bs_workspace_bytes(int64_t numel, int64_t hidden, int64_t ispp, int E) {
  const int block = mxfp4_bs_block(numel, E);
  if (block == 0) return 0;
  Carver c(nullptr);
  carve_mx(c, numel, numel + (int64_t)(E + 1) * (block - 1), hidden, ispp);
  return c.off;
}

int launch_mxfp4_bs(const void* A, const uint8_t* w13, const uint8_t* w13_scale, const uint8_t* w2,
                    const uint8_t* w2_scale, const void* b13, const void* b2, const Routing& r, int64_t hidden,
                    int64_t ispp, int E, int top_k, float limit, void* ws, int* status, const __nv_bfloat16** rows_out,
                    cudaStream_t stream) {
  Carver carve(ws);
  const MxBuffers buf = carve_mx(carve, r.numel, r.max_pad, hidden, ispp);
  *rows_out = buf.rows;
  const __nv_bfloat16* a = static_cast<const __nv_bfloat16*>(A);
  const SplitRows x{buf.x[0], buf.x[1], buf.x[2], buf.x[kTerms]};
  GatherGrid g;
  int rc = gather_grid(r.numel / top_k, hidden / 8, r.job != nullptr, &g);
  if (rc != XKB_OK) return rc;
  if (r.job != nullptr) {
    const size_t smem = align::small_smem(r.job->E);
    if (smem > 48 * 1024)
      XKB_CHECK_CUDA(cudaFuncSetAttribute(gather_split_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    gather_split_kernel<true><<<g.blocks, g.threads, smem, stream>>>(a, nullptr, x, (int)hidden, top_k, r.max_pad, g.pieces,
                                                                     g.units, status, *r.job);
  } else if (r.by_position) {
    XKB_CHECK_CUDA(launch_chained(gather_split_positions_kernel, dim3(position_blocks(r.max_pad)), dim3(kGatherThreads), 0, stream,
                                  a, r.sorted_ids, r.num_post, x, r.numel, (int)hidden, top_k, r.max_pad, status));
  } else {
    XKB_CHECK_CUDA(launch_chained(gather_split_kernel<false>, dim3(g.blocks), dim3(g.threads), 0, stream, a, r.slot_pos, x,
                                  (int)hidden, top_k, r.max_pad, g.pieces, g.units, status, align::Job{}));
  }
  XKB_CHECK_LAUNCH("gather_split_kernel");

  CUtensorMap up[6], down[6];
  rc = weight_maps(up, w13, w13_scale, (int64_t)E * 2 * ispp, hidden, "w13");
  if (rc == XKB_OK) rc = token_maps(up + 2, buf.x, r.max_pad, hidden, r.block);
  if (rc == XKB_OK) rc = weight_maps(down, w2, w2_scale, (int64_t)E * hidden, ispp, "w2");
  if (rc == XKB_OK) rc = token_maps(down + 2, buf.act, r.max_pad, ispp, r.block);
  if (rc != XKB_OK) return rc;

  int32_t* done = r.block_counters;
  MxParams prm;
  prm.sorted_ids = r.sorted_ids;
  prm.expert_ids = r.expert_ids;
  prm.num_post = r.num_post;
  prm.status = status;
  prm.numel = r.numel;
  prm.max_blocks = (int)r.max_blocks;
  prm.num_experts = E;
  prm.bias = static_cast<const __nv_bfloat16*>(b13);
  for (int i = 0; i < kTerms; ++i) prm.act[i] = buf.act[i];
  prm.act_scale = buf.act[kTerms];
  prm.rows = nullptr;
  prm.N = (int)ispp;
  prm.K = (int)hidden;
  prm.rows_per_expert = (int)(2 * ispp);
  prm.mat_row = (int)ispp;
  prm.tile_step = kRows;
  prm.limit = limit;
  prm.done_signal = done;
  prm.done_wait = nullptr;
  prm.done_target = (int)(ispp / kRows) * 4 * (r.block <= 16 ? 1 : 2);
  GemmTimerScope timed(stream);   // both GEMMs in one scope: they overlap
  rc = launch_mx_by_block<true>(r.block, up, prm, r.max_blocks * (ispp / kRows), stream);
  if (rc != XKB_OK) return rc;
  prm.bias = static_cast<const __nv_bfloat16*>(b2);
  prm.rows = buf.rows;
  prm.N = (int)hidden;
  prm.K = (int)ispp;
  prm.rows_per_expert = (int)hidden;
  prm.mat_row = kRows;
  prm.tile_step = 2 * kRows;
  prm.limit = 0.f;
  prm.done_signal = nullptr;
  prm.done_wait = done;
  return launch_mx_by_block<false>(r.block, down, prm, r.max_blocks * (hidden / (2 * kRows)), stream);
}

}  // namespace xkb
