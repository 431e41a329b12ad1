// C = op(A^T B) at fp32 accuracy from scaled fp16 planes (gemm_half.h) on 5th-generation tensor cores.
//
// acc[m, n] = sum_k Za[k, m] * Zb[k, n], both operands K-contiguous.  Each fp32 value is a pair of fp16 numbers times a
// power of two, so a product is three fp16 MMAs, l*h + h*l + h*h (two, or one, where an operand comes from 16-bit values
// and has no l), against one tf32 MMA (half the fp16 rate) and two bf16 ones of the mixed form in gemm_tf32x3.cu: 3/4 of
// the tensor time, half the operand bytes, and a representation that is off by 2^-23 instead of 2^-20.
//
// Structure (192 KB of stages, one CTA per SM, 576 threads):
//   warp 0, one lane : TMA producer - up to four boxes of 128 rows x 64 fp16 (128-byte swizzle) per stage
//   warp 1, one lane : MMA issuer
//   warps 2..17      : promotion and epilogue
// PAIR: the two CTAs of a cluster share a 256 x 256 tile (cta_group::2, each stages its own 128 rows of A and half of the
// rows of B, no multicast); otherwise one CTA computes 128 x 128.  TMA zero-fills rows and K beyond the operands.
//
// The tensor core adds into its accumulator with truncation, so the accumulator is drained every 64 of K (one k-block) into
// a register-resident sum (round-to-nearest), multiplied by the scale of A's block of 128 on the way; B's scales are per
// column and applied once, in the epilogue.  Within a k-block the small products come first.
//
// What bounds a pair's tile of 256 x 256 (cycles, K = 4096, two-term operands): 98k of products at the tensor core's rate, some 5k over that
// between k-blocks, 8k from the start to the first full accumulator (barriers, TMEM, first loads), 5k to 10k of epilogue, and Adam's
// 20k and more where all tiles of a wave reach memory at once.  4096^3 331 -> 315 us, 8192^3 2334 -> 2251 (1.47 PFLOP/s: the power cap), Adam
// 8192^3 3003 -> 2617, 256 x 512 x 256 on single CTAs 15 -> 10 us, by draining with sixteen warps instead of eight (two columns per addition),
// looking ahead while products are issued, and fetching the epilogue's inputs meanwhile.  Accumulators of 128 columns, four in TMEM,
// hide the hand-over entirely but cost more than they hide on pairs (M 256 x N 128 products: 4096^3 391 us).
//
// Where the device word `wide` is set (RangeGuard: rows or columns that fp16 pairs do not hold) the same kernel runs the
// mixed form: four boxes of the same size, 32 of K each, tf32 and bf16 MMAs in gemm_tf32x3.cu's order, two k-blocks per drain,
// and bit for bit its results.  One launch serves both, so that nobody waits for the decision on the host.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <stdexcept>
#include <string>
#include <type_traits>

#include "gemm.h"
#include "gemm_half.h"
#include "launch_util.h"
#include "ptx.cuh"
#include "split_write.cuh"
#include "tensor_map.h"

namespace soapb200 {
namespace {

constexpr int kBM = 128;
constexpr int kBK = 64;                          // one 128-byte swizzle row of fp16
// One k-block per promotion, 64 of K, as the mixed form drains.  Truncated additions of a one-sided sum (a diagonal of
// squares, a rotation along a leading singular vector) all err to one side, and small products that meet a main sum are
// truncated at its size.  Relative error of products of positive operands, drained every 64 / every 128 / mixed form: two
// terms 2.7e-7 / 6.6e-7 / 4.6e-7 at K = 8192 and 2.1e-7 / 6.6e-7 / 4.5e-7 at K = 128, one term against two 2.1e-7 / 3.7e-7 /
// 3.1e-7 and 1.3e-7 / 3.6e-7 / 2.7e-7.  The price: two terms 4096^3 340 us instead of 319, one term against two 290 instead of 247.
constexpr int kScaleBlocks = kHalfScaleBlock / kBK;      // k-blocks that share one of A's scales
constexpr int kMixedBK = 32;                     // one 128-byte swizzle row of fp32, or of the interleaved bf16 plane
constexpr int kMixedDrain = 2;                   // its k-blocks per promotion
constexpr int kBoxBytes = 128 * kBK * 2;
constexpr int kStagePool = 12 * kBoxBytes;       // 3 stages of four boxes, 4 of three, 6 of two
constexpr int kMaxStages = 6;
constexpr int kEpiWarps = 16;
constexpr int kThreads = 64 + 32 * kEpiWarps;
constexpr int kScaleBytes = 256 * 4;              // B's scales of the tile's columns
constexpr int kSmemBytes = kStagePool + kScaleBytes + 1024 + 256;
// Between A's factor and B's the sums are kept 2^-16 below scale: B's planes are 2^14 and more above scale where B is of
// order one, and a large A must not overflow before B's factor brings the product back into range.
constexpr float kDown = 1.0f / 65536.0f, kUp = 65536.0f;

// What brings a column's sums back to scale: kUp and the column's scale in an order that rounds once.  A scale below one takes
// kUp in (together exact); above one it comes after kUp (both only enlarge a sum that is below the product).  Sums are about
// half as large as A's elements times their number, so bits are lost below 2^-124 only, where fp32 operands lose them too,
// and what overflows is A above 2^128 over that number.
struct ColumnFactor {
  float first, second;
  __device__ __forceinline__ explicit ColumnFactor(float scale = 0.f)
      : first(scale < 1.f ? scale * kUp : kUp), second(scale < 1.f ? 1.f : scale) {}
  __device__ __forceinline__ float operator()(float sum) const { return (sum * first) * second; }
};

struct alignas(64) HalfMaps {
  CUtensorMap a_h, a_l, b_h, b_l;
  CUtensorMap mixed[4];                          // A's tf32 values and corrections, B's: read where `wide` says so
};

struct HalfArgs {
  HalfProblem p;
  const float* a_scale;
  int64_t a_stride;
  const float* b_scale;
  int a_terms, b_terms;
};

// One CTA's way along K: k-blocks, stages, and drains of the accumulator.
struct KLoop {
  int blocks, drains, a_terms, b_terms, stages, stage_bytes, b_at;
  template <bool MIXED>
  __device__ __forceinline__ static KLoop over(const HalfArgs& args) {
    KLoop l;
    l.blocks = (args.p.K + (MIXED ? kMixedBK : kBK) - 1) / (MIXED ? kMixedBK : kBK);
    l.drains = MIXED ? (l.blocks + kMixedDrain - 1) / kMixedDrain : l.blocks;
    l.a_terms = MIXED ? 2 : args.a_terms;
    l.b_terms = MIXED ? 2 : args.b_terms;
    const int boxes = l.a_terms + l.b_terms;
    l.stages = 12 / boxes;                     // 3, 4 or 6 stages of four, three or two boxes
    l.stage_bytes = boxes * kBoxBytes;
    l.b_at = l.a_terms * kBoxBytes;            // a stage holds A's planes, then B's
    return l;
  }
};
static_assert(kMixedBK * kMixedDrain == kBK, "both forms drain as often");

constexpr int kUnroll = 4;       // columns per warp whose loads are in flight together
constexpr int kRowsPerLane = 4;  // a column of the tile is 128 rows: rows lane, lane + 32, lane + 64, lane + 96

// One column of the tile (four values per lane: rows 2 * lane, 2 * lane + 1, and those 64 further) as an operand of the next
// product, with the scale of its own 128 rows.
__device__ __forceinline__ void store_half_column(const HalfProblem& p, int m0, int n, int lane, const float (&v)[4]) {
  uint32_t most = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) most = max(most, __float_as_uint(v[i]) & 0x7fffffffu);
  const HalfScale s = half_scale(__reduce_max_sync(0xffffffffu, most));
  if (lane == 0) p.Cscale[(m0 / kHalfScaleBlock) * p.ldscale + n] = s.inverse;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int m = m0 + 64 * i + 2 * lane;
    if (m < p.M) {       // pitches are multiples of 64: the second half of a last odd row lands in the padding
      const float x0 = v[2 * i] * s.multiplier, x1 = v[2 * i + 1] * s.multiplier;
      const __half2 h = __floats2half2_rn(x0, x1);
      const float2 back = __half22float2(h);
      *reinterpret_cast<__half2*>(p.Ch + m + static_cast<int64_t>(n) * p.ldp) = h;
      *reinterpret_cast<__half2*>(p.Cl + m + static_cast<int64_t>(n) * p.ldp) = __floats2half2_rn(x0 - back.x, x1 - back.y);
    }
  }
}

// The same column as an operand in the mixed form.
__device__ __forceinline__ void store_mixed_column(const HalfProblem& p, int m0, int n, int lane, const float (&v)[4]) {
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int m = m0 + 64 * i + 2 * lane;
    if (m < p.M) write_split(p.mixed, true, m, n, p.M, v[2 * i], v[2 * i + 1], 1);
  }
}

__device__ __forceinline__ void store_column(const HalfProblem& p, bool wide, int m0, int n, int lane, const float (&v)[4]) {
  if (wide) store_mixed_column(p, m0, n, lane, v);
  else store_half_column(p, m0, n, lane, v);
}

// One line of L2 per lane: the epilogue's loads of what it reads back would otherwise all reach memory at the end of a wave of tiles
// (Adam, 8192^3: 3003 -> 2617 us).  Not the old result of symmetric products on pairs, whose loop is too short to hide it (one term,
// 4096: 123 us without, 145 with; on single CTAs 1024: 29 and 26).
template <int BN, int MODE>
__device__ __forceinline__ void prefetch_old(const HalfProblem& p, int m0, int n0, int ew, int lane) {
  auto columns = [&](const float* base, int64_t ld) {
    const int row = m0 + 32 * (lane & 3);
    for (int nl = 8 * ew + (lane >> 2); nl < BN; nl += 8 * kEpiWarps)
      if (row < p.M && n0 + nl < p.N) asm volatile("prefetch.global.L2 [%0];" ::"l"(base + row + static_cast<int64_t>(n0 + nl) * ld));
  };
  if constexpr (MODE == kEpiAdam) {
    columns(p.mom, p.ldm);
    columns(p.var, p.ldv);
  } else if constexpr (MODE == kEpiStore) {
    if (BN == 128 && p.beta != 0.f) columns(p.C, p.ldc);
  }
}

// Epilogue over the staged tile: tile[n_local * PITCH + m_local] holds sums 2^-16 below scale, without B's scales (`wide`: the
// sums themselves).  Accesses are four bytes per lane along M, so that no alignment of the outputs is needed, with kUnroll
// columns in flight.
template <int BN, int MODE, int PITCH>
__device__ __forceinline__ void half_epilogue(const HalfArgs& args, const float* column_scales, bool wide, float* tile, int m0, int n0,
                                              int ew, int lane) {
  const HalfProblem& p = args.p;
  const int rows = min(kBM, p.M - m0), cols = min(BN, p.N - n0);
  const float alpha = p.alpha;
  if constexpr (MODE == kEpiRowMajor) {
    ColumnFactor scaled[BN / 32];
#pragma unroll
    for (int j = 0; j < BN / 32; ++j) scaled[j] = ColumnFactor(column_scales[lane + 32 * j]);
    for (int r = ew; r < rows; r += kEpiWarps) {
      float* dst = p.C + static_cast<int64_t>(m0 + r) * p.ldc + n0;
#pragma unroll
      for (int j = 0; j < BN / 32; ++j) {
        const int n = lane + 32 * j;
        if (n < cols) dst[n] = alpha * scaled[j](tile[n * PITCH + r]);
      }
    }
  } else if constexpr (MODE == kEpiSplit) {
    for (int nl = ew; nl < cols; nl += kEpiWarps) {
      const ColumnFactor scaled(column_scales[nl]);
      float v[4];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float2 x = *reinterpret_cast<const float2*>(tile + nl * PITCH + 64 * i + 2 * lane);
        v[2 * i] = alpha * scaled(x.x);
        v[2 * i + 1] = alpha * scaled(x.y);
      }
      store_column(p, wide, m0, n0 + nl, lane, v);
    }
  } else if constexpr (MODE == kEpiAdam) {
    for (int base = ew * kUnroll; base < cols; base += kEpiWarps * kUnroll) {
      float mo[kUnroll][kRowsPerLane], va[kUnroll][kRowsPerLane];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int n = n0 + base + u;
        const bool here = base + u < cols;
#pragma unroll
        for (int i = 0; i < kRowsPerLane; ++i) {
          const int r = lane + 32 * i;
          const bool inside = here && r < rows;
          mo[u][i] = inside ? p.mom[m0 + r + static_cast<int64_t>(n) * p.ldm] : 0.f;
          va[u][i] = inside ? p.var[m0 + r + static_cast<int64_t>(n) * p.ldv] : 0.f;
        }
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        if (base + u >= cols) break;
        const int n = n0 + base + u;
        float* column = tile + (base + u) * PITCH;
        const ColumnFactor scaled(column_scales[base + u]);
#pragma unroll
        for (int i = 0; i < kRowsPerLane; ++i) {
          const int r = lane + 32 * i;
          const float g = alpha * scaled(column[r]);
          const float m_new = fmaf(p.beta1, mo[u][i], (1.0f - p.beta1) * g);
          const float v_new = fmaf(p.beta2, va[u][i], (1.0f - p.beta2) * g * g);
          float update = 0.f;
          if (r < rows) {
            p.mom[m0 + r + static_cast<int64_t>(n) * p.ldm] = m_new;
            p.var[m0 + r + static_cast<int64_t>(n) * p.ldv] = v_new;
            update = (m_new * p.inv_bc1) / (sqrtf(v_new) * p.inv_sqrt_bc2 + p.eps);
          }
          column[r] = update;
        }
        __syncwarp();
        float v[4];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float2 x = *reinterpret_cast<const float2*>(column + 64 * i + 2 * lane);
          v[2 * i] = x.x;
          v[2 * i + 1] = x.y;
        }
        store_column(p, wide, m0, n, lane, v);
      }
    }
  } else {
    // kEpiStore.  Symmetric: entries on and below the diagonal, whose final values go back into the tile for the mirror.
    for (int base = ew * kUnroll; base < cols; base += kEpiWarps * kUnroll) {
      float old[kUnroll][kRowsPerLane];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int n = n0 + base + u;
        const bool here = base + u < cols;
#pragma unroll
        for (int i = 0; i < kRowsPerLane; ++i) {
          const int r = lane + 32 * i;
          const bool wanted = here && p.beta != 0.f && r < rows && (!p.symmetric || n <= m0 + r);
          old[u][i] = wanted ? p.C[m0 + r + static_cast<int64_t>(n) * p.ldc] : 0.f;
        }
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int n = n0 + base + u;
        if (base + u >= cols) break;
        float* column = tile + (base + u) * PITCH;
        const ColumnFactor scaled(column_scales[base + u]);
#pragma unroll
        for (int i = 0; i < kRowsPerLane; ++i) {
          const int r = lane + 32 * i;
          if (r < rows && (!p.symmetric || n <= m0 + r)) {
            float v = alpha * scaled(column[r]);
            if (p.beta != 0.f) v = fmaf(p.beta, old[u][i], v);
            p.C[m0 + r + static_cast<int64_t>(n) * p.ldc] = v;
            if (p.symmetric) column[r] = v;
          }
        }
      }
    }
    if (p.symmetric) {
      // the mirror is written along its own rows: C[n, m] for the n < m of this tile, lanes along n
      asm volatile("bar.sync 1, %0;" ::"r"(kEpiWarps * 32) : "memory");
      for (int r = ew; r < rows; r += kEpiWarps) {
        const int m = m0 + r;
        const int limit = min(cols, m - n0);
        float* dst = p.C + static_cast<int64_t>(m) * p.ldc + n0;
        for (int n = lane; n < limit; n += 32) dst[n] = tile[n * PITCH + r];
      }
    }
  }
}

template <bool PAIR>
constexpr int kColumns = (PAIR ? 256 : 128) / (kEpiWarps / 4);      // of the tile, per epilogue thread

template <bool PAIR, typename Prefetch, typename Epilogue>
__device__ __forceinline__ void half_kernel_body(const HalfMaps& maps, const HalfArgs& args, int block, int* status, Prefetch prefetch,
                                                 Epilogue epilogue) {
  constexpr int BN = PAIR ? 256 : 128;
  constexpr int kCtas = PAIR ? 2 : 1;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* column_scales = reinterpret_cast<float*>(smem + kStagePool);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + kStagePool + kScaleBytes);      // PAIR: used in the leader CTA only
  uint64_t* empty_bar = full_bar + kMaxStages;      // each CTA its own: "my stage may be refilled"
  uint64_t* acc_full = empty_bar + kMaxStages;      // [2] each CTA its own: tensor core -> epilogue
  uint64_t* acc_empty = acc_full + 2;               // [2] PAIR: leader's only, epilogue warps of both CTAs -> tensor core
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const HalfProblem& prob = args.p;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t cta = PAIR ? cluster_cta_rank() : 0;

  // Grouped raster: kGroup tile-rows share their B panels in L2 while they sweep the tile columns.
  constexpr int kTileM = kCtas * kBM;
  constexpr int kGroup = PAIR ? 8 : 16;
  const int tiles_m = (prob.M + kTileM - 1) / kTileM;
  const int tiles_n = (prob.N + BN - 1) / BN;
  const int index = PAIR ? block >> 1 : block;
  const int per_group = kGroup * tiles_n;
  const int first_m = index / per_group * kGroup;
  const int rows_in_group = min(kGroup, tiles_m - first_m);
  const int tile_m0 = (first_m + index % per_group % rows_in_group) * kTileM;
  const int m0 = tile_m0 + static_cast<int>(cta) * kBM;      // this CTA's rows of the result
  const int n0 = index % per_group / rows_in_group * BN;
  const int b_row0 = n0 + static_cast<int>(cta) * (BN / kCtas);
  // symmetric products: tiles strictly above the diagonal are produced by mirroring (same decision in both CTAs)
  if (prob.symmetric && n0 > min(tile_m0 + kTileM, prob.M) - 1) {
    wait_for_predecessor();      // (no part of this grid ends before its predecessor has)
    return;
  }

  if (threadIdx.x == 0) {
    for (int s = 0; s < kMaxStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], kCtas * kEpiWarps);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_descriptor(&maps.a_h);
    tma_prefetch_descriptor(&maps.b_h);
    if (args.a_terms == 2) tma_prefetch_descriptor(&maps.a_l);
    if (args.b_terms == 2) tma_prefetch_descriptor(&maps.b_l);
  }
  if (warp == 1) {
    if constexpr (PAIR) {
      tmem_alloc_pair(tmem_slot, 2 * BN);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(tmem_slot, 2 * BN);
      tmem_relinquish();
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if constexpr (PAIR) cluster_sync_all();      // both CTAs' barriers exist before anything arrives on them remotely
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  // The same in every CTA.  Where the decision is older than the kernel ahead -- which waited for the one that made it before
  // it let this one start -- it is read while that one still runs.
  auto decision = [&] { return prob.wide && *static_cast<const volatile int*>(prob.wide); };
  bool wide = prob.settled && decision();
  wait_for_predecessor();
  let_successor_start();
  if (!prob.settled) wide = decision();


  // The roles, for either form.
  auto produce = [&](auto mixed) {
    // ---------------- TMA producer (each CTA loads its own tiles; PAIR: the bytes are credited to the leader) ----------------
    constexpr bool kMixed = decltype(mixed)::value;
    const KLoop loop = KLoop::over<kMixed>(args);
    const CUtensorMap* a_first = kMixed ? &maps.mixed[0] : &maps.a_h;
    const CUtensorMap* a_second = kMixed ? &maps.mixed[1] : &maps.a_l;
    const CUtensorMap* b_first = kMixed ? &maps.mixed[2] : &maps.b_h;
    const CUtensorMap* b_second = kMixed ? &maps.mixed[3] : &maps.b_l;
    int s = 0;
    uint32_t parity = 1;                       // of the previous round's release
    for (int kb = 0; kb < loop.blocks; ++kb) {
      if (kb >= loop.stages && !mbar_wait_bounded(&empty_bar[s], parity, abort_flag, status, kStatusSlotWaitTimeout)) break;
      uint8_t* stage = smem + s * loop.stage_bytes;
      const int k0 = kb * (kMixed ? kMixedBK : kBK), k1 = kb * kBK;        // the interleaved plane has 64 elements per 32 of K
      if constexpr (PAIR) {
        if (cta == 0) mbar_expect_tx(&full_bar[s], 2 * loop.stage_bytes);
        const uint32_t bar = map_to_cta(smem_u32(&full_bar[s]), 0);
        tma_load_2d_pair(stage, a_first, bar, k0, m0);
        if (loop.a_terms == 2) tma_load_2d_pair(stage + kBoxBytes, a_second, bar, k1, m0);
        tma_load_2d_pair(stage + loop.b_at, b_first, bar, k0, b_row0);
        if (loop.b_terms == 2) tma_load_2d_pair(stage + loop.b_at + kBoxBytes, b_second, bar, k1, b_row0);
      } else {
        mbar_expect_tx(&full_bar[s], loop.stage_bytes);
        tma_load_2d(stage, a_first, &full_bar[s], k0, m0);
        if (loop.a_terms == 2) tma_load_2d(stage + kBoxBytes, a_second, &full_bar[s], k1, m0);
        tma_load_2d(stage + loop.b_at, b_first, &full_bar[s], k0, b_row0);
        if (loop.b_terms == 2) tma_load_2d(stage + loop.b_at + kBoxBytes, b_second, &full_bar[s], k1, b_row0);
      }
      if (++s == loop.stages) {
        s = 0;
        parity ^= 1;
      }
    }
    if (*abort_flag) {
      // give copies that are still in flight time to land before the CTA's shared memory is released
      for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    }
  };

  auto issue = [&](auto mixed) {
    // ---------------- MMA issuer (PAIR: leader CTA only) ----------------
    constexpr bool kMixed = decltype(mixed)::value;
    const KLoop loop = KLoop::over<kMixed>(args);
    constexpr uint32_t idesc16 = kMixed ? umma_idesc_bf16(kCtas * kBM, BN) : umma_idesc_fp16(kCtas * kBM, BN);
    constexpr uint32_t idesc32 = umma_idesc_tf32(kCtas * kBM, BN);
    auto mma16 = [&](uint32_t acc, uint64_t a, uint64_t b, uint32_t accumulate) {
      if constexpr (PAIR) umma_f16_ss_pair(acc, a, b, idesc16, accumulate);
      else umma_f16_ss(acc, a, b, idesc16, accumulate);
    };
    auto mma32 = [&](uint32_t acc, uint64_t a, uint64_t b, uint32_t accumulate) {
      if constexpr (PAIR) umma_tf32_ss_pair(acc, a, b, idesc32, accumulate);
      else umma_tf32_ss(acc, a, b, idesc32, accumulate);
    };
    auto commit = [&](uint64_t* bar) {
      if constexpr (PAIR) umma_commit_pair(bar);
      else umma_commit(bar);
    };
    bool ok = true;
    int s = 0, kb = 0;
    uint32_t parity = 0;
    // Whether the next k-block's operands and accumulator are there is looked up while this one's products are still being issued:
    // a wait between two k-blocks, however short, drains the tensor core's queue of a few products (350 of 1860 cycles of a k-block).
    bool loaded = false, drained = false;
    for (int d = 0; d < loop.drains; ++d) {
      const int buf = d & 1;
      if (d >= 2) {
        ok = drained || mbar_wait_bounded(&acc_empty[buf], ((d >> 1) - 1) & 1, abort_flag, status, kStatusAccumWaitTimeout);
        if (!ok) break;
        tc_fence_after_sync();
      }
      const uint32_t acc = tmem_base + static_cast<uint32_t>(buf * BN);
      uint32_t more = 0;                       // 0: the first product since the last drain overwrites the accumulator
#pragma unroll
      for (int i = 0; i < (kMixed ? kMixedDrain : 1); ++i, ++kb) {
        if (kMixed && kb == loop.blocks) break;
        ok = loaded || mbar_wait_bounded(&full_bar[s], parity, abort_flag, status, kStatusTmaWaitTimeout);
        if (!ok) break;
        tc_fence_after_sync();
        auto look_ahead = [&] {
          const int next = s + 1 == loop.stages ? 0 : s + 1;
          loaded = kb + 1 < loop.blocks && mbar_test(&full_bar[next], next ? parity : parity ^ 1);
          drained = d >= 1 && d + 1 < loop.drains && mbar_test(&acc_empty[buf ^ 1], (((d + 1) >> 1) - 1) & 1);
        };
        const uint32_t stage = smem_u32(smem + s * loop.stage_bytes);
        const uint64_t a_0 = umma_desc_kmajor<128>(stage);
        const uint64_t b_0 = umma_desc_kmajor<128>(stage + loop.b_at);
        constexpr uint64_t kSecond = kBoxBytes >> 4, kStep = 32 >> 4;      // 16 fp16 or 8 fp32 = 32 bytes along the swizzle row
        if constexpr (kMixed) {
          constexpr uint64_t kLb = 64 >> 4;    // lb follows hb in a row of the interleaved plane
          const bool main_first = kb & 1;      // one change of the MMAs' kind per k-block
          if (main_first) {
#pragma unroll
            for (int k = 0; k < kMixedBK / 8; ++k, more = 1) mma32(acc, a_0 + k * kStep, b_0 + k * kStep, more);
          }
#pragma unroll
          for (int k = 0; k < kMixedBK / 16; ++k, more = 1) {
            const uint64_t a_1 = a_0 + kSecond + k * kStep, b_1 = b_0 + kSecond + k * kStep;
            mma16(acc, a_1 + kLb, b_1, more);                                                                          // lb * hb
            mma16(acc, a_1, b_1 + kLb, 1);                                                                             // hb * lb
          }
          look_ahead();
          if (!main_first) {
#pragma unroll
            for (int k = 0; k < kMixedBK / 8; ++k) mma32(acc, a_0 + k * kStep, b_0 + k * kStep, 1);
          }
        } else {
          if (loop.a_terms == 2) {
#pragma unroll
            for (int k = 0; k < kBK / 16; ++k, more = 1) mma16(acc, a_0 + kSecond + k * kStep, b_0 + k * kStep, more);  // l * h
          }
          if (loop.b_terms == 2) {
#pragma unroll
            for (int k = 0; k < kBK / 16; ++k, more = 1) mma16(acc, a_0 + k * kStep, b_0 + kSecond + k * kStep, more);  // h * l
          }
          look_ahead();
#pragma unroll
          for (int k = 0; k < kBK / 16; ++k, more = 1) mma16(acc, a_0 + k * kStep, b_0 + k * kStep, more);              // h * h
        }
        commit(&empty_bar[s]);                 // the stage may be refilled once these products have read it
        if (++s == loop.stages) {
          s = 0;
          parity ^= 1;
        }
      }
      if (!ok) break;
      commit(&acc_full[buf]);
    }
  };

  if (warp == 0 && lane == 0) {
    if (wide) produce(std::true_type{});
    else produce(std::false_type{});
  } else if (warp == 1 && lane == 0 && cta == 0) {
    if (wide) issue(std::true_type{});
    else issue(std::false_type{});
  } else if (warp >= 2) {
    // ---------------- promotion + epilogue (each CTA its own 128 rows) ----------------
    const int ew = warp - 2;
    const int quarter = warp & 3;              // TMEM lane quarter this warp may read
    constexpr int kCols = kColumns<PAIR>;      // of the tile, per thread
    const int col0 = (ew >> 2) * kCols;
    // What the epilogue reads is fetched while the products run: B's scales into shared memory, and what it reads back into L2.
    for (int n = threadIdx.x - 64; n < BN; n += 32 * kEpiWarps)
      column_scales[n] = wide || n0 + n >= prob.N ? kDown : args.b_scale[n0 + n];      // kDown undoes kUp: a factor of one
    prefetch(m0, n0, ew, lane);
    const float* a_scale = args.a_scale + min(m0 + quarter * 32 + lane, prob.M - 1);     // this thread's row
    const uint32_t drained = PAIR ? map_to_cta(smem_u32(&acc_empty[0]), 0) : 0;
    uint64_t sum[kCols / 2];                   // pairs of neighbouring columns
#pragma unroll
    for (int j = 0; j < kCols / 2; ++j) sum[j] = 0;
    const int64_t a_stride = wide ? 0 : args.a_stride;
    const int drains = (prob.K + kBK - 1) / kBK;         // of either form
    float scale = wide ? 1.0f : *a_scale * kDown;
    for (int d = 0; d < drains; ++d) {
      const int buf = d & 1;
      // the next k-block's scale travels while this one is waited for
      const float next = a_stride ? a_scale[min(d + 1, drains - 1) / kScaleBlocks * a_stride] * kDown : scale;
      if (!mbar_wait_bounded(&acc_full[buf], (d >> 1) & 1, abort_flag, status, kStatusAccumWaitTimeout)) break;
      tc_fence_after_sync();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(buf * BN + col0);
      const uint64_t scales = pack_floats(scale, scale);
#pragma unroll
      for (int cc = 0; cc < kCols; cc += 16) {
        uint32_t raw[16];
        tmem_ld_32x16(taddr + static_cast<uint32_t>(cc), raw);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j) fma_pair(sum[cc / 2 + j], pack_pair(raw[2 * j], raw[2 * j + 1]), scales);
      }
      scale = next;
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        if constexpr (PAIR) mbar_arrive_cluster(drained + static_cast<uint32_t>(buf * sizeof(uint64_t)));
        else mbar_arrive(&acc_empty[buf]);
      }
    }
    // The stages are idle once the accumulator has been drained for the last time: the sums are staged there and the epilogue runs as a
    // compact rolled loop over the tile.
    epilogue(reinterpret_cast<float*>(smem), column_scales, wide, sum, col0, quarter * 32 + lane, abort_flag, m0, n0, ew, lane);
  }

  tc_fence_before_sync();
  __syncthreads();
  if constexpr (PAIR) cluster_sync_all();      // nobody leaves while the other CTA may still touch its shared memory or TMEM
  if (warp == 1) {
    tc_fence_after_sync();
    if constexpr (PAIR) tmem_dealloc_pair(tmem_base, 2 * BN);
    else tmem_dealloc(tmem_base, 2 * BN);
  }
}

// Column pitch of the staged tile in floats: odd where columns are read across (row-major and mirrored stores), even where
// two neighbouring rows are read as one 8-byte word.
template <int MODE>
constexpr int kPitch = (MODE == kEpiSplit || MODE == kEpiAdam) ? kBM + 2 : kBM + 1;
static_assert(256 * (kBM + 2) * 4 <= kStagePool, "the staged tile fits where the stages were");

template <bool PAIR, int MODE>
__device__ __forceinline__ void half_kernel_impl(const HalfMaps& maps, const HalfArgs& args, int block, int* status) {
  constexpr int BN = PAIR ? 256 : 128;
  half_kernel_body<PAIR>(maps, args, block, status, [&](int m0, int n0, int ew, int lane) { prefetch_old<BN, MODE>(args.p, m0, n0, ew, lane); },
                         [&](float* tile, const float* column_scales, bool wide, uint64_t (&sum)[kColumns<PAIR> / 2], int col0, int row, volatile int* abort_flag,
                                                 int m0, int n0, int ew, int lane) {
#pragma unroll
    for (int j = 0; j < kColumns<PAIR>; ++j) tile[(col0 + j) * kPitch<MODE> + row] = pair_element(sum[j / 2], j & 1);
    asm volatile("bar.sync 1, %0;" ::"r"(kEpiWarps * 32) : "memory");
    // read after the barrier, so that all warps of the CTA agree (the epilogue has a barrier of its own)
    if (*abort_flag == 0 && m0 < args.p.M) half_epilogue<BN, MODE, kPitch<MODE>>(args, column_scales, wide, tile, m0, n0, ew, lane);
  });
}

template <int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
half_pair_kernel(const __grid_constant__ HalfMaps maps, const __grid_constant__ HalfArgs args, int* status) {
  half_kernel_impl<true, MODE>(maps, args, blockIdx.x, status);
}

// N products of single CTAs in one launch, one after another in the grid.  (With N = 1 the search for the problem is compiled away; the
// parameters of eight take 11 KB, which a launch of one does not pay for.)
template <int N>
struct HalfGroup {
  HalfMaps maps[N];
  HalfArgs args[N];
  GroupBlocks<N> blocks;
};

template <int MODE, int N>
__global__ void __launch_bounds__(kThreads, 1)
half_single_kernel(const __grid_constant__ HalfGroup<N> group, int* status) {
  const int member = group.blocks.member(blockIdx.x);
  half_kernel_impl<false, MODE>(group.maps[member], group.args[member], blockIdx.x - group.blocks.first(member), status);
}

// ---------------------------------------------------------------------------------------------
// K-contiguous fp16 plane [rows][K] with row pitch ld: boxes of 64 elements x 128 rows.
CUtensorMap make_map(const uint16_t* base, int64_t K, int64_t rows, int64_t ld) {
  if (ld % 64 != 0 || ld < K) throw std::invalid_argument("gemm_half: planes need a pitch that is a multiple of 64 covering K");
  return encode_k_major(CU_TENSOR_MAP_DATA_TYPE_FLOAT16, base, K, rows, 2 * ld, kBK, 128, CU_TENSOR_MAP_SWIZZLE_128B);
}

int single_tiles(const HalfProblem& p) { return ((p.M + kBM - 1) / kBM) * ((p.N + 127) / 128); }

template <int MODE, int N>
cudaError_t launch_singles(const HalfMaps* maps, const HalfArgs* args, int count, int* status, cudaStream_t stream) {
  static PerDeviceOnce configured;
  allow_dynamic_smem(reinterpret_cast<const void*>(half_single_kernel<MODE, N>), kSmemBytes, configured, "gemm_half");
  HalfGroup<N> group;
  for (int i = 0; i < count; ++i) {
    group.maps[i] = maps[i];
    group.args[i] = args[i];
    group.blocks.add(single_tiles(args[i].p));
  }
  return launch_dependent(half_single_kernel<MODE, N>, dim3(group.blocks.total()), dim3(kThreads), kSmemBytes, stream, group, status);
}

template <int MODE>
void launch(bool pairs, const HalfMaps* maps, const HalfArgs* args, int count, int* status, cudaStream_t stream) {
  cudaError_t err;
  if (pairs) {
    static PerDeviceOnce configured;
    allow_dynamic_smem(reinterpret_cast<const void*>(half_pair_kernel<MODE>), kSmemBytes, configured, "gemm_half");
    const HalfProblem& p = args->p;
    const int tiles = ((p.M + 2 * kBM - 1) / (2 * kBM)) * ((p.N + 255) / 256);
    err = launch_dependent(half_pair_kernel<MODE>, dim3(2 * tiles), dim3(kThreads), kSmemBytes, stream, *maps, *args, status);
  } else {
    err = count == 1 ? launch_singles<MODE, 1>(maps, args, count, status, stream)
                     : launch_singles<MODE, kHalfGroup>(maps, args, count, status, stream);
  }
  if (err != cudaSuccess) throw std::runtime_error(std::string("gemm_half launch: ") + cudaGetErrorString(err));
}

void launch_mode(bool pairs, const HalfMaps* maps, const HalfArgs* args, int count, int* status, cudaStream_t stream) {
  switch (args->p.mode) {
    case kEpiStore: launch<kEpiStore>(pairs, maps, args, count, status, stream); return;
    case kEpiSplit: launch<kEpiSplit>(pairs, maps, args, count, status, stream); return;
    case kEpiAdam: launch<kEpiAdam>(pairs, maps, args, count, status, stream); return;
    case kEpiRowMajor: launch<kEpiRowMajor>(pairs, maps, args, count, status, stream); return;
    default: throw std::invalid_argument("gemm_half: unknown epilogue mode");
  }
}

}  // namespace

void half_maps(CUtensorMap (&maps)[2], const uint16_t* h, const uint16_t* l, int64_t ld, int64_t K, int64_t cols) {
  maps[0] = make_map(h, K, cols, ld);
  maps[1] = l ? make_map(l, K, cols, ld) : maps[0];
}

void mixed_maps(CUtensorMap (&maps)[2], const SplitTarget& planes, int64_t K, int64_t cols) {
  maps[0] = encode_k_major(CU_TENSOR_MAP_DATA_TYPE_FLOAT32, planes.hi, K, cols, 4 * planes.ldo, kMixedBK, 128, CU_TENSOR_MAP_SWIZZLE_128B);
  maps[1] = encode_interleaved(planes.hl, K, cols, planes.ld16, 2 * kMixedBK, 128);
}

bool half_fills_pairs(int M, int N, bool symmetric) {
  // A pair's 256 x 256 tile takes about 1.5 times as long as a CTA's 128 x 128 one (it loads half as much per product): pairs
  // unless single CTAs get by with so few waves that they finish earlier.  Pairs against singles, two terms: 1024^3 27 and
  // 20 us, 1536^3 34 and 27, 1792^3 40 and 58, 2048^3 44 and 64, 3072^3 132 and 178, 4096^3 319 and 409; symmetric, two terms and one: 1024
  // 30 and 22, 26 and 17; 2048 46 and 39, 37 and 29; 3072 130 and 140, 96 and 97; 4096 196 and 267, 143 and 191.
  auto tiles_of = [&](int64_t side) {
    const int64_t m = (M + side - 1) / side, n = (N + side - 1) / side;
    return symmetric ? m * (m + 1) / 2 : m * n;
  };
  return 3 * ((tiles_of(256) + 73) / 74) <= 2 * ((tiles_of(128) + 147) / 148);
}

bool half_on_pairs(int M, int N, bool symmetric) { return gemm_cta_pairs_wanted() && half_fills_pairs(M, N, symmetric); }

namespace {
// Checks a product and fills what its kernel reads.
void prepare(const HalfOperand& a, const HalfOperand& b, const HalfProblem& prob, HalfMaps& maps, HalfArgs& args) {
  if (prob.K <= 0) throw std::invalid_argument("gemm_half needs K >= 1");
  if (b.scale_stride != 0) throw std::invalid_argument("gemm_half: the second operand has one scale per column");
  if (prob.symmetric && (prob.mode != kEpiStore || prob.M != prob.N))
    throw std::invalid_argument("gemm_half: symmetric results are square and stored plainly");
  const bool to_planes = prob.mode == kEpiSplit || prob.mode == kEpiAdam;
  if (to_planes && (!prob.Ch || !prob.Cl || !prob.Cscale || prob.ldp % 64 != 0 || prob.ldp < prob.M ||
                    (reinterpret_cast<uintptr_t>(prob.Ch) & 15) != 0 || (reinterpret_cast<uintptr_t>(prob.Cl) & 15) != 0))
    throw std::invalid_argument("gemm_half: output planes need 16-byte alignment and a pitch that is a multiple of 64");
  if (prob.wide) {
    if (!a.mixed || !b.mixed) throw std::invalid_argument("gemm_half: a decided product needs both operands' mixed form");
    if (to_planes && (!prob.mixed.hi || !prob.mixed.hl || prob.mixed.ldo < prob.M || prob.mixed.ld16 < bf16_plane_index(prob.M - 1) + 33 ||
                      !writes_pairs(prob.mixed)))
      throw std::invalid_argument("gemm_half: mixed output planes need 8-byte alignment and an even pitch");
  }
  CUtensorMap made[2];
  if (!a.maps) half_maps(made, a.h, a.l, a.ld, prob.K, prob.M);
  maps.a_h = a.maps ? a.maps[0] : made[0];
  maps.a_l = a.maps ? a.maps[1] : made[1];
  if (!b.maps) half_maps(made, b.h, b.l, b.ld, prob.K, prob.N);
  maps.b_h = b.maps ? b.maps[0] : made[0];
  maps.b_l = b.maps ? b.maps[1] : made[1];
  if (prob.wide) {
    for (int i = 0; i < 2; ++i) {
      maps.mixed[i] = a.mixed[i];
      maps.mixed[2 + i] = b.mixed[i];
    }
  }
  args = HalfArgs{prob, a.scale, a.scale_stride, b.scale, a.l ? 2 : 1, b.l ? 2 : 1};
}
}  // namespace

void gemm_half(const HalfOperand& a, const HalfOperand& b, const HalfProblem& prob, int* status, cudaStream_t stream) {
  if (prob.M <= 0 || prob.N <= 0) return;
  HalfMaps maps;
  HalfArgs args;
  prepare(a, b, prob, maps, args);
  const bool pairs = prob.tiles ? prob.tiles == 2 : half_on_pairs(prob.M, prob.N, prob.symmetric);
  launch_mode(pairs, &maps, &args, 1, status, stream);
}

void gemm_half_group(const HalfJob* jobs, int count, int* status, cudaStream_t stream) {
  if (count < 1 || count > kHalfGroup) throw std::invalid_argument("gemm_half: too many products for one launch");
  HalfMaps maps[kHalfGroup];
  HalfArgs args[kHalfGroup];
  for (int i = 0; i < count; ++i) {
    if (jobs[i].problem.M <= 0 || jobs[i].problem.N <= 0 || jobs[i].problem.mode != jobs[0].problem.mode)
      throw std::invalid_argument("gemm_half: products of one launch are not empty and end in the same epilogue");
    prepare(jobs[i].a, jobs[i].b, jobs[i].problem, maps[i], args[i]);
  }
  launch_mode(false, maps, args, count, status, stream);
}

}  // namespace soapb200
