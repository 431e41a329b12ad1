// Panel factorisation that retires TWO Householder columns per all-to-all exchange.
//
// The one-column kernel (qr.cu) is bound by its chain of exchanges: per column one sweep of dot
// products, one exchange between the CTAs, one update sweep.  Here a step takes the pivot columns
// x = a_c and y = a_{c+1} together:
//
//   sweep 1   D1_j = x . a_j and D2_j = y . a_j for every column j (one pass over the registers)
//   exchange  sums of D1, D2 over the CTAs and the pivot-row entries p1_j = a_j[c], p2_j = a_j[c+1]
//   scalars   H_c from (p1_c, D1_c) as before.  Everything H_{c+1} needs follows WITHOUT touching the
//             data again, because H_c is orthogonal:  with k = tau_c (v_c . y) and y' = H_c y,
//               y'[c]   = p1_{c+1} - k                      y'[c+1] = p2_{c+1} - k s_c p2_c
//               |y'|^2 over rows > c        = D2_{c+1} - y'[c]^2
//               y' . (H_c a_j) over rows >= c = D2_j
//             so v_{c+1} . (H_c a_j), the entries of V^T V that the compact-WY factor needs, and the
//             coefficients of the rank-2 update are per-column arithmetic on (D1_j, D2_j, p1_j, p2_j).
//   sweep 2   a_j <- a_j - A_j x - B_j y   (one pass), next two pivot columns published
//
// The subtraction D2_{c+1} - y'[c]^2 cancels when y is nearly parallel to x (rank-deficient input,
// repeated columns).  The step then retires column c only -- the decision is taken from exchanged
// sums that are bitwise identical on every CTA -- and column c + 1 becomes the next step's x, so
// the worst case is the one-column algorithm.  With the guard at half of |y|^2, rank-deficient,
// graded and duplicated inputs keep the orthogonality of Q at the one-column kernel's level (the NumPy
// restatement in utils/panel_pairs_reference.py shows 1e-3 without a guard, 2e-5 with a guard of 0.05).
//
// Bound by a chain of 64 steps of some 6900 cycles (5 CTAs that exchange through L2; 9700 with 33): the exchange 1800 (4300), sweep 1
// 1200, pivot entries and publishing 1100, scalars and coefficients 1000, sweep 2 1200.  A warp owns one slice of 32 columns: a 16-byte
// load of a pivot column is then one address for all lanes, 1.55 cycles of shared memory instead of the 2.2 that four slices in a
// warp took (sweep 1 was 2130 cycles).  Panels of 1024 / 3000 / 8192 rows, exchanging through L2: 324 / 329 / 411 us with four slices
// a warp, element-wise loads and outputs staged through shared memory; 263 / 285 / 364 us so.  (As a cluster, see kCluster: 230 / 280.)
//
// Exchange words ({value, sequence} in 64 bits, bounded polls) are those of qr.cu.  T is built in the shadow of the exchange by the last
// CTA, which has no rows of its own where a launch has more than one and room for one more.
#include <cuda_runtime.h>

#include <atomic>
#include <stdexcept>
#include <string>

#include "ptx.cuh"
#include "qr.h"
#include "qr_device.cuh"

namespace soapb200 {
namespace {

using namespace qrdev;

constexpr float kPairThreshold = 0.5f;    // |y'|^2 / |y|^2 below which the second column waits for the next step

// Extract (and optionally retire) entry `k` of a thread's register slice; `k` is warp-uniform, so the
// switch is one indirect branch instead of a chain of predicated selects.
#define SOAP_ENTRY_CASE(K) case K: if (K < kPer) { value = P[K < kPer ? K : 0]; if (clear) P[K < kPer ? K : 0] = 0.f; } break;
template <int kPer>
__device__ __forceinline__ float take_entry(float (&P)[kPer], int k, bool clear) {
  float value = 0.f;
  switch (k) {
    SOAP_ENTRY_CASE(0) SOAP_ENTRY_CASE(1) SOAP_ENTRY_CASE(2) SOAP_ENTRY_CASE(3) SOAP_ENTRY_CASE(4) SOAP_ENTRY_CASE(5)
    SOAP_ENTRY_CASE(6) SOAP_ENTRY_CASE(7) SOAP_ENTRY_CASE(8) SOAP_ENTRY_CASE(9) SOAP_ENTRY_CASE(10) SOAP_ENTRY_CASE(11)
    SOAP_ENTRY_CASE(12) SOAP_ENTRY_CASE(13) SOAP_ENTRY_CASE(14) SOAP_ENTRY_CASE(15) SOAP_ENTRY_CASE(16) SOAP_ENTRY_CASE(17)
    SOAP_ENTRY_CASE(18) SOAP_ENTRY_CASE(19) SOAP_ENTRY_CASE(20) SOAP_ENTRY_CASE(21) SOAP_ENTRY_CASE(22) SOAP_ENTRY_CASE(23)
    SOAP_ENTRY_CASE(24) SOAP_ENTRY_CASE(25) SOAP_ENTRY_CASE(26) SOAP_ENTRY_CASE(27) SOAP_ENTRY_CASE(28) SOAP_ENTRY_CASE(29)
    SOAP_ENTRY_CASE(30) SOAP_ENTRY_CASE(31) SOAP_ENTRY_CASE(32) SOAP_ENTRY_CASE(33) SOAP_ENTRY_CASE(34) SOAP_ENTRY_CASE(35)
    SOAP_ENTRY_CASE(36) SOAP_ENTRY_CASE(37) SOAP_ENTRY_CASE(38) SOAP_ENTRY_CASE(39) SOAP_ENTRY_CASE(40) SOAP_ENTRY_CASE(41)
    SOAP_ENTRY_CASE(42) SOAP_ENTRY_CASE(43) SOAP_ENTRY_CASE(44) SOAP_ENTRY_CASE(45) SOAP_ENTRY_CASE(46) SOAP_ENTRY_CASE(47)
    SOAP_ENTRY_CASE(48) SOAP_ENTRY_CASE(49) SOAP_ENTRY_CASE(50) SOAP_ENTRY_CASE(51) SOAP_ENTRY_CASE(52) SOAP_ENTRY_CASE(53)
    SOAP_ENTRY_CASE(54) SOAP_ENTRY_CASE(55) SOAP_ENTRY_CASE(56) SOAP_ENTRY_CASE(57) SOAP_ENTRY_CASE(58) SOAP_ENTRY_CASE(59)
    SOAP_ENTRY_CASE(60) SOAP_ENTRY_CASE(61) SOAP_ENTRY_CASE(62) SOAP_ENTRY_CASE(63)
    default: break;
  }
  return value;
}
#undef SOAP_ENTRY_CASE

__device__ __forceinline__ unsigned long long pack_word(float value, unsigned int seq) {
  return (static_cast<unsigned long long>(seq) << 32) | __float_as_uint(value);
}

// Where a compiler could round once or twice (the sum of two products, a square that is used twice) the operations are spelled
// out: the sign of a basis's last column hangs on the last bits of what comes before it, and must not change with the code around.
__device__ __forceinline__ void householder_scalars(float alpha, float normsq, float& tau, float& scale) {
  tau = 0.f;
  scale = 0.f;
  const float tail = __fsub_rn(normsq, __fmul_rn(alpha, alpha));
  if (tail > 0.f && normsq > 0.f) {
    const float beta = -copysignf(sqrtf(normsq), alpha);
    tau = (beta - alpha) * __frcp_rn(beta);
    scale = __frcp_rn(alpha - beta);
  }
}

// kPer rows of one column per thread: 64 (256-row CTAs, fewest SMs) or 32 (128-row CTAs: the sweeps are bound
// by shared-memory load latency, and with half the registers taken by the slab every load of a sweep can be in
// flight at once).
// kCluster: up to sixteen CTAs (3840 rows), or eight where the device takes no larger cluster, are one cluster and write their sums into
// each other's shared memory instead of polling words in global memory; the same values are added in the same order.  Panels of
// 300 / 1024 / 2048 / 3000 rows 257 / 262 / 275 / 288 us by polling, 214 / 229 / 244 / 277 as a cluster.  Finding sixteen free SMs in one
// of the chip's groups beside other kernels does not cost what that gives: refresh 3000 x 2000 9.82 ms by polling, 9.34 with
// clusters of up to eight, 8.99 of up to sixteen (8192 x 8192 75 to 77 ms with any).
constexpr int kClusterCtas = 16, kPortableClusterCtas = 8;
template <bool kCluster>
struct Inbox {};
template <>
struct Inbox<true> {
  float2 dots[2][kClusterCtas][kB];    // {D1_j, D2_j} of every CTA, by step parity
  float rows[2][2][kB];                // the two pivot rows
  uint64_t arrived[2];                 // all of a step's bytes
};

// A value into the shared memory of CTA `rank` of the cluster, its bytes credited to a barrier there.
__device__ __forceinline__ void send(const float* to, float value, const uint64_t* bar, int rank) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(map_to_cta(smem_u32(to), rank)),
               "r"(__float_as_uint(value)), "r"(map_to_cta(smem_u32(bar), rank))
               : "memory");
}
__device__ __forceinline__ void send(const float2* to, float x, float y, const uint64_t* bar, int rank) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::"r"(map_to_cta(smem_u32(to), rank)),
               "r"(__float_as_uint(x)), "r"(__float_as_uint(y)), "r"(map_to_cta(smem_u32(bar), rank))
               : "memory");
}

template <int kPer, bool kCluster>
__global__ void __launch_bounds__(kPanelThreads, 1) qr_panel_pairs_kernel(PanelArgs a) {
  constexpr int kCtaRows = 4 * kPer;
  constexpr int kVec = kPer / 4;       // 128-bit loads per sweep and pivot column
  constexpr int kPollPairs = kPer == 64 ? 7 : 17;   // 128-bit loads a thread keeps in flight per polling round
  __shared__ __align__(16) float xcol[2][kCtaRows];     // pivot column c (double buffered); zero above the pivot row
  __shared__ __align__(16) float ycol[2][kCtaRows];     // column c + 1 as it is before H_c is applied
  __shared__ float2 slices[4][kB];                      // dot products of the four row slices with every column
  __shared__ float4 sums[kB];                           // {D1_j, D2_j, p1_j, p2_j}, the same in every CTA
  __shared__ float taus[kB];
  __shared__ float scol1[kB];                           // column c of S = V^T V (entries above the diagonal)
  __shared__ float scol2[kB];                           // column c + 1 of S
  __shared__ float row1_local[kB];                      // single-CTA launches: rows c and c + 1 without the exchange
  __shared__ float row2_local[kB];
  __shared__ int abort_flag;
  __shared__ Inbox<kCluster> inbox;
  extern __shared__ float dyn[];
  float (*T)[kPitch] = reinterpret_cast<float (*)[kPitch]>(dyn);   // last CTA: compact-WY factor

  const int t = threadIdx.x;
  // A warp owns one slice of 32 columns, so that a sweep's loads of a pivot column are one address for all its lanes.  The
  // exchange is carried out by lane quads, one per column.
  const int j = ((t >> 7) << 5) | (t & 31);
  const int q = (t >> 5) & 3;            // kPer-row slice within the CTA's slab
  const int jx = t >> 2, qx = t & 3;     // column and part of its exchange
  const int row0 = blockIdx.x * kCtaRows;
  const int rows_here = min(kCtaRows, a.r - row0);
  const int ctas = gridDim.x;
  const int my_first = q * kPer;
  // The compact-WY factor T is built by the LAST CTA.  With more than one data CTA the host launches one
  // CTA more than the rows need: it owns no rows, publishes zeros at once and spends the time the others
  // sweep their slabs on T, so that no CTA the others wait for carries that work.
  const bool builds_t = blockIdx.x == gridDim.x - 1;
  const bool has_rows = rows_here > 0;

  float P[kPer];
  {
    const int64_t off = row0 + my_first + static_cast<int64_t>(j) * a.ldp;
    if (a.aligned && my_first + kPer <= rows_here && j < a.b) {
#pragma unroll
      for (int k = 0; k < kPer; k += 4) {
        const float4 h = *reinterpret_cast<const float4*>(a.p_hi + off + k), l = *reinterpret_cast<const float4*>(a.p_lo + off + k);
        P[k] = h.x + l.x;
        P[k + 1] = h.y + l.y;
        P[k + 2] = h.z + l.z;
        P[k + 3] = h.w + l.w;
      }
    } else {
#pragma unroll
      for (int k = 0; k < kPer; ++k) P[k] = (my_first + k < rows_here && j < a.b) ? a.p_hi[off + k] + a.p_lo[off + k] : 0.f;
    }
  }
  if (t < kB) taus[t] = 0.f;
  if (t == 0) abort_flag = 0;
  if constexpr (kCluster) {
    if (t == 0) {
      mbar_init(&inbox.arrived[0], 1);
      mbar_init(&inbox.arrived[1], 1);
      mbar_fence_init();
    }
  }
  if (builds_t)
    for (int idx = t; idx < kB * kPitch; idx += kPanelThreads) dyn[idx] = 0.f;
  if (j < 2) {
    float* dst = (j == 0) ? &xcol[0][my_first] : &ycol[0][my_first];
#pragma unroll
    for (int k = 0; k < kPer; ++k) dst[k] = P[k];
  }
  __syncthreads();
  if constexpr (kCluster) cluster_sync_all();      // the barriers exist before anything arrives on them

  const int reflectors = min(a.b, a.r);
  const unsigned int seq_base = a.epoch * 256u;
  float my_scale = 1.f;                  // 1 / (alpha - beta) of this lane's column once it has been a pivot
  int c = 0, step = 0;
  int built_c = -1, built_pair = 0;      // columns of T that the last CTA still owes from the previous step

  while (c < reflectors) {
    const int parity = step & 1;
    const unsigned int seq = seq_base + static_cast<unsigned int>(step) + 1u;
    // [parity][ctas + 1][kB][2]: words {D1, D2} of every CTA, then {p1, p2} in row `ctas`
    unsigned long long* slots = a.exchange + static_cast<int64_t>(parity) * (ctas + 1) * kB * 2;
    const bool can_pair = c + 1 < reflectors;
    const bool row2_exists = c + 1 < a.r;
    const int local1 = c - row0 - my_first, local2 = c + 1 - row0 - my_first;
    const bool mine1 = local1 >= 0 && local1 < kPer;
    const bool mine2 = local2 >= 0 && local2 < kPer && row2_exists;

    if constexpr (kCluster) {
      // Bytes of this step may be here already: a sender needs this CTA's sums of the step before, not its end.  The phase stays open all
      // the same until this arrival, and the buffer of this parity was read before this CTA sent those sums.
      if (t == 0) mbar_expect_tx(&inbox.arrived[parity], static_cast<uint32_t>(kB * (8 * ctas + (row2_exists ? 8 : 4))));
    }

    // ---- sweep 1: dot products of both pivot columns with this thread's slice of column j ----
    if (has_rows) {
      uint64_t x01 = 0, x23 = 0, y01 = 0, y23 = 0;
      const ulonglong2* x4 = reinterpret_cast<const ulonglong2*>(&xcol[parity][my_first]);
      const ulonglong2* y4 = reinterpret_cast<const ulonglong2*>(&ycol[parity][my_first]);
#pragma unroll
      for (int k4 = 0; k4 < kVec; ++k4) {
        const ulonglong2 x = x4[k4];
        const ulonglong2 y = y4[k4];
        const uint64_t low = pack_floats(P[4 * k4], P[4 * k4 + 1]), high = pack_floats(P[4 * k4 + 2], P[4 * k4 + 3]);
        fma_pair(x01, low, x.x);
        fma_pair(x23, high, x.y);
        fma_pair(y01, low, y.x);
        fma_pair(y23, high, y.y);
      }
      slices[q][j] = make_float2((pair_element(x01, 0) + pair_element(x01, 1)) + (pair_element(x23, 0) + pair_element(x23, 1)),
                                 (pair_element(y01, 0) + pair_element(y01, 1)) + (pair_element(y23, 0) + pair_element(y23, 1)));
    }
    // entries (c, j) and (c + 1, j), on the warps that hold them
    unsigned long long* rows = &slots[(static_cast<int64_t>(ctas) * kB + j) * 2];
    if (mine1) {
      const float entry = take_entry<kPer>(P, local1, false);
      if constexpr (kCluster) {
        for (int g = 0; g < ctas; ++g) send(&inbox.rows[parity][0][j], entry, &inbox.arrived[parity], g);
      } else if (ctas > 1) {
        ll_publish(rows, entry, seq);
      } else {
        row1_local[j] = entry;
      }
    }
    if (mine2) {
      const float entry = take_entry<kPer>(P, local2, false);
      if constexpr (kCluster) {
        for (int g = 0; g < ctas; ++g) send(&inbox.rows[parity][1][j], entry, &inbox.arrived[parity], g);
      } else if (ctas > 1) {
        ll_publish(rows + 1, entry, seq);
      } else {
        row2_local[j] = entry;
      }
    }
    if (ctas == 1 && !row2_exists && q == 0) row2_local[j] = 0.f;
    __syncthreads();                                                              // barrier 1
    float partial1 = 0.f, partial2 = 0.f;                     // this CTA's dot products with column jx
    if ((kCluster || qx == 0) && has_rows) {
      partial1 = (slices[0][jx].x + slices[1][jx].x) + (slices[2][jx].x + slices[3][jx].x);
      partial2 = (slices[0][jx].y + slices[1][jx].y) + (slices[2][jx].y + slices[3][jx].y);
    }
    if constexpr (kCluster) {
      for (int g = qx; g < ctas; g += 4)
        send(&inbox.dots[parity][blockIdx.x][jx], partial1, partial2, &inbox.arrived[parity], g);
    } else if (qx == 0 && ctas > 1) {
      unsigned long long* mine = &slots[(static_cast<int64_t>(blockIdx.x) * kB + jx) * 2];
      asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(mine), "l"(pack_word(partial1, seq)),
                   "l"(pack_word(partial2, seq))
                   : "memory");
    }

    // ---- the last CTA, while the published words travel: the columns of T the previous step produced ----
    if (builds_t && built_c >= 0) {
      t_column(T, scol1, taus, built_c, t);
      if (built_pair) {
        __syncthreads();
        t_column(T, scol2, taus, built_c + 1, t);
      }
    }

    // ---- exchange: lane qx polls CTAs qx, qx + 4, qx + 8, ... (index `ctas` holds the two pivot rows) ----
    if (kCluster || ctas > 1) {
      float total1 = 0.f, total2 = 0.f, p1 = 0.f, p2 = 0.f;
      float part1 = 0.f, part2 = 0.f;
      bool failed = false;
      if constexpr (kCluster) {
        failed = !mbar_wait_bounded(&inbox.arrived[parity], (step >> 1) & 1, &abort_flag, nullptr, 0);
        for (int g = qx; g < ctas; g += 4) {
          const float2 dots = inbox.dots[parity][g][jx];
          part1 += dots.x;
          part2 += dots.y;
        }
        if (qx == 0) {
          p1 = inbox.rows[parity][0][jx];
          p2 = row2_exists ? inbox.rows[parity][1][jx] : 0.f;
        }
      }
      for (int base = 0; !kCluster && base <= ctas && !failed; base += 4 * kPollPairs) {
        unsigned long long w1[kPollPairs], w2[kPollPairs];
        bool pending = true;
        unsigned int polls = 0;
        while (pending && polls < (1u << 20)) {
          pending = false;
#pragma unroll
          for (int u = 0; u < kPollPairs; ++u) {
            const int g = base + qx + 4 * u;
            if (g <= ctas)
              asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];"
                           : "=l"(w1[u]), "=l"(w2[u])
                           : "l"(&slots[(static_cast<int64_t>(g) * kB + jx) * 2])
                           : "memory");
          }
#pragma unroll
          for (int u = 0; u < kPollPairs; ++u) {
            const int g = base + qx + 4 * u;
            if (g <= ctas) {
              if (static_cast<unsigned int>(w1[u] >> 32) != seq) pending = true;
              if (static_cast<unsigned int>(w2[u] >> 32) != seq && (g < ctas || row2_exists)) pending = true;
            }
          }
          ++polls;
        }
        failed = pending;
#pragma unroll
        for (int u = 0; u < kPollPairs; ++u) {
          const int g = base + qx + 4 * u;
          if (g < ctas) {
            part1 += __uint_as_float(static_cast<unsigned int>(w1[u]));
            part2 += __uint_as_float(static_cast<unsigned int>(w2[u]));
          } else if (g == ctas) {
            p1 = __uint_as_float(static_cast<unsigned int>(w1[u]));
            p2 = row2_exists ? __uint_as_float(static_cast<unsigned int>(w2[u])) : 0.f;
          }
        }
      }
      if (failed) {
        abort_flag = 1;
        atomicCAS(a.status, 0, kStatusPanelExchangeTimeout);
      }
      // fixed-shape reductions over the four lanes: identical on every CTA
      float o = __shfl_xor_sync(0xffffffffu, part1, 1);
      float pair_sum = (qx & 1) ? (o + part1) : (part1 + o);
      o = __shfl_xor_sync(0xffffffffu, pair_sum, 2);
      total1 = (qx & 2) ? (o + pair_sum) : (pair_sum + o);
      o = __shfl_xor_sync(0xffffffffu, part2, 1);
      pair_sum = (qx & 1) ? (o + part2) : (part2 + o);
      o = __shfl_xor_sync(0xffffffffu, pair_sum, 2);
      total2 = (qx & 2) ? (o + pair_sum) : (pair_sum + o);
      p1 += __shfl_xor_sync(0xffffffffu, p1, 1);
      p1 += __shfl_xor_sync(0xffffffffu, p1, 2);              // exactly one lane held the pivot-row words
      p2 += __shfl_xor_sync(0xffffffffu, p2, 1);
      p2 += __shfl_xor_sync(0xffffffffu, p2, 2);
      if (qx == 0) sums[jx] = make_float4(total1, total2, p1, p2);
    } else if (qx == 0) {
      sums[jx] = make_float4(partial1, partial2, row1_local[jx], row2_local[jx]);
    }
    __syncthreads();                                                              // barrier 2
    if (abort_flag) break;

    // ---- scalars of the step (every thread computes the same values) ----
    const float4 own = sums[j], first = sums[c];
    const float total1 = own.x, total2 = own.y, p1 = own.z, p2 = own.w;
    const float a1 = first.z;
    const float n1 = first.x;
    const float p2c = first.w;
    float t1, s1;
    householder_scalars(a1, n1, t1, s1);
    bool pair = false;
    float k = 0.f, yc = 0.f, yc1 = 0.f, t2 = 0.f, s2 = 0.f, p1c1 = 0.f, p2c1 = 0.f, d1c1 = 0.f;
    if (can_pair) {
      const float4 second = sums[c + 1];
      p1c1 = second.z;
      d1c1 = second.x;
      p2c1 = second.w;
      const float d2c1 = second.y;
      const float w1c1 = p1c1 + s1 * (d1c1 - a1 * p1c1);       // v_c . y
      k = t1 * w1c1;
      yc = p1c1 - k;
      yc1 = p2c1 - k * s1 * p2c;
      const float n2 = d2c1 - yc * yc;
      if (n2 > kPairThreshold * d2c1) {
        pair = true;
        householder_scalars(yc1, n2, t2, s2);
      }
    }
    // ---- this thread's column ----
    const float sj = (j < c) ? my_scale : 1.f;                  // finished columns are kept unscaled in the registers
    const float w1 = (p1 + s1 * (total1 - a1 * p1)) * sj;       // v_c . column_j
    float w2 = 0.f;
    if (pair) {
      if (j > c + 1) {                                          // v_{c+1} . (H_c a_j)
        const float ajc = p1 - t1 * w1;
        const float ajc1 = p2 - t1 * w1 * s1 * p2c;
        w2 = ajc1 + s2 * (total2 - yc * ajc - yc1 * ajc1);
      } else if (j < c) {                                       // v_{c+1} . v_j
        const float sum_y = total2 - p1c1 * p1 - p2c1 * p2;
        const float sum_x = total1 - a1 * p1 - p2c * p2;
        w2 = (p2 + s2 * (sum_y - k * s1 * sum_x)) * sj;
      } else if (j == c) {                                      // v_c . v_{c+1}
        const float tail_x = fmaf(-p2c, p2c, __fsub_rn(n1, __fmul_rn(a1, a1)));
        const float sxy = fmaf(-__fmul_rn(k, s1), tail_x, fmaf(-p2c, p2c1, fmaf(-a1, p1c1, d1c1)));
        w2 = fmaf(s1, p2c, __fmul_rn(__fmul_rn(s1, s2), sxy));
      }
    }
    if (j == c) my_scale = s1;
    if (pair && j == c + 1) my_scale = s2;
    if (builds_t && q == 0) {
      if (j < c) {
        scol1[j] = w1;
        scol2[j] = w2;
      }
      if (j == c) {
        scol2[c] = w2;
        taus[c] = t1;
        a.tau[c] = t1;
      }
      if (pair && j == c + 1) {
        taus[c + 1] = t2;
        a.tau[c + 1] = t2;
      }
    }

    // ---- sweep 2: a_j <- a_j - A x - B y for the columns right of c, next pivot columns published ----
    const int next = c + (pair ? 2 : 1);
    if (j > c && has_rows) {
      float B = 0.f;
      if (pair && j > c + 1) B = t2 * w2 * s2;
      const float A = fmaf(__fmul_rn(t1, w1), s1, -__fmul_rn(__fmul_rn(B, k), s1));               // column c + 1 of a pair: y' = y - k s_c x (unscaled v)
      const ulonglong2* x4 = reinterpret_cast<const ulonglong2*>(&xcol[parity][my_first]);
      const uint64_t minus_a = pack_floats(-A, -A), minus_b = pack_floats(-B, -B);
      if (pair) {
        const ulonglong2* y4 = reinterpret_cast<const ulonglong2*>(&ycol[parity][my_first]);
#pragma unroll
        for (int k4 = 0; k4 < kVec; ++k4) {
          const ulonglong2 x = x4[k4];
          const ulonglong2 y = y4[k4];
          uint64_t low = pack_floats(P[4 * k4], P[4 * k4 + 1]), high = pack_floats(P[4 * k4 + 2], P[4 * k4 + 3]);
          fma_pair(low, minus_a, x.x);
          fma_pair(high, minus_a, x.y);
          fma_pair(low, minus_b, y.x);
          fma_pair(high, minus_b, y.y);
          P[4 * k4] = pair_element(low, 0);
          P[4 * k4 + 1] = pair_element(low, 1);
          P[4 * k4 + 2] = pair_element(high, 0);
          P[4 * k4 + 3] = pair_element(high, 1);
        }
      } else if (A != 0.f) {
#pragma unroll
        for (int k4 = 0; k4 < kVec; ++k4) {
          const ulonglong2 x = x4[k4];
          uint64_t low = pack_floats(P[4 * k4], P[4 * k4 + 1]), high = pack_floats(P[4 * k4 + 2], P[4 * k4 + 3]);
          fma_pair(low, minus_a, x.x);
          fma_pair(high, minus_a, x.y);
          P[4 * k4] = pair_element(low, 0);
          P[4 * k4 + 1] = pair_element(low, 1);
          P[4 * k4 + 2] = pair_element(high, 0);
          P[4 * k4 + 3] = pair_element(high, 1);
        }
      }
      // The pivot rows right of the pivots now hold R entries nobody reads again: zero them so that later
      // pivot columns leave the registers already masked above their pivot row.
      if (mine1) take_entry<kPer>(P, local1, true);
      if (pair && mine2) take_entry<kPer>(P, local2, true);
      if (j == next || j == next + 1) {
        float* dst = (j == next) ? &xcol[parity ^ 1][my_first] : &ycol[parity ^ 1][my_first];
        float4* d4 = reinterpret_cast<float4*>(dst);
#pragma unroll
        for (int k4 = 0; k4 < kVec; ++k4) d4[k4] = make_float4(P[4 * k4], P[4 * k4 + 1], P[4 * k4 + 2], P[4 * k4 + 3]);
      }
    }
    __syncthreads();                                                              // barrier 3
    built_c = c;
    built_pair = pair ? 1 : 0;
    c = next;
    ++step;
  }

  if (a.trace && blockIdx.x == 0 && t == 0) a.trace[0] = step;   // diagnostics: exchange steps taken

  // ---- the last CTA: the columns of T of the last step, then T and T^T as operand planes ----
  if (builds_t && !abort_flag) {
    if (built_c >= 0) {
      t_column(T, scol1, taus, built_c, t);
      if (built_pair) {
        __syncthreads();
        t_column(T, scol2, taus, built_c + 1, t);
      }
    }
    __syncthreads();
    for (int idx = t; idx < kB * kB; idx += kPanelThreads) {
      const int r = idx & (kB - 1), cidx = idx >> 7;
      if (r < a.b && cidx < a.b) {
        const float v = T[r][cidx];
        const float h = tf32_rn(v);
        a.t_hi[r + cidx * a.ldt] = h;
        a.t_lo[r + cidx * a.ldt] = v - h;
        const float vt = T[cidx][r];
        const float ht = tf32_rn(vt);
        a.tt_hi[r + cidx * a.ldt] = ht;
        a.tt_lo[r + cidx * a.ldt] = vt - ht;
      }
    }
    __syncthreads();
  }

  // ---- outputs: V (r x b) and V^T (b x r), from the registers: 16 bytes a thread along V's columns, and along the rows of V^T
  // (lanes are neighbouring columns) 128 bytes a warp ----
  if (j < a.b) {
    const float out_scale = (j < reflectors) ? my_scale : 0.f;
#pragma unroll
    for (int k = 0; k < kPer; k += 4) {
      float v[4], h[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int gi = row0 + my_first + k + u;
        v[u] = (j < reflectors) ? ((gi > j) ? P[k + u] * out_scale : (gi == j ? 1.f : 0.f)) : 0.f;
        h[u] = tf32_rn(v[u]);
        v[u] -= h[u];
        if (my_first + k + u < rows_here) {
          const int64_t off = j + static_cast<int64_t>(gi) * a.ldvt;
          a.vt_hi[off] = h[u];
          a.vt_lo[off] = v[u];
        }
      }
      const int64_t off = row0 + my_first + k + static_cast<int64_t>(j) * a.ldv;
      if (a.aligned && my_first + k + 4 <= rows_here) {
        *reinterpret_cast<float4*>(a.v_hi + off) = make_float4(h[0], h[1], h[2], h[3]);
        *reinterpret_cast<float4*>(a.v_lo + off) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (my_first + k + u < rows_here) {
            a.v_hi[off + u] = h[u];
            a.v_lo[off + u] = v[u];
          }
        }
      }
    }
  }
  if constexpr (kCluster) cluster_sync_all();      // nobody leaves while another CTA may still write into its shared memory
}

}  // namespace

namespace {

struct ClusterLaunch {
  cudaLaunchAttribute cluster{};
  cudaLaunchConfig_t config{};
  ClusterLaunch(int ctas, size_t smem, cudaStream_t stream) {
    cluster.id = cudaLaunchAttributeClusterDimension;
    cluster.val.clusterDim.x = static_cast<unsigned>(ctas);
    cluster.val.clusterDim.y = cluster.val.clusterDim.z = 1;
    config.gridDim = dim3(ctas);
    config.blockDim = dim3(kPanelThreads);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    config.attrs = &cluster;
    config.numAttrs = 1;
  }
  ClusterLaunch(const ClusterLaunch&) = delete;      // (the configuration points into the object)
};

// CTAs of the largest cluster that this device takes of the kernel, which is made ready for it; looked up once for each device.
template <int kPer>
int largest_cluster(size_t smem) {
  constexpr int kDevices = 64;
  static std::atomic<int> known[kDevices] = {};
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= kDevices) return 0;
  if (const int largest = known[device].load()) return largest;
  auto* kernel = qr_panel_pairs_kernel<kPer, true>;
  PerDeviceOnce once;
  allow_dynamic_smem(reinterpret_cast<const void*>(kernel), smem, once, "qr_panel_pairs");
  int clusters = 0;
  ClusterLaunch launch(kClusterCtas, smem, nullptr);
  const bool large = cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel), cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                     cudaOccupancyMaxActiveClusters(&clusters, kernel, &launch.config) == cudaSuccess && clusters > 0;
  if (!large) cudaGetLastError();      // (a refusal is not this launch's error)
  known[device] = large ? kClusterCtas : kPortableClusterCtas;
  return known[device];
}

template <int kPer>
void launch_pairs(PanelArgs args, int r, cudaStream_t stream) {
  const size_t smem = static_cast<size_t>(kB) * kPitch * sizeof(float);
  int ctas = (r + 4 * kPer - 1) / (4 * kPer);
  if (ctas > 1 && ctas < 148) ++ctas;   // the rowless CTA that builds T (see the kernel)
  cudaError_t err;
  if (ctas > 1 && ctas <= largest_cluster<kPer>(smem)) {
    // a cluster's CTAs are resident together by definition
    ClusterLaunch launch(ctas, smem, stream);
    err = cudaLaunchKernelEx(&launch.config, qr_panel_pairs_kernel<kPer, true>, args);
  } else {
    static PerDeviceOnce configured;
    allow_dynamic_smem(reinterpret_cast<const void*>(qr_panel_pairs_kernel<kPer, false>), smem, configured, "qr_panel_pairs");
    void* params[] = {&args};
    // Cooperative launch: the CTAs exchange data through global memory while running, so all of them
    // must be resident at the same time; the runtime refuses the launch otherwise.
    err = cudaLaunchCooperativeKernel(reinterpret_cast<void*>(qr_panel_pairs_kernel<kPer, false>), dim3(ctas), dim3(kPanelThreads),
                                      params, smem, stream);
  }
  if (err != cudaSuccess) throw std::runtime_error(std::string("qr_panel_pairs launch: ") + cudaGetErrorString(err));
}

}  // namespace

void qr_panel_pairs(const float* p_hi, const float* p_lo, int64_t ldp, int r, int b, float* v_hi, float* v_lo, int64_t ldv,
                    float* vt_hi, float* vt_lo, int64_t ldvt, float* tau, float* t_hi, float* t_lo, float* tt_hi,
                    float* tt_lo, int64_t ldt, float* exchange, int* status, cudaStream_t stream, int rows_per_cta,
                    long long* steps_taken) {
  if (r <= 0 || b <= 0) return;
  if (b > kB) throw std::invalid_argument("qr_panel_pairs: panel wider than 128 columns");
  if (r > kQrMaxRows) throw std::invalid_argument("qr_panel_pairs: more rows than one cooperative grid can hold");
  if (rows_per_cta != 128 && rows_per_cta != 256) throw std::invalid_argument("qr_panel_pairs: rows_per_cta is 128 or 256");
  if (rows_per_cta == 128 && r > 148 * 128) rows_per_cta = 256;   // one CTA per SM at most
  const unsigned int epoch = next_panel_epoch();
  const bool aligned = ((reinterpret_cast<uintptr_t>(p_hi) | reinterpret_cast<uintptr_t>(p_lo) | reinterpret_cast<uintptr_t>(v_hi) |
                         reinterpret_cast<uintptr_t>(v_lo)) & 15) == 0 && ldp % 4 == 0 && ldv % 4 == 0;
  PanelArgs args{p_hi, p_lo, ldp, r, b, v_hi, v_lo, ldv, vt_hi, vt_lo, ldvt, tau, t_hi, t_lo, tt_hi, tt_lo, ldt,
                 reinterpret_cast<unsigned long long*>(exchange), epoch, status, steps_taken, aligned, 0};
  if (rows_per_cta == 128) launch_pairs<32>(args, r, stream);
  else launch_pairs<64>(args, r, stream);
}

}  // namespace soapb200
