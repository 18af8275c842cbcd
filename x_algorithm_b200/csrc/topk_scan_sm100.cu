// Corpus scan of the exhaustive top-k on Blackwell tensor cores (reference: users_bf16 @ posts^T,
// phoenix/xrex/models/recsys_two_tower_model.py:2455-2456; its int8 form 2518-2533): the score tile of 128 corpus rows x NQ
// queries is formed in TMEM and consumed there, so the only HBM traffic is the corpus itself, read once.
//
// Persistent kernel, one CTA per SM, 576 threads (640 in the int8 collect pass with the threshold bias):
//   warp 0      TMA producer: the query matrix once (stays in shared memory), then one corpus tile of 128 rows per
//               stage (128-byte swizzle, 128-byte boxes: 64 bf16 or 128 int8 columns)
//   warp 1      MMA issuer: tcgen05.mma M=128 (corpus rows) x N=NQ (queries), 32 bytes of a row per instruction
//               (kind::f16: 16 bf16, fp32 sums; kind::i8: 32 int8, int32 sums), into one of two TMEM accumulators
//   (with the bias: warps 18, 19 write the rows' side of it, see bias_x)
//   warps 2-17  consumers: each warp reads its 32-row lane quadrant and a quarter (ScanCfg::SPLIT: half) of the query columns with
//               tcgen05.ld and either appends rows whose score reaches the query's threshold to the survivor list
//               (collect pass) or reduces the 32-row maximum per query (sample pass)
// An int8 row of 128 columns is the byte image of a bf16 row of 64: tiles, swizzle, descriptors and tensor maps are the
// same, only the instruction kind and what a consumer makes of an accumulator differ.
// Measured (256 queries, k = 1000, one 12.5 M-row shard of 128 columns, whole top-k call, each pair on one box): int8 rows 1198 -> 840 us
// when their thresholds went into the sum, 835 -> 772 with the consumers' loop compiled twice; bf16 rows 910 us.
// All mbarrier waits are bounded; on expiry *err_flag is raised and the kernel unwinds.
#include "common.cuh"
#include "sm100_ptx.cuh"
#include "topk_scan.cuh"

#include <float.h>

#include <type_traits>

namespace phx {
namespace {

using namespace sm100;

constexpr int TC_ROWS = 128;      // corpus rows per tile
constexpr int TC_QBOX = 64;       // query rows per TMA box
constexpr int TC_CWARPS = 16;     // consumer warps: four per scheduler, what hides the latency of the filter's chains
constexpr int TC_THREADS = 64 + 32 * TC_CWARPS;
constexpr int TC_STAGES = 4;
constexpr int TC_BWARPS = 2;      // int8 collect pass: warps that write the rows' side of the bias
// the collect pass with the bias has rows of two k-blocks in one stage less, beside its bias operands
__host__ __device__ constexpr int scan_threads(bool bias) { return TC_THREADS + (bias ? 32 * TC_BWARPS : 0); }
__host__ __device__ constexpr int scan_stages(bool bias, int kblk) { return bias && kblk == 2 ? TC_STAGES - 1 : TC_STAGES; }
__host__ __device__ constexpr int scan_bias_bytes(bool bias, int nq) { return bias ? TC_STAGES * TC_ROWS * 32 + nq * 32 + nq * 4 + 16 : 0; }
constexpr int QCAP = 64;          // per-warp queue of survivors (records of 16 bytes)
constexpr int QFLUSH = 20;        // flush a warp's queue once it holds this many records

__device__ __forceinline__ uint32_t ord32(float f) {
  if (f == 0.f) f = 0.f;  // -0 -> +0
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// Survivors of one consumer warp on their way to the global lists.  An append is an atomic whose result the store depends
// on, a memory round trip: records wait in the warp's shared-memory queue, and a flush only issues the atomics - the stores
// of a flush are made at the next one, when the slots have long arrived.  A warp that stalled here for one round trip would come
// late for its next accumulator and hold up the whole CTA.  Together with the row-at-a-time test below: 256 queries, k = 1000,
// 12.5 M rows 1.08 -> 1.00 ms (bf16), 1.38 -> 1.26 ms (int8).
struct Flight {
  bool on = false;
  uint32_t lo = 0, hi = 0, u = 0;
  int slot = 0;
  __device__ __forceinline__ void land(const TcScanArgs& a) {
    if (on && slot < a.cap) a.surv[(size_t)u * a.cap + slot] = ((unsigned long long)hi << 32) | lo;
    on = false;
  }
};
__device__ __forceinline__ void flush_queue(const TcScanArgs& a, const uint4* queue, int n, int lane, Flight& f) {
  for (int i = 0; i < n; i += 32) {
    f.land(a);
    if (i + lane < n) {
      const uint4 rec = queue[i + lane];
      f.lo = rec.x; f.hi = rec.y; f.u = rec.z;
      f.slot = atomicAdd(&a.counts[rec.z], 1);
      f.on = true;
    }
  }
}

// D[tmem] (+)= A[smem desc] * B[smem desc], signed int8 inputs, int32 accumulate, K = 32
__device__ __forceinline__ void umma_s8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum)
      : "memory");
}
// instruction descriptor of kind::i8: D int32, A / B signed, both K-major
__host__ __device__ constexpr uint32_t make_idesc_s8(int M, int N) {
  return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
template <int CH>
__device__ __forceinline__ void tmem_ld_chunk(uint32_t taddr, uint32_t* r) {
  if (CH == 32) tmem_ld32_nowait(taddr, r); else tmem_ld16_nowait(taddr, r);
}
// The threshold inside the int8 sum.  One more MMA step of 32 bytes adds -x(row) * t(query) to every dot product: the row's
// 32 bytes all hold x = floor(c / row scale), the query's 32 bytes sum to -t, t = floor(threshold / (query scale * c)) a little
// reduced, so that x t is at most the smallest dot product whose score can reach the threshold.  A sum below zero is then no
// hit, whatever its query, and 32 columns are tested by and-ing sign bits: no conversion, no scale, no group's smallest threshold.
// c maps one of the smaller scales among the rows that count (over 32 rows of the corpus) to x = 100; x ends at 127 and t at
// 4096, which only lets more rows through to the second filter.  A group with a query about which the bias can say nothing (bias_t < 0) goes to
// the second filter as a whole (it is open).
constexpr float BIAS_X = 100.0f;
constexpr int BIAS_T_MAX = 4096;
__device__ __forceinline__ int bias_x(float c, float row_scale) {
  // No statement about a row whose scale is not an ordinary positive number: 1 / scale of a denormal one would come out infinite.  Zero
  // scores are no hits where the bias says anything (thresholds are positive there): the largest x keeps such rows out.
  if (!(row_scale >= FLT_MIN)) return row_scale == 0.f ? 127 : 0;
  float inv;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(row_scale));   // 1 ulp, covered by the reduction of t; 0 for scales above 2^126
  return (int)fminf(c * inv, 127.f);
}
__device__ __forceinline__ int bias_t(float c, float thr, float query_scale) {
  // no statement about thresholds that are not positive (or close to the denormals: sums below zero may reach them), where
  // dot * scale may overflow, or where c or threshold / query scale is denormal (their rounding is not relative) or infinite
  if (!(thr >= 1e-30f) || !(query_scale * 4194304.f < INFINITY) || !(c >= FLT_MIN && c < INFINITY)) return -1;
  const float ratio = __fdiv_rn(thr, query_scale);
  if (!(ratio >= FLT_MIN && ratio < INFINITY)) return -1;
  return (int)fminf(__fdiv_rn(ratio, c) * 0.999f, (float)BIAS_T_MAX);
}
// The int32 accumulator of an int8 dot product as fp32 (exact: |dot| <= 128 * 128 * 256 = 2^22) times the query's scale;
// the row's scale follows: (float(dot) * query scale) * row scale, in that order.
__device__ __forceinline__ float s8_value(uint32_t acc, float query_scale) { return (float)(int)acc * query_scale; }

constexpr float S8_OFFSET = 12582912.0f;            // 1.5 * 2^23: its bit pattern plus an integer below 2^22 in size is the float of their sum
constexpr uint32_t S8_OFFSET_BITS = 0x4B400000u;

// How the consumer warps share the tiles: all sixteen on every tile, a quarter of the columns each, or (SPLIT: some collect passes with 64
// columns, split_tiles) eight on every other tile, half of the columns each.  A warp that has rows to test is late for its next tile, and an
// accumulator goes back to the MMA warp when the last of its warps has read it: split, fewer warps wait for one another, each has two
// tiles' time, and what a tile costs beside its columns (wait, vote, release) is paid half as often; but twice the columns share one
// smallest threshold, and a group's rows are tested by one warp instead of two.  With 128 columns it takes as much from short lists as it gives long
// ones (12.5 M int8 rows, us, k = 1 / 1000: 396 / 477 -> 414 / 460); with 256 a warp's half would take two turns, and rows to test in the first would
// hold the accumulator (581 / 710 -> 726 / 918).
template <int NQ, bool SPLIT> struct ScanCfg {
  static constexpr int CW = SPLIT ? NQ / 2 : NQ / 4; // query columns per consumer warp
  static constexpr int CH = CW < 32 ? CW : 32;       // columns per group; the collect filter's threshold is the smallest of the group's
  static constexpr int GROUPS = NQ / CH;
  static constexpr int DRAIN = (SPLIT ? TC_CWARPS / 2 : TC_CWARPS) * 32;   // threads that release an accumulator
};

template <int MODE, bool I8, int NQ, bool BIAS, bool SPLIT>
__global__ void __launch_bounds__(scan_threads(BIAS), 1)
scan_tc_kernel(const __grid_constant__ CUtensorMap map_corpus, const __grid_constant__ CUtensorMap map_users,
               TcScanArgs a, int* err_flag) {
  using cfg = ScanCfg<NQ, SPLIT>;
  constexpr int CW = cfg::CW, CH = cfg::CH;
  static_assert(!BIAS || (MODE == 1 && I8), "the bias belongs to the int8 collect pass");
  extern __shared__ uint8_t smem_raw[];
  const int kblk = a.row_bytes / 128;                            // 128-byte k-blocks: 1 or 2
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t users_smem = smem_base;                         // kblk x [NQ x 128 B]
  const uint32_t users_bytes = (uint32_t)kblk * NQ * 128;
  const uint32_t stage_bytes = (uint32_t)kblk * TC_ROWS * 128;
  const uint32_t stage_base = users_smem + users_bytes;
  const int stages = scan_stages(BIAS, kblk);
  const uint32_t bias_smem = stage_base + stages * stage_bytes;    // BIAS: per stage [128 x 32 B] of x; [NQ x 32 B] of -t, [NQ] t
  const uint32_t bias_q = bias_smem + TC_STAGES * TC_ROWS * 32;
  const uint32_t thr_smem = bias_smem + scan_bias_bytes(BIAS, NQ);  // [256] thresholds, [256] query scales, [8] + [8] per group, [128] query scale pairs
  const uint32_t queue_smem = thr_smem + 2 * 256 * 4 + 64 + 128 * 16;         // [consumer warps][QCAP] records
  const uint32_t rows_smem = queue_smem + TC_CWARPS * QCAP * 16;   // [consumer warps][32] scores of one corpus row
  const uint32_t bars = rows_smem + TC_CWARPS * 128;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (TC_STAGES + s); };
  auto tfull_bar = [&](int x) { return bars + 8u * (2 * TC_STAGES + x); };
  auto tempty_bar = [&](int x) { return bars + 8u * (2 * TC_STAGES + 2 + x); };
  const uint32_t users_bar = bars + 8u * (2 * TC_STAGES + 4);
  auto xfull_bar = [&](int s) { return bars + 8u * (2 * TC_STAGES + 5 + s); };
  const uint32_t tmem_slot = bars + 8u * (3 * TC_STAGES + 5);
  uint32_t* tmem_slot_ptr = reinterpret_cast<uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));
  float* s_thr = reinterpret_cast<float*>(smem_raw + (thr_smem - smem_u32(smem_raw)));
  float* s_us = s_thr + 256;
  float* s_thr_min = s_us + 256;     // [8] smallest threshold of a group
  float* s_us_max = s_thr_min + 8;   // [8] largest query scale of a group
  int* s_t = reinterpret_cast<int*>(smem_raw + (bias_q + NQ * 32 - smem_u32(smem_raw)));   // BIAS: [NQ] t
  int* s_open = s_t + NQ;            // BIAS: bit g: group g is not filtered by the bias
  float4* s_us2 = reinterpret_cast<float4*>(s_us_max + 8);   // [128] {scale, scale, -offset * scale, -offset * scale} of two queries
  uint4* s_queue = reinterpret_cast<uint4*>(smem_raw + (queue_smem - smem_u32(smem_raw)));

  const int warp = warp_index(), lane = threadIdx.x & 31;
  volatile int* verr = err_flag;
  // work list: MODE 1 every tile; MODE 0 tiles 0, stride, 2*stride, ...
  const long long n_tiles = (a.rows + TC_ROWS - 1) / TC_ROWS;
  const long long n_work = (MODE == 0) ? (n_tiles + a.stride - 1) / a.stride : n_tiles;

  // the kernels in front wrote the queries and thresholds; what follows may set up from here on
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (threadIdx.x == 0) {
    *gave_up() = 0;
    prefetch_map(&map_corpus); prefetch_map(&map_users);
    for (int s = 0; s < TC_STAGES; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    for (int x = 0; x < 2; ++x) { mbar_init(tfull_bar(x), 1); mbar_init(tempty_bar(x), cfg::DRAIN); }
    for (int s = 0; s < TC_STAGES; ++s) mbar_init(xfull_bar(s), 1);
    mbar_init(users_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int u = threadIdx.x; u < NQ; u += scan_threads(BIAS)) {
    if (MODE == 1) {
      // collect when the score >= thr, with thr a little below the midpoint under the pivot: a superset of
      // { bf16(score) >= pivot }; the exact selection happens later on the rounded scores
      float t = INFINITY;
      if (u < a.B) {
        const float p = a.pivot[u];
        t = (p == -INFINITY) ? -INFINITY : p - fabsf(p) * 0.00390625f - 1e-37f;
      }
      s_thr[u] = t;
    }
    if (I8) s_us[u] = (u < a.B) ? a.user_scale[u] : 0.f;
  }
  float bias_c = 0.f;
  if (BIAS) {
    // reference of the rows' factor, the same in every thread: each warp ranks the scales of 32 rows spread over the corpus
    // (without those that are not ordinary positive numbers).  Lists are made of rows with large scales, so the reference is taken
    // among the scales from a quarter of the second largest up: rows that hold nothing (the quantiser gives them 1e-12) or have far
    // smaller scales would otherwise leave a coarse x, or none, to the rows that count.  256 queries, k = 1000, 12.5 M rows, device us with
    // no threshold in the sum / the 1/8 quantile of all scales / this: 15 % empty rows 1163 / 1426 / 811, scales over six decades
    // 1171 / 1524 / 810, no such rows 1147 / 804 / 814.
    float s = __ldg(a.row_scale + ((long long)lane * (a.rows - 1)) / 31);
    if (!(s >= FLT_MIN && s < INFINITY)) s = INFINITY;
    const int n_pos = __popc(__ballot_sync(0xffffffffu, s < INFINITY));
    int below = 0;                                   // smaller scales, equal ones in front counted too
#pragma unroll
    for (int l = 0; l < 32; ++l) {
      const float o = __shfl_sync(0xffffffffu, s, l);
      below += (o < s || (o == s && l < lane)) ? 1 : 0;
    }
    if (threadIdx.x == 0) *s_open = a.scales_negative ? ~0 : 0;   // scales below zero turn the order of the sums round
    const uint32_t up = __ballot_sync(0xffffffffu, n_pos > 0 && below == (n_pos > 1 ? n_pos - 2 : 0));
    if (up) {
      const float upper = __shfl_sync(0xffffffffu, s, __ffs(up) - 1);
      const int low = __popc(__ballot_sync(0xffffffffu, s < 0.25f * upper));
      const uint32_t m = __ballot_sync(0xffffffffu, below == low + (n_pos - low) / 8);
      bias_c = BIAS_X * __shfl_sync(0xffffffffu, s, __ffs(m) - 1);
    }
    __syncthreads();                                 // thresholds and query scales are written
    for (int u = threadIdx.x; u < NQ; u += scan_threads(BIAS)) {
      int t = u < a.B ? bias_t(bias_c, s_thr[u], s_us[u]) : BIAS_T_MAX;
      if (t < 0) { atomicOr(s_open, 1 << (u / CH)); t = 0; }
      s_t[u] = t;
      const int each = t >> 5, more = t & 31;        // 32 bytes that sum to -t
      uint32_t w[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        w[i] = 0;
#pragma unroll
        for (int b = 0; b < 4; ++b) w[i] |= (uint32_t)((-(each + (4 * i + b < more ? 1 : 0))) & 0xFF) << (8 * b);
      }
      uint4* dst = reinterpret_cast<uint4*>(smem_raw + (bias_q - smem_u32(smem_raw)) + u * 32);
      dst[0] = make_uint4(w[0], w[1], w[2], w[3]); dst[1] = make_uint4(w[4], w[5], w[6], w[7]);   // (a swizzle only permutes the addends)
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tmem_slot, 2 * NQ);
  tc_fence_before();
  __syncthreads();
  if (MODE == 1) {   // per group: smallest threshold, largest query scale
    if (threadIdx.x < cfg::GROUPS) {
      float t = INFINITY, m = 0.f;
      for (int k = 0; k < CH; ++k) {
        t = fminf(t, s_thr[threadIdx.x * CH + k]);
        if (I8) m = fmaxf(m, s_us[threadIdx.x * CH + k]);
      }
      // a scale whose offset product overflows leaves no bound (-inf, NaN): such a group is not filtered
      s_thr_min[threadIdx.x] = t; s_us_max[threadIdx.x] = (m * S8_OFFSET < INFINITY) ? m : INFINITY;
    }
    if (I8 && threadIdx.x < NQ / 2) {
      const float x = s_us[2 * threadIdx.x], y = s_us[2 * threadIdx.x + 1];
      s_us2[threadIdx.x] = make_float4(x, y, -S8_OFFSET * x, -S8_OFFSET * y);
    }
    __syncthreads();
  }
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;
  // from 128 query columns on a call whose groups are all open leaves the bias out; the same in every thread
  constexpr bool TWO_LOOPS = BIAS && NQ >= 128;
  const bool biased = BIAS && !(TWO_LOOPS && (~*s_open & ((1 << cfg::GROUPS) - 1)) == 0);

  if (warp == 0) {
    if (elect_one()) {
      mbar_expect_tx(users_bar, users_bytes);
      for (int kb = 0; kb < kblk; ++kb)
        for (int q = 0; q < NQ; q += TC_QBOX) tma_load_2d(users_smem + (kb * NQ + q) * 128, &map_users, users_bar, kb * BK, q);
      int stage = 0; uint32_t phase = 0;
      for (long long w = blockIdx.x; w < n_work; w += gridDim.x) {
        const long long tile = (MODE == 0) ? w * a.stride : w;
        if (!mbar_wait(empty_bar(stage), phase ^ 1, verr)) break;
        const uint32_t dst = stage_base + stage * stage_bytes;
        mbar_expect_tx(full_bar(stage), stage_bytes);
        for (int kb = 0; kb < kblk; ++kb)
          tma_load_2d(dst + kb * TC_ROWS * 128, &map_corpus, full_bar(stage), kb * BK, (int)(tile * TC_ROWS));
        if (++stage == stages) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = I8 ? make_idesc_s8(TC_ROWS, NQ) : make_idesc(TC_ROWS, NQ);
      bool ok = mbar_wait(users_bar, 0, verr);
      int stage = 0; uint32_t phase = 0, it = 0;
      for (long long w = blockIdx.x; w < n_work && ok; w += gridDim.x, ++it) {
        const uint32_t acc = it & 1, acc_phase = (it >> 1) & 1;
        if (!mbar_wait(tempty_bar(acc), acc_phase ^ 1, verr)) break;
        if (!mbar_wait(full_bar(stage), phase, verr)) break;
        tc_fence_after();
        const uint32_t src = stage_base + stage * stage_bytes;
        for (int kb = 0; kb < kblk; ++kb) {
          const uint64_t adesc = make_smem_desc(src + kb * TC_ROWS * 128);
          const uint64_t bdesc = make_smem_desc(users_smem + kb * NQ * 128);
#pragma unroll
          for (int k = 0; k < 4; ++k) {   // 32 bytes of every row per instruction
            if (I8) umma_s8(tmem_base + acc * NQ, adesc + (uint64_t)(k * 2), bdesc + (uint64_t)(k * 2), idesc, (kb | k) != 0);
            else umma_bf16(tmem_base + acc * NQ, adesc + (uint64_t)(k * 2), bdesc + (uint64_t)(k * 2), idesc, (kb | k) != 0);
          }
        }
        if (biased) {
          if (!mbar_wait(xfull_bar(stage), phase, verr)) break;
          tc_fence_after();
          umma_s8(tmem_base + acc * NQ, make_smem_desc_32b(bias_smem + stage * TC_ROWS * 32), make_smem_desc_32b(bias_q), idesc, 1);
        }
        umma_commit(empty_bar(stage));
        umma_commit(tfull_bar(acc));
        if (++stage == stages) { stage = 0; phase ^= 1; }
      }
    }
  } else if (BIAS && warp >= 2 + TC_CWARPS) {
    // ---- the rows' side of the bias: each warp every other tile, four rows a lane, into the tile's stage ----
    // scales of AHEAD tiles are on their way (a tile takes less than a round trip to memory); the loop over them is unrolled
    // because moving a register that a load has yet to fill waits for it
    constexpr int AHEAD = 3;
    const int first = warp - (2 + TC_CWARPS);
    const long long step = (long long)TC_BWARPS * gridDim.x;
    float s[AHEAD][4];
    auto fetch = [&](long long w, float (&v)[4]) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const long long row = w * TC_ROWS + i * 32 + lane;
        v[i] = (w < n_work && row < a.rows) ? __ldg(a.row_scale + row) : 0.f;
      }
    };
    const long long w_first = blockIdx.x + (long long)first * gridDim.x;
#pragma unroll
    for (int d = 0; d < AHEAD; ++d) fetch(w_first + d * step, s[d]);
    int stage = first; uint32_t phase = 0;             // TC_BWARPS <= stages
    bool ok = true;
    for (long long w0 = biased ? w_first : n_work; w0 < n_work && ok; w0 += AHEAD * step) {
#pragma unroll
      for (int d = 0; d < AHEAD; ++d) {
        const long long w = w0 + d * step;
        if (w < n_work && ok) {
          // the stage is free once the MMAs of the tile before it are done, as for the copies
          ok = __all_sync(0xffffffffu, mbar_wait(empty_bar(stage), phase ^ 1, verr));
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t x = (uint32_t)bias_x(bias_c, s[d][i]) * 0x01010101u;
            uint4* dst = reinterpret_cast<uint4*>(smem_raw + (bias_smem - smem_u32(smem_raw)) + stage * TC_ROWS * 32 + (i * 32 + lane) * 32);
            dst[0] = make_uint4(x, x, x, x); dst[1] = make_uint4(x, x, x, x);
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0 && ok) mbar_arrive(xfull_bar(stage));
          fetch(w + AHEAD * step, s[d]);
          stage += TC_BWARPS;
          if (stage >= stages) { stage -= stages; phase ^= 1; }
        }
      }
    }
  } else {
    // FOLDED: the thresholds are part of the sums.  128 and 256 columns have a loop without that as well, for calls whose scores are not
    // above zero (12.5 M rows, all of them below, 256 / 100 queries: 10.25 / 6.35 ms before there was a bias, 10.65 / 6.62 with one loop,
    // 9.84 / 6.11 with two), and of the two the one with the bias is compiled with fewer spilled registers (scores above zero: 813 -> 710 us,
    // 502 -> 477).  64 columns: 310 us with one loop, 319 with two.
    auto consume = [&](auto folded) {
      constexpr bool FOLDED = decltype(folded)::value;
      const int ew = warp - 2;
      const int part = SPLIT ? (ew >> 2) & 1 : ew >> 2;   // which half or quarter of the query columns
      const int quad = warp & 3;       // TMEM lane quadrant
      uint4* const queue = s_queue + ew * QCAP;
      uint32_t* const s_row = reinterpret_cast<uint32_t*>(smem_raw + (rows_smem - smem_u32(smem_raw))) + ew * 32;
      int nq = 0;                      // records in the queue (the same in every lane)
      Flight flight;
      // threshold and query scale of the column this lane tests in each group
      float t_lane[CW / CH], us_lane[CW / CH];
      int bt_lane[CW / CH];            // t of that column
#pragma unroll
      for (int c = 0; c < CW / CH; ++c) {
        t_lane[c] = (MODE == 1 && lane < CH) ? s_thr[part * CW + c * CH + lane] : INFINITY;
        us_lane[c] = (I8 && lane < CH) ? s_us[part * CW + c * CH + lane] : 0.f;
        bt_lane[c] = (FOLDED && lane < CH) ? s_t[part * CW + c * CH + lane] : 0;
      }
      const int open = FOLDED ? *s_open : 0;
      constexpr int EACH = SPLIT ? 2 : 1;                 // a warp's tiles: every one, or every other one
      uint32_t it = SPLIT ? ew >> 3 : 0;
      for (long long w = blockIdx.x + (long long)it * gridDim.x; w < n_work; w += (long long)EACH * gridDim.x, it += EACH) {
        const long long tile = (MODE == 0) ? w * a.stride : w;
        const uint32_t acc = it & 1, acc_phase = (it >> 1) & 1;
        const long long row = tile * TC_ROWS + quad * 32 + lane;
        const bool row_ok = MODE == 1 || (row < a.rows && row_eligible(a.mask, a.mask_row0, row));   // collect pass: asked of rows that pass
        // the row's scale; with the bias it is fetched only when a row passes the filter
        float rs = (I8 && !FOLDED && row < a.rows) ? __ldg(a.row_scale + row) : 0.f;
        bool have_rs = false;
        int x_row = 0;
        bool ok = mbar_wait(tfull_bar(acc), acc_phase, verr);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        const uint32_t taddr = tmem_base + acc * NQ + ((uint32_t)(quad * 32) << 16) + part * CW;
        if (MODE == 1) {
          // the warp's whole slice of the tile (32 rows x CW queries) in one round trip to TMEM, then the accumulator
          // goes straight back to the MMA warp: the filtering below works from registers
          uint32_t rr[CW / CH][CH];
#pragma unroll
          for (int c = 0; c < CW / CH; ++c) tmem_ld_chunk<CH>(taddr + c * CH, rr[c]);
          tmem_ld_wait();
          tc_fence_before();
          mbar_arrive(tempty_bar(acc));
#pragma unroll
          for (int c = 0; c < CW / CH; ++c) {
            uint32_t (&r)[CH] = rr[c];
            const int u0 = part * CW + c * CH;
            // First a filter.  Survivors are a few in 10^4 .. 10^5 elements, so for most groups the warp stops here; the exact
            // per-column test below runs only for the rows that pass.
            bool pass = true;
            if (FOLDED) {
              // sums below zero are no hits (the threshold is part of the sum)
              uint32_t sign = r[0] & r[1];
#pragma unroll
              for (int k = 2; k < CH; k += 2) sign &= r[k] & r[k + 1];
              pass = (int)sign >= 0 || ((open >> (u0 / CH)) & 1);
            } else if (!I8) {
              // the largest of the row's CH scores against the smallest of the CH thresholds
              float mx = max3(__uint_as_float(r[0]), __uint_as_float(r[1]), __uint_as_float(r[2]));
#pragma unroll
              for (int k = 3; k + 1 < CH; k += 2) mx = max3(mx, __uint_as_float(r[k]), __uint_as_float(r[k + 1]));
              mx = fmaxf(mx, __uint_as_float(r[CH - 1]));
              pass = mx >= s_thr_min[u0 / CH];
            }
            uint32_t rows_left = __ballot_sync(0xffffffffu, pass);
            if (rows_left) rows_left &= __ballot_sync(0xffffffffu, row < a.rows && row_eligible(a.mask, a.mask_row0, row));
            if (FOLDED && rows_left && !have_rs) {
              rs = row < a.rows ? __ldg(a.row_scale + row) : 0.f;
              x_row = bias_x(bias_c, rs);
              have_rs = true;
            }
            if (FOLDED ? __popc(rows_left) > 4 : I8) {
              // More rows than are worth testing one by one: the bias said nothing about some query (its threshold is not
              // positive, or out of the bias' range), or the rows' scales lie too far apart.  Or there is no bias.  The largest of the row's
              // scores against the smallest threshold, then.  float(dot) * query scale without a conversion per element (those run
              // at a fraction of the fp32 rate): 1.5 * 2^23 + dot is the integer sum of the bit patterns, and the fma takes the
              // offset's product off again.  Two roundings: the product's, at most 0.75 of the query scale, and the fma's, at
              // most 0.25 while |dot| < 2^22 (it is at most 128 * 127 * 256, which leaves 0.998 in all).  With the margin of one
              // scale the bound is not below the unrounded dot * scale, so the roundings of the tested value, which keep order,
              // cannot put it above the bound's.  A scale below zero (or no number) turns the order round: no filter then.
              float mx = -INFINITY;
#pragma unroll
              for (int k = 0; k < CH; k += 2) {
                const float4 s2 = s_us2[(u0 + k) >> 1];
                uint32_t d0 = r[k], d1 = r[k + 1];
                if (FOLDED) { d0 += (uint32_t)(x_row * s_t[u0 + k]); d1 += (uint32_t)(x_row * s_t[u0 + k + 1]); }
                const float2 x = make_float2(__uint_as_float(d0 + S8_OFFSET_BITS), __uint_as_float(d1 + S8_OFFSET_BITS));
                const float2 v = __ffma2_rn(x, make_float2(s2.x, s2.y), make_float2(s2.z, s2.w));
                mx = max3(mx, v.x, v.y);
              }
              pass = pass && (!(rs >= 0.f) || !((mx + s_us_max[u0 / CH]) * rs < s_thr_min[u0 / CH]));
              rows_left &= __ballot_sync(0xffffffffu, pass);
            }
            // The few rows that pass, one at a time: the row's scores go through shared memory so that lane k holds column
            // k's, every lane compares with its own column's threshold, and the hits line up in the queue by ballot.  (Each
            // lane testing its own row over all columns cost the warp 150 instructions per group and 90 per hit.)
            while (rows_left) {
              const int src = __ffs(rows_left) - 1;
              rows_left &= rows_left - 1;
              if (lane == src) {
#pragma unroll
                for (int k = 0; k < CH; k += 4) *reinterpret_cast<uint4*>(s_row + k) = make_uint4(r[k], r[k + 1], r[k + 2], r[k + 3]);
              }
              __syncwarp();
              const uint32_t word = lane < CH ? s_row[lane] : 0u;
              const int dot = (int)word + (FOLDED ? __shfl_sync(0xffffffffu, x_row, src) * bt_lane[c] : 0);
              const float v = I8 ? s8_value((uint32_t)dot, us_lane[c]) * __shfl_sync(0xffffffffu, rs, src) : __uint_as_float(word);
              const bool hit = lane < CH && v >= t_lane[c];
              const uint32_t hm = __ballot_sync(0xffffffffu, hit);
              if (hm) {
                const int n = __popc(hm);
                if (nq + n > QCAP) { flush_queue(a, queue, nq, lane, flight); nq = 0; __syncwarp(); }
                if (hit) {
                  const uint32_t grow = (uint32_t)(a.row_offset + row - lane + src);
                  queue[nq + __popc(hm & ((1u << lane) - 1u))] = make_uint4(0xFFFFFFFFu - grow, ord32(round_bf(v)), (uint32_t)(u0 + lane), 0u);
                }
                nq += n;
              }
              __syncwarp();
            }
          }
        } else {
#pragma unroll 1
          for (int c = 0; c < CW / CH; ++c) {
            uint32_t r[CH];
            tmem_ld_chunk<CH>(taddr + c * CH, r);
            tmem_ld_wait();
            const int u0 = part * CW + c * CH;
            const long long grp = w * 4 + quad;
            float m[CH];
#pragma unroll
            for (int k = 0; k < CH; ++k) {
              const float v = I8 ? s8_value(r[k], s_us[u0 + k]) * rs : __uint_as_float(r[k]);
              m[k] = row_ok ? round_bf(v) : -INFINITY;
            }
            // Maximum over the 32 rows for every column: at each exchange a lane keeps the half of its columns that its lane
            // bit names and hands over the other half, so lane k ends with column k's and one store writes the group
            // (a warp-wide reduction and a store of its own per column took 3 times the instructions: 995 -> 964 us for the whole
            // call on bf16 rows, 1262 -> 1202 on int8).
            if (CH == 16) {
#pragma unroll
              for (int k = 0; k < CH; ++k) m[k] = fmaxf(m[k], __shfl_xor_sync(0xffffffffu, m[k], 16));
            }
#pragma unroll
            for (int o = CH / 2; o >= 1; o >>= 1) {
              const bool upper = lane & o;
#pragma unroll
              for (int k = 0; k < o; ++k) {
                const float keep = upper ? m[k + o] : m[k], give = upper ? m[k] : m[k + o];
                m[k] = fmaxf(keep, __shfl_xor_sync(0xffffffffu, give, o));
              }
            }
            if (lane < CH && u0 + lane < a.B) a.gmax[(size_t)(u0 + lane) * a.n_groups + grp] = m[0];
          }
          tc_fence_before();
          mbar_arrive(tempty_bar(acc));
        }
        if (MODE == 1 && nq >= QFLUSH) {
          flush_queue(a, queue, nq, lane, flight);
          nq = 0;
          __syncwarp();
        }
      }
      if (MODE == 1) {   // what is left
        flush_queue(a, queue, nq, lane, flight);
        flight.land(a);
      }
    };
    if constexpr (TWO_LOOPS) {
      if (biased) consume(std::true_type()); else consume(std::false_type());
    } else {
      consume(std::integral_constant<bool, BIAS>());
    }
  }

  settle();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 2 * NQ);
  }
}

template <int MODE, bool I8, int NQ, bool BIAS, bool SPLIT>
phx_status launch_scan_tc(const CUtensorMap& map_corpus, const CUtensorMap& map_users, const TcScanArgs& a, int grid, int* err_flag,
                          cudaStream_t stream, std::string& err) {
  const int kblk = a.row_bytes / 128;
  const size_t smem = (size_t)kblk * NQ * 128 + (size_t)scan_stages(BIAS, kblk) * kblk * TC_ROWS * 128 + scan_bias_bytes(BIAS, NQ) + 2 * 256 * 4 + 64 + 128 * 16 + TC_CWARPS * (QCAP * 16 + 128) + 256 + 1024;
  static SmemLimit limit;
  PHX_CUDA_TRY(limit.raise(scan_tc_kernel<MODE, I8, NQ, BIAS, SPLIT>, 226 * 1024), err);
  PHX_CUDA_TRY(launch_programmatic(scan_tc_kernel<MODE, I8, NQ, BIAS, SPLIT>, grid, scan_threads(BIAS), smem, stream, map_corpus, map_users, a, err_flag), err);
  return PHX_OK;
}
// Collect passes of up to 64 queries: int8 rows while no more than a dozen of a tile are expected to pass for some query - the tests of more hold
// the eight warps up - and any rows for up to 16 queries, whose tests half of the warps would be without otherwise.  Whole calls, us, every warp on
// every tile / split: int8 rows, 64 queries, k = 1000: 12.5 M rows 389 / 339, 4 M 161 / 149 (six of a tile), 2 M 113 / 117 (twelve), 1 M 90 / 101, 500 k 78 / 90; 33
// queries: 12.5 M 357 / 315, 2 M 107 / 99, 1 M 84 / 83 (twelve), 150 k 58 / 62; 16 queries: 500 k 66 / 56, 150 k 54 / 48.  bf16 rows, whose copies
// take longer than the tests where few pass: 64 queries, k = 1000: 12.5 M 479 / 480, 1 M 91 / 103, 150 k 71 / 81; 16 queries: 500 k 63 / 56, 150 k 53 / 47.
bool split_tiles(const TcScanArgs& a, double expected) {
  return a.B <= 16 || (a.row_scale != nullptr && expected * a.B * TC_ROWS <= 12.0 * (double)a.rows);
}
template <int MODE, bool I8, bool BIAS>
phx_status launch_scan_nq(const CUtensorMap& map_corpus, const CUtensorMap& map_users, const TcScanArgs& a, double expected, int grid, int* err_flag,
                          cudaStream_t stream, std::string& err) {
  // query columns: the multiple of 64 that holds the batch (the tensor core and the consumers work on all NQ of them)
  if (a.B <= 64) {
    if constexpr (MODE == 1) {
      if (split_tiles(a, expected)) {
        dispatch_note(DK_FORM_SCAN_SPLIT);
        return launch_scan_tc<MODE, I8, 64, BIAS, true>(map_corpus, map_users, a, grid, err_flag, stream, err);
      }
    }
    return launch_scan_tc<MODE, I8, 64, BIAS, false>(map_corpus, map_users, a, grid, err_flag, stream, err);
  }
  if (a.B <= 128) return launch_scan_tc<MODE, I8, 128, BIAS, false>(map_corpus, map_users, a, grid, err_flag, stream, err);
  return launch_scan_tc<MODE, I8, 256, BIAS, false>(map_corpus, map_users, a, grid, err_flag, stream, err);
}

}  // namespace

bool tc_scan_supported(int row_bytes) { return row_bytes == 128 || row_bytes == 256; }

phx_status tc_scan_make_maps(CUtensorMap* map_corpus, CUtensorMap* map_users, const void* corpus, long long rows, int row_bytes,
                             const void* queries, std::string& err) {
  // both are moved as 16-bit columns whatever they hold: the copies and the swizzle only see bytes
  phx_status s = sm100::make_map(map_corpus, static_cast<const bf16*>(corpus), rows, row_bytes / 2, TC_ROWS, err);
  if (s) return s;
  return sm100::make_map(map_users, static_cast<const bf16*>(queries), 256, row_bytes / 2, TC_QBOX, err);
}

phx_status tc_scan_launch(const CUtensorMap& map_corpus, const CUtensorMap& map_users, const TcScanArgs& a, int mode,
                          double expected, int num_sms, int* err_flag, cudaStream_t stream, std::string& err) {
  const long long n_tiles = (a.rows + TC_ROWS - 1) / TC_ROWS;
  const long long n_work = (mode == 0) ? (n_tiles + a.stride - 1) / a.stride : n_tiles;
  const int grid = (int)(n_work < num_sms ? n_work : num_sms);
  if (grid <= 0) return PHX_OK;
  const bool i8 = a.row_scale != nullptr;
  if (mode == 0)
    return i8 ? launch_scan_nq<0, true, false>(map_corpus, map_users, a, expected, grid, err_flag, stream, err)
              : launch_scan_nq<0, false, false>(map_corpus, map_users, a, expected, grid, err_flag, stream, err);
  if (!i8) return launch_scan_nq<1, false, false>(map_corpus, map_users, a, expected, grid, err_flag, stream, err);
  // Scales below zero turn the order of the sums round, and the sign of a sum says nothing in a corpus that has one: every group is
  // open, or the bias is left out (one such row, 12.5 M rows, device us open / without: 256 queries 1545 / 1103, 100 847 / 690, one 539 / 589)
  return a.scales_negative && a.B > 64 ? launch_scan_nq<1, true, false>(map_corpus, map_users, a, expected, grid, err_flag, stream, err)
                           : launch_scan_nq<1, true, true>(map_corpus, map_users, a, expected, grid, err_flag, stream, err);
}

}  // namespace phx
