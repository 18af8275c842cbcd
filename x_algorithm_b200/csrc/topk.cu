// Exhaustive dot-product top-k over a corpus shard without materialising the score matrix
// (reference: users_bf16 @ posts^T -> bf16 scores -> top_k_by_key,
// phoenix/xrex/models/recsys_two_tower_model.py:2455-2516, phoenix/xrex/cuda/top_k_by_key/).
//
//   1. sample pass   every `stride`-th 64-row tile is scored; per user and 16-row group the maximum
//                    score is kept; the pivot of a user is the j-th largest group maximum, with j
//                    chosen so that about 3k corpus rows (more for short lists) are expected at or above it
//   2. collect pass  the whole shard is scored once (corpus read once from HBM, scores live only in
//                    registers); rows with bf16(score) >= pivot are appended to the user's survivor
//                    list as 64-bit keys  ordered(score) << 32 | ~global_row
//   3. select        per user an MSB-first radix select finds the k-th largest key (keys are unique,
//                    so exactly k survive), the k keys are sorted in shared memory and written out
// Ordering by the 64-bit key is (score descending, row ascending): the definitional top-k with ties
// broken by the lower id (jax.lax.top_k, cuda/top_k_by_key/__init__.py:78-80).  The result is exact
// whenever the survivor list holds at least k and at most `cap` rows; otherwise the call reports
// PHX_E_CAPACITY instead of returning a wrong answer.
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include <mutex>
#include <vector>

#include "comm.cuh"
#include "common.cuh"
#include "topk_scan.cuh"

namespace phx {
namespace {

constexpr int TILE_ROWS = 64;
constexpr int SCAN_THREADS = 256;
constexpr int SEL_THREADS = 1024;

__device__ __forceinline__ uint32_t ordered32(float f) {
  if (f == 0.f) f = 0.f;  // -0 -> +0
  uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float from_ordered32(uint32_t o) {
  uint32_t u = (o & 0x80000000u) ? (o & 0x7FFFFFFFu) : ~o;
  return __uint_as_float(u);
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool pred) {
  int sz = pred ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(sz));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N)); }

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// The kernels of one call form a chain of short launches: the conversion of the queries, the tcgen05 scans and the pivot are launched with
// launch_programmatic, let the next one start its set-up as soon as they run themselves, and wait for the one in front before they touch
// memory (the select, the masked rows' padding and the mma.sync scans follow in plain stream order).  One query over 1 M rows 136 -> 131 us
// a call, 16 queries over 50 k rows 99 -> 90.
__device__ __forceinline__ void chain_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// a call's flag and status to the host (close_call)
__global__ void publish_state_kernel(const int* state, volatile int* host) {
  chain_wait();
  if (threadIdx.x < 3) host[threadIdx.x] = state[threadIdx.x];
}

// queries to bf16, and the survivor counts of the call that follows to zero
__global__ void users_to_bf16_kernel(const float* __restrict__ users, bf16* __restrict__ out, int B, int Bpad, int dim, int* counts) {
  chain_wait();
  if (blockIdx.x == 0 && counts) counts[threadIdx.x] = 0;      // 256 threads
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= Bpad * dim) return;
  const int b = i / dim;
  out[i] = (b < B) ? f2bf(users[i]) : f2bf(0.f);
}

__device__ __forceinline__ float to_f32(float x) { return x; }
__device__ __forceinline__ float to_f32(bf16 x) { return __bfloat162float(x); }
__device__ __forceinline__ void mma_16832_s8(int (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Symmetric int8 form of one vector per warp: scale = max(max|x| / 127, 1e-12), q = clip(round_half_even(x / scale),
// -127, 127) - the query side of the reference's int8 scoring (recsys_two_tower_model.py:2523-2526).  Rows past
// n_valid are zero with scale 0.
template <typename Tin>
__global__ void quantize_rows_int8_kernel(const Tin* __restrict__ in, long long n_valid, long long n_rows, int dim,
                                          signed char* __restrict__ out, float* __restrict__ scale, int* counts) {
  chain_wait();
  if (blockIdx.x == 0 && counts) counts[threadIdx.x] = 0;      // 256 threads
  const long long row = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= n_rows) return;
  if (row >= n_valid) {
    for (int d = lane; d < dim; d += 32) out[row * dim + d] = 0;
    if (lane == 0) scale[row] = 0.f;
    return;
  }
  float mx = 0.f;
  for (int d = lane; d < dim; d += 32) mx = fmaxf(mx, fabsf(to_f32(in[row * dim + d])));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  const float sc = fmaxf(mx / 127.0f, 1e-12f);
  for (int d = lane; d < dim; d += 32) {
    const float q = fminf(fmaxf(rintf(to_f32(in[row * dim + d]) / sc), -127.f), 127.f);
    out[row * dim + d] = (signed char)(int)q;
  }
  if (lane == 0) scale[row] = sc;
}

struct ScanArgs {
  const bf16* corpus;      // [rows, dim] bf16, or (i8) [rows, dim] int8
  const bf16* users;       // [Bpad, dim] bf16, or (i8) int8
  long long rows;
  long long row_offset;    // global id of local row 0
  int dim, B, Bpad;
  int stride;              // MODE 0: score tiles t with t % stride == 0
  float* gmax;             // MODE 0: [B][n_groups] group maxima
  long long n_groups;      // sampled groups per user
  const float* pivot;      // MODE 1: [B]
  unsigned long long* surv;  // MODE 1: [B][cap]
  int* counts;             // MODE 1: [B]
  int cap;
  const unsigned int* mask = nullptr;   // eligibility bits of the shard's rows (row_eligible), null = all
  long long mask_row0 = 0;
  const unsigned long long* thr = nullptr;   // MODE 2 / 3: [B] threshold keys (a row counts / is kept when key >= thr[u])
  // int8 corpus (recsys_two_tower_model.py:2518-2533): score = bf16((float(int32 dot) * user_scale[u]) * row_scale[row])
  int i8 = 0;
  const float* user_scale = nullptr;   // [Bpad]
  const float* row_scale = nullptr;    // [rows] of the scanned window
};

// NT = n-tiles (8 users each) per warp; a CTA covers 2 * NT * 8 users x 64 corpus rows per tile.
// MODE 0 sample pass (group maxima), 1 collect pass against a score pivot, 2 count the rows whose 64-bit key is at or
// above a per-user threshold key, 3 collect those rows (the exact passes: no sampling, nothing estimated).
// I8: corpus and queries are int8; every load below moves 16-bit units, so an int8 row is dim / 2 of them and one
// m16n8k32 s8 MMA consumes the bytes one m16n8k16 bf16 MMA would (the fragments' byte layouts coincide).
template <int NT, int MODE, bool I8>
__global__ void __launch_bounds__(SCAN_THREADS) scan_kernel(ScanArgs a) {
  extern __shared__ __align__(16) uint8_t ssm[];
  const int dimw = I8 ? a.dim / 2 : a.dim;   // 16-bit units per row
  const int LD = dimw + 8;
  bf16* s_users = reinterpret_cast<bf16*>(ssm);                    // [Bpad][LD]
  bf16* s_tile = s_users + (size_t)a.Bpad * LD;                    // [2][TILE_ROWS][LD]
  float* s_pivot = reinterpret_cast<float*>(s_tile + 2 * TILE_ROWS * LD);  // [Bpad]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t4 = lane & 3;
  const int mt = warp & 3, half = warp >> 2;
  const int chunks_per_row = dimw / 8;

  for (int c = threadIdx.x; c < a.Bpad * chunks_per_row; c += SCAN_THREADS) {
    const int r = c / chunks_per_row, dc = (c % chunks_per_row) * 8;
    *reinterpret_cast<uint4*>(&s_users[r * LD + dc]) = *reinterpret_cast<const uint4*>(a.users + (size_t)r * dimw + dc);
  }
  if (MODE == 1)
    for (int u = threadIdx.x; u < a.Bpad; u += SCAN_THREADS) s_pivot[u] = (u < a.B) ? a.pivot[u] : INFINITY;
  // exact passes: threshold keys and (MODE 2) this CTA's counts live behind the pivots' slot
  unsigned long long* s_thr = reinterpret_cast<unsigned long long*>(s_pivot + a.Bpad);   // [Bpad]
  int* s_cnt = reinterpret_cast<int*>(s_thr + a.Bpad);                                   // [Bpad]
  if (MODE >= 2)
    for (int u = threadIdx.x; u < a.Bpad; u += SCAN_THREADS) { s_thr[u] = (u < a.B) ? a.thr[u] : ~0ull; s_cnt[u] = 0; }
  float* s_us = reinterpret_cast<float*>(s_cnt + a.Bpad);                                // [Bpad] query scales (int8)
  if (I8)
    for (int u = threadIdx.x; u < a.Bpad; u += SCAN_THREADS) s_us[u] = a.user_scale[u];

  const long long n_tiles = (a.rows + TILE_ROWS - 1) / TILE_ROWS;
  const long long step = (long long)gridDim.x * (MODE == 0 ? a.stride : 1);
  const long long first = (long long)blockIdx.x * (MODE == 0 ? a.stride : 1);

  auto load_tile = [&](long long tile, int buf) {
    const long long r0 = tile * TILE_ROWS;
    bf16* dst = s_tile + (size_t)buf * TILE_ROWS * LD;
    for (int c = threadIdx.x; c < TILE_ROWS * chunks_per_row; c += SCAN_THREADS) {
      const int r = c / chunks_per_row, dc = (c % chunks_per_row) * 8;
      const bool ok = (r0 + r) < a.rows;
      const bf16* src = a.corpus + (size_t)(ok ? (r0 + r) : 0) * dimw + dc;
      cp_async16((uint32_t)__cvta_generic_to_shared(dst + r * LD + dc), src, ok);
    }
    cp_async_commit();
  };

  int buf = 0;
  if (first < n_tiles) load_tile(first, 0);
  for (long long tile = first; tile < n_tiles; tile += step) {
    const long long next = tile + step;
    if (next < n_tiles) { load_tile(next, buf ^ 1); cp_async_wait<1>(); } else { cp_async_wait<0>(); }
    __syncthreads();
    const bf16* tl = s_tile + (size_t)buf * TILE_ROWS * LD;
    float acc[NT][4];
    int acci[I8 ? NT : 1][4];
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
      if (I8) { acci[j][0] = acci[j][1] = acci[j][2] = acci[j][3] = 0; }
    }
    for (int ks = 0; ks < dimw / 16; ++ks) {
      uint32_t af[4];
      ldmatrix_x4(af, (uint32_t)__cvta_generic_to_shared(tl + (mt * 16 + (lane & 15)) * LD + ks * 16 + ((lane >> 4) << 3)));
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        const bf16* up = s_users + ((half * NT + j) * 8 + g) * LD + ks * 16 + 2 * t4;
        if (I8) mma_16832_s8(acci[I8 ? j : 0], af, *reinterpret_cast<const uint32_t*>(up), *reinterpret_cast<const uint32_t*>(up + 8));
        else mma_16816(acc[j], af, *reinterpret_cast<const uint32_t*>(up), *reinterpret_cast<const uint32_t*>(up + 8));
      }
    }
    const long long row_a = tile * TILE_ROWS + mt * 16 + g, row_b = row_a + 8;
    const bool ok_a = row_a < a.rows && row_eligible(a.mask, a.mask_row0, row_a);
    const bool ok_b = row_b < a.rows && row_eligible(a.mask, a.mask_row0, row_b);
    if (I8) {   // (float(dot) * query scale) * row scale, in that order, the cast to bf16 follows below
      const float rs_a = row_a < a.rows ? __ldg(a.row_scale + row_a) : 0.f, rs_b = row_b < a.rows ? __ldg(a.row_scale + row_b) : 0.f;
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        const int u0 = (half * NT + j) * 8 + 2 * t4;
        const float us0 = s_us[u0], us1 = s_us[u0 + 1];
        acc[j][0] = ((float)acci[I8 ? j : 0][0] * us0) * rs_a; acc[j][1] = ((float)acci[I8 ? j : 0][1] * us1) * rs_a;
        acc[j][2] = ((float)acci[I8 ? j : 0][2] * us0) * rs_b; acc[j][3] = ((float)acci[I8 ? j : 0][3] * us1) * rs_b;
      }
    }
    if (MODE == 0) {
      // 16-row group maximum per user (rows past the end count as -inf)
      const long long grp = (tile / a.stride) * 4 + mt;
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        float m0 = fmaxf(ok_a ? round_bf(acc[j][0]) : -INFINITY, ok_b ? round_bf(acc[j][2]) : -INFINITY);
        float m1 = fmaxf(ok_a ? round_bf(acc[j][1]) : -INFINITY, ok_b ? round_bf(acc[j][3]) : -INFINITY);
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) {
          m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, o));
          m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, o));
        }
        if (g == 0) {
          const int u0 = (half * NT + j) * 8 + 2 * t4;
          if (u0 < a.B) a.gmax[(size_t)u0 * a.n_groups + grp] = m0;
          if (u0 + 1 < a.B) a.gmax[(size_t)(u0 + 1) * a.n_groups + grp] = m1;
        }
      }
    } else if (MODE >= 2) {
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        const int u0 = (half * NT + j) * 8 + 2 * t4;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int u = u0 + (e & 1);
          const long long row = (e & 2) ? row_b : row_a;
          if (!((e & 2) ? ok_b : ok_a) || u >= a.B) continue;
          const unsigned long long key = ((unsigned long long)ordered32(round_bf(acc[j][e])) << 32) |
                                         (unsigned long long)(0xFFFFFFFFu - (uint32_t)(a.row_offset + row));
          if (key < s_thr[u]) continue;
          if (MODE == 2) atomicAdd(&s_cnt[u], 1);
          else {
            const int slot = atomicAdd(&a.counts[u], 1);
            if (slot < a.cap) a.surv[(size_t)u * a.cap + slot] = key;
          }
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        const int u0 = (half * NT + j) * 8 + 2 * t4;
        const float2 pv = *reinterpret_cast<const float2*>(&s_pivot[u0]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float v = round_bf(acc[j][e]);
          const float p = (e & 1) ? pv.y : pv.x;
          const long long row = (e & 2) ? row_b : row_a;
          if (v >= p && ((e & 2) ? ok_b : ok_a)) {
            const int u = u0 + (e & 1);
            const int slot = atomicAdd(&a.counts[u], 1);
            if (slot < a.cap)
              a.surv[(size_t)u * a.cap + slot] =
                  ((unsigned long long)ordered32(v) << 32) | (unsigned long long)(0xFFFFFFFFu - (uint32_t)(a.row_offset + row));
          }
        }
      }
    }
    __syncthreads();
    buf ^= 1;
  }
  if (MODE == 2)
    for (int u = threadIdx.x; u < a.B; u += SCAN_THREADS) if (s_cnt[u]) atomicAdd(&a.counts[u], s_cnt[u]);
}

// The digit whose bin holds the `remaining`-th entry from the top of a 256-bin histogram, and its rank inside that bin:
// sel[0], sel[1].  Warp 0 only: lane l sums the eight bins 255 - 8 l .. 248 - 8 l, a prefix sum over the lanes finds the
// lane, that lane walks its bins.  One thread walking all 256 took longer than the rest of a pass: with this, and without the
// merge of a single list, a top-500 of one query over 1 M rows takes 136 us instead of 212, 256 queries over 12.5 M 1.09 ms
// instead of 1.16.
__device__ __forceinline__ void digit_of_rank(const int* s_hist, int remaining, int* sel) {
  if (threadIdx.x >= 32) return;
  const int lane = threadIdx.x;
  int c[8], sum = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) { c[i] = s_hist[255 - 8 * lane - i]; sum += c[i]; }
  int incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += v; }
  int cum = incl - sum;
  // the lane in which the rank is reached; the last one stands in when the histogram holds fewer entries
  const unsigned int reached = __ballot_sync(0xffffffffu, incl >= remaining);
  const int owner = reached ? __ffs(reached) - 1 : 31;
  if (lane == owner) {
    int i = 0;
    while (i < 7 && cum + c[i] < remaining) { cum += c[i]; ++i; }
    sel[0] = 255 - 8 * lane - i; sel[1] = remaining - cum;
  }
}

// ---- MSB-first radix select of the k-th largest 64-bit key among n (one CTA) ------------------------
__device__ unsigned long long radix_kth_largest(const unsigned long long* keys, int n, int k, int* s_hist, int* s_sel) {
  unsigned long long prefix = 0, mask = 0;
  int remaining = k;
  for (int shift = 56; shift >= 0; shift -= 8) {
    for (int i = threadIdx.x; i < 256; i += blockDim.x) s_hist[i] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const unsigned long long v = keys[i];
      if ((v & mask) == prefix) atomicAdd(&s_hist[(int)((v >> shift) & 0xFF)], 1);
    }
    __syncthreads();
    digit_of_rank(s_hist, remaining, s_sel);
    __syncthreads();
    const unsigned long long d = (unsigned long long)s_sel[0];
    remaining = s_sel[1];
    prefix |= d << shift;
    mask |= 0xFFull << shift;
    __syncthreads();
  }
  return prefix;  // the k-th largest key itself
}

// The largest of the block's values, in every thread.
__device__ __forceinline__ uint32_t block_max(uint32_t v, uint32_t* s_red) {
  v = __reduce_max_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = v;
  __syncthreads();
  return __reduce_max_sync(0xffffffffu, s_red[threadIdx.x & 31]);     // 32 warps
}
// Where an entry falls among the 256 uppermost codes (the upper 16 bits of an ordered score) below the largest, 0 = there or further down.
// Scores of one list lie within a few binades of 128 codes each, so that one histogram pass finds the entry of a rank that digits
// take two to eight passes for.
__device__ __forceinline__ int top_bin(uint32_t top, uint32_t ordered) {
  const uint32_t below = (top >> 16) - (ordered >> 16);
  return below < 255u ? 255 - (int)below : 0;
}

__device__ void bitonic_sort_desc(unsigned long long* s, int n_pow2) {
  for (int size = 2; size <= n_pow2; size <<= 1) {
    for (int strd = size >> 1; strd > 0; strd >>= 1) {
      __syncthreads();
      for (int i = threadIdx.x; i < n_pow2 / 2; i += blockDim.x) {
        const int lo = 2 * i - (i & (strd - 1));
        const int hi = lo + strd;
        const bool desc = ((lo & size) == 0);
        const unsigned long long x = s[lo], y = s[hi];
        if ((x < y) == desc) { s[lo] = y; s[hi] = x; }
      }
    }
  }
  __syncthreads();
}

// pivot[u] = j-th largest of gmax[u][0..n_groups); j <= 0 or j > n_groups -> -inf
__global__ void __launch_bounds__(SEL_THREADS) pivot_kernel(const float* __restrict__ gmax, long long n_groups, int j,
                                                            float* __restrict__ pivot) {
  __shared__ int s_hist[256];
  __shared__ int s_sel[2];
  __shared__ uint32_t s_red[32];
  chain_wait();
  const int u = blockIdx.x;
  if (j <= 0 || j > n_groups) { if (threadIdx.x == 0) pivot[u] = -INFINITY; return; }
  const float* gm = gmax + (size_t)u * n_groups;
  // one pass over the codes below the largest, the values in registers as far as they fit (one query over 1 M rows 4.9 -> 2.8 us, 256 queries over
  // 12.5 M 12.6 -> 9.3)
  {
    constexpr int KEEP = 4;
    uint32_t mine[KEEP], top = 0;
#pragma unroll
    for (int e = 0; e < KEEP; ++e) {
      const long long i = threadIdx.x + e * SEL_THREADS;
      mine[e] = i < n_groups ? ordered32(gm[i]) : 0u;
      top = max(top, mine[e]);
    }
    for (long long i = threadIdx.x + KEEP * SEL_THREADS; i < n_groups; i += SEL_THREADS) top = max(top, ordered32(gm[i]));
    if (threadIdx.x < 256) s_hist[threadIdx.x] = 0;
    top = block_max(top, s_red);
#pragma unroll
    for (int e = 0; e < KEEP; ++e) if (threadIdx.x + e * SEL_THREADS < n_groups) atomicAdd(&s_hist[top_bin(top, mine[e])], 1);
    for (long long i = threadIdx.x + KEEP * SEL_THREADS; i < n_groups; i += SEL_THREADS) atomicAdd(&s_hist[top_bin(top, ordered32(gm[i]))], 1);
    __syncthreads();
    digit_of_rank(s_hist, j, s_sel);
    __syncthreads();
    const int d = s_sel[0];
    if (d > 0) {
      if (threadIdx.x == 0) pivot[u] = from_ordered32(((top >> 16) - (uint32_t)(255 - d)) << 16);
      return;
    }
    __syncthreads();
  }
  // further down: two 256-bin passes over the 16 significant bits (values are bf16-representable: the top 16 bits of the ordered key
  // carry everything)
  uint32_t prefix = 0, mask = 0;
  int remaining = j;
  for (int shift = 24; shift >= 16; shift -= 8) {
    for (int i = threadIdx.x; i < 256; i += blockDim.x) s_hist[i] = 0;
    __syncthreads();
    for (long long i = threadIdx.x; i < n_groups; i += blockDim.x) {
      const uint32_t v = ordered32(gm[i]);
      if ((v & mask) == prefix) atomicAdd(&s_hist[(v >> shift) & 0xFF], 1);
    }
    __syncthreads();
    digit_of_rank(s_hist, remaining, s_sel);
    __syncthreads();
    prefix |= (uint32_t)s_sel[0] << shift;
    mask |= 0xFFu << shift;
    remaining = s_sel[1];
    __syncthreads();
  }
  if (threadIdx.x == 0) pivot[u] = from_ordered32(prefix);
}

// keys that the select kernel's shared memory holds: the list and as many again with the last one's code (32 KB at most, or the list)
__host__ __device__ constexpr int sel_room(int kpow2) { return kpow2 < 16 ? 32 : kpow2 < 4096 ? 2 * kpow2 : kpow2; }
// keys[u][0..n_u) -> top k sorted; n_u = min(counts[u], cap) or fixed_n.  status[0] |= 1 on underflow, 2 on overflow
__global__ void __launch_bounds__(SEL_THREADS) select_kernel(const unsigned long long* __restrict__ keys, const int* counts,
                                                             int fixed_n, int cap, int k, int kpow2,
                                                             float* __restrict__ out_scores, long long* __restrict__ out_ids,
                                                             int* status, unsigned long long* __restrict__ out_keys = nullptr,
                                                             int ostride = 0) {
  // ostride: entries per query in the output arrays when they hold more than this kernel's k (the tail is padded by
  // the caller); 0 = k
  // out_keys: write the sorted 64-bit keys themselves (ordered score << 32 | ~row; 0 = empty slot) instead of
  // (score, id) pairs - the form per-shard lists travel in before a merge
  extern __shared__ __align__(16) uint8_t selsm[];
  unsigned long long* s_keys = reinterpret_cast<unsigned long long*>(selsm);  // [sel_room(kpow2)]
  __shared__ int s_hist[256];
  __shared__ int s_sel[2];
  __shared__ uint32_t s_red[32];
  __shared__ int s_first[256], s_next[256];
  __shared__ int s_fill;
  chain_wait();
  const int u = blockIdx.x;
  const size_t ob = (size_t)u * (ostride > 0 ? ostride : k);
  int n = counts ? counts[u] : fixed_n;
  if (counts && n > cap) { if (threadIdx.x == 0) atomicOr(status, 2); n = cap; }
  if (n < k) {
    if (threadIdx.x == 0) atomicOr(status, 1);
    for (int i = threadIdx.x; i < k; i += blockDim.x) {
      if (out_keys) out_keys[ob + i] = 0ull;
      else { out_scores[ob + i] = -INFINITY; out_ids[ob + i] = -1; }
    }
    return;
  }
  const unsigned long long* ku = keys + (size_t)u * cap;
  // One histogram of the codes below the largest finds the k-th entry's code.  Grouped by code the keys from there on are all but sorted: a
  // key's place is its code's first one plus the number of larger keys of the same code (and of equal ones in front of it).  Every key is fetched once, up to four a thread.
  // Lists that reach further down or have many keys of one code take the digits and a sort, as every list did (kernel, us: one query, k = 500
  // 16.3 -> 4.9, 256 queries, k = 1000 39.7 -> 12.1 to 16.4).
  constexpr int KEEP = 4, BIN_MAX = 256;
  unsigned long long mine[KEEP];
  uint32_t top = 0;
#pragma unroll
  for (int e = 0; e < KEEP; ++e) {
    const int i = threadIdx.x + e * SEL_THREADS;
    mine[e] = i < n ? ku[i] : 0ull;
    top = max(top, (uint32_t)(mine[e] >> 32));
  }
  for (int i = threadIdx.x + KEEP * SEL_THREADS; i < n; i += SEL_THREADS) top = max(top, (uint32_t)(ku[i] >> 32));
  if (threadIdx.x < 256) s_hist[threadIdx.x] = 0;
  top = block_max(top, s_red);
#pragma unroll
  for (int e = 0; e < KEEP; ++e) if (threadIdx.x + e * SEL_THREADS < n) atomicAdd(&s_hist[top_bin(top, (uint32_t)(mine[e] >> 32))], 1);
  for (int i = threadIdx.x + KEEP * SEL_THREADS; i < n; i += SEL_THREADS) atomicAdd(&s_hist[top_bin(top, (uint32_t)(ku[i] >> 32))], 1);
  __syncthreads();
  digit_of_rank(s_hist, k, s_sel);
  if (threadIdx.x < 32) {          // first place of every code, and the most keys of one among those taken
    const int lane = threadIdx.x;
    __syncwarp();
    const int d = s_sel[0];
    int c[8], sum = 0, most = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) { const int bin = 255 - 8 * lane - i; c[i] = s_hist[bin]; sum += c[i]; if (bin >= d) most = max(most, c[i]); }
    int at = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, at, o); if (lane >= o) at += v; }
    at -= sum;
#pragma unroll
    for (int i = 0; i < 8; ++i) { s_first[255 - 8 * lane - i] = s_next[255 - 8 * lane - i] = at; at += c[i]; }
    most = __reduce_max_sync(0xffffffffu, most);
    if (lane == 0) s_fill = most;
  }
  __syncthreads();
  const int d = s_sel[0], count = k - s_sel[1] + s_hist[d], most = s_fill;
  if (d > 0 && count <= sel_room(kpow2) && most <= BIN_MAX && (top >> 16) >= 255u) {   // (below that, empty slots have a code of their own)
    auto group = [&](unsigned long long v) {
      const int bin = top_bin(top, (uint32_t)(v >> 32));
      if (bin >= d) s_keys[atomicAdd(&s_next[bin], 1)] = v;
    };
#pragma unroll
    for (int e = 0; e < KEEP; ++e) if (threadIdx.x + e * SEL_THREADS < n) group(mine[e]);
    for (int i = threadIdx.x + KEEP * SEL_THREADS; i < n; i += SEL_THREADS) group(ku[i]);
    __syncthreads();
    for (int i = threadIdx.x; i < count; i += SEL_THREADS) {
      const unsigned long long v = s_keys[i];
      const int bin = top_bin(top, (uint32_t)(v >> 32)), lo = s_first[bin], hi = lo + s_hist[bin];
      int place = lo;
      for (int x = lo; x < hi; ++x) place += s_keys[x] > v || (s_keys[x] == v && x < i) ? 1 : 0;   // (lists to merge may share entries)
      if (place >= k) continue;
      if (out_keys) out_keys[ob + place] = v;
      else {
        out_scores[ob + place] = from_ordered32((uint32_t)(v >> 32));
        out_ids[ob + place] = (long long)(0xFFFFFFFFu - (uint32_t)(v & 0xFFFFFFFFull));
      }
    }
    return;
  }
  __syncthreads();
  const unsigned long long kth = radix_kth_largest(ku, n, k, s_hist, s_sel);
  if (threadIdx.x == 0) s_fill = 0;
  for (int i = threadIdx.x; i < kpow2; i += blockDim.x) s_keys[i] = 0ull;
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const unsigned long long v = ku[i];
    // non-empty keys are unique, so exactly k of them are >= the k-th largest; key 0 (an empty slot of a list that
    // held fewer than k entries) repeats and is never collected: the slots it would fill are zero already
    if (v >= kth && v != 0ull) { const int slot = atomicAdd(&s_fill, 1); if (slot < kpow2) s_keys[slot] = v; }
  }
  __syncthreads();
  bitonic_sort_desc(s_keys, kpow2);
  for (int i = threadIdx.x; i < k; i += blockDim.x) {
    const unsigned long long v = s_keys[i];
    if (out_keys) { out_keys[ob + i] = v; continue; }
    // key 0 is an empty slot (the lists held fewer than k entries): the same (-inf, -1) the underflow path writes
    out_scores[ob + i] = v ? from_ordered32((uint32_t)(v >> 32)) : -INFINITY;
    out_ids[ob + i] = v ? (long long)(0xFFFFFFFFu - (uint32_t)(v & 0xFFFFFFFFull)) : -1ll;
  }
}

// [P][B][k] keys -> keys[B][P*k] (the layout the select kernel reads one query's candidates in)
__global__ void regroup_keys_kernel(const unsigned long long* __restrict__ in, int P, int B, int k, unsigned long long* __restrict__ out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)P * B * k) return;
  const int p = (int)(i / ((long long)B * k));
  const int b = (int)((i / k) % B);
  const int j = (int)(i % k);
  out[((size_t)b * P + p) * k + j] = in[i];
}

// [P][B][k] (score, id) lists -> keys[B][P*k]
__global__ void merge_keys_kernel(const float* __restrict__ scores, const long long* __restrict__ ids, int P, int B, int k,
                                  unsigned long long* __restrict__ keys, int* status) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)P * B * k) return;
  const int p = (int)(i / ((long long)B * k));
  const int b = (int)((i / k) % B);
  const int j = (int)(i % k);
  const long long id = ids[i];
  unsigned long long key = 0ull;  // empty slot (id < 0) sorts last
  if (id > 0xFFFFFFFFll) atomicOr(status, 4);   // does not fit the key's 32 row bits: left out, reported
  else if (id >= 0) key = ((unsigned long long)ordered32(scores[i]) << 32) | (unsigned long long)(0xFFFFFFFFu - (uint32_t)id);
  keys[((size_t)b * P + p) * k + j] = key;
}

int next_pow2(int v) { int p = 1; while (p < v) p <<= 1; return p; }

// Fewer eligible rows than k: the reference's top-k runs over every row with the masked ones at the bf16 minimum
// (recsys_two_tower_model.py:2492-2493), so its list ends with masked rows in ascending row order at that score.
// pad_rows [n_pad] = the first masked rows of the window (global ids); written behind the `have` real entries.
__global__ void pad_masked_kernel(const long long* __restrict__ pad_rows, int n_pad, int have, int k, int B,
                                  float* __restrict__ out_scores, long long* __restrict__ out_ids,
                                  unsigned long long* __restrict__ out_keys) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= B * n_pad) return;
  const int u = i / n_pad, j = i % n_pad;
  const float lowest = __uint_as_float(0xFF7F0000u);            // finfo(bfloat16).min
  const size_t o = (size_t)u * k + have + j;
  if (out_keys) out_keys[o] = ((unsigned long long)ordered32(lowest) << 32) | (unsigned long long)(0xFFFFFFFFu - (uint32_t)pad_rows[j]);
  else { out_scores[o] = lowest; out_ids[o] = pad_rows[j]; }
}

// one word per rank for the all-gather beside the lists: scan status in the low byte, the bounded-wait flag above it
__global__ void pack_status_kernel(const int* status, const int* err_flag, int* out) {
  *out = (*status & 0xFF) | ((*err_flag != 0) ? 0x100 : 0);
}

}  // namespace
}  // namespace phx

using namespace phx;

struct phx_corpus {
  int device = 0;
  long long rows = 0, row_offset = 0;
  int dim = 0, max_queries = 0, max_k = 0, cap = 0;
  int num_sms = 148;
  bf16* data = nullptr;
  bf16* users_bf = nullptr;
  float* gmax = nullptr;
  long long gmax_elems = 0;
  float* pivot = nullptr;
  unsigned long long* surv = nullptr;
  unsigned long long* merge_keys = nullptr;
  size_t merge_keys_elems = 0;
  int* counts = nullptr;
  int* err_flag = nullptr;       // [0] raised by a bounded device-side wait that ran out, [1] its limit, [2] = status
  int* status = nullptr;
  int* state_host = nullptr;     // pinned: flag and status as the last call left them (close_call)
  bool state_fresh = false;      // ... and nothing has changed them since
  bool state_wanted = true;      // false inside phx_retrieve_topk, which gathers the ranks' status words itself
  bool use_tc = false;           // tcgen05 scan of the bf16 rows (dim 64 / 128), else the mma.sync scan
  bool use_tc_i8 = false;        // the same of the int8 rows (dim 128 / 256)
  // int8 form of the corpus (phx_corpus_upload_int8 / phx_corpus_quantize_int8) and whether calls score with it
  signed char* q8 = nullptr;     // [rows, dim]
  float* row_scale = nullptr;    // [rows]
  std::vector<bool> negative;    // rows whose scale is below zero, as uploaded last; empty until there is one
  long long n_negative = 0;
  float* user_scale = nullptr;   // [256]
  bool int8 = false;
  CUtensorMap map_corpus, map_users;
  CUtensorMap map_corpus_i8, map_users_i8;
  CUtensorMap map_window;                    // corpus map of the last scanned window (phx_corpus_topk_window_device)
  long long win_begin = -1, win_end = -1;
  bool win_i8 = false;
  unsigned int* mask = nullptr;              // eligibility bits of the shard's rows (phx_corpus_set_mask), null = all
  std::vector<unsigned int> mask_host;
  long long elig_begin = -1, elig_end = -1, elig_count = 0;   // eligible rows of the last window asked for
  long long* pad_rows = nullptr;             // device [max_k]: the window's first masked rows, for lists longer than its eligible rows
  long long pad_begin = -1, pad_end = -1; int pad_have = 0;
  cudaStream_t stream = nullptr;       // the stream the shard's work is enqueued on: its own, or the caller's
  cudaStream_t own_stream = nullptr;
  unsigned long long* keys_out = nullptr;   // set for one call by phx_corpus_topk_keys_device
  // exact passes (the sampled pivot missed, or phx_corpus_set_exact): per-user threshold keys found by bisection
  bool exact = false;
  bool dense = false;            // set for one call: the sample is drawn for 3k rows whatever the list's length
  unsigned long long* thr = nullptr;        // device [256]
  long long exact_runs = 0;                 // calls completed through the exact passes
  int reran = 0;                            // set by a sync that had to redo the last call
  // the last top-k call, kept so that phx_corpus_sync can redo it when its status says the pivot missed
  struct LastCall {
    bool valid = false; const float* users = nullptr; int B = 0, k = 0; long long row_begin = 0, row_end = 0;
    bool sparse = false;         // its sample was drawn for more than 3k rows
    float* scores = nullptr; long long* ids = nullptr; unsigned long long* keys = nullptr;
  } last;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  std::string err;
};

namespace {

template <int NT, bool I8>
phx_status launch_scan(phx_corpus* c, const ScanArgs& a, int mode, int grid, size_t smem) {
  if (mode == 2) {
    PHX_CUDA_TRY(cudaFuncSetAttribute(scan_kernel<NT, 2, I8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), c->err);
    scan_kernel<NT, 2, I8><<<grid, SCAN_THREADS, smem, c->stream>>>(a);
  } else if (mode == 3) {
    PHX_CUDA_TRY(cudaFuncSetAttribute(scan_kernel<NT, 3, I8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), c->err);
    scan_kernel<NT, 3, I8><<<grid, SCAN_THREADS, smem, c->stream>>>(a);
  } else if (mode == 0) {
    PHX_CUDA_TRY(cudaFuncSetAttribute(scan_kernel<NT, 0, I8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), c->err);
    scan_kernel<NT, 0, I8><<<grid, SCAN_THREADS, smem, c->stream>>>(a);
  } else {
    PHX_CUDA_TRY(cudaFuncSetAttribute(scan_kernel<NT, 1, I8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), c->err);
    scan_kernel<NT, 1, I8><<<grid, SCAN_THREADS, smem, c->stream>>>(a);
  }
  PHX_CUDA_TRY(cudaGetLastError(), c->err);
  return PHX_OK;
}

phx_status run_scan(phx_corpus* c, const ScanArgs& a, int mode, int grid) {
  const int dimw = a.i8 ? a.dim / 2 : a.dim;
  const size_t smem = ((size_t)a.Bpad + 2 * TILE_ROWS) * (dimw + 8) * 2 + (size_t)a.Bpad * (4 + 8 + 4 + 4);   // + pivots, threshold keys, counts, query scales
  if (smem > 200 * 1024) { c->err = "topk: query batch x dim does not fit shared memory"; return PHX_E_CAPACITY; }
  if (a.i8) {
    if (a.Bpad == 16) return launch_scan<1, true>(c, a, mode, grid, smem);
    if (a.Bpad == 64) return launch_scan<4, true>(c, a, mode, grid, smem);
    return launch_scan<16, true>(c, a, mode, grid, smem);
  }
  if (a.Bpad == 16) return launch_scan<1, false>(c, a, mode, grid, smem);
  if (a.Bpad == 64) return launch_scan<4, false>(c, a, mode, grid, smem);
  return launch_scan<16, false>(c, a, mode, grid, smem);
}

// queries into the form the scan in use reads: bf16, or int8 with one scale per query
phx_status convert_users(phx_corpus* c, const float* users_dev, int B, int Bpad) {
  if (c->int8) {
    PHX_CUDA_TRY(launch_programmatic(quantize_rows_int8_kernel<float>, (Bpad + 7) / 8, 256, 0, c->stream, users_dev, (long long)B, (long long)Bpad, c->dim,
                                     reinterpret_cast<signed char*>(c->users_bf), c->user_scale, c->counts), c->err);
  } else {
    PHX_CUDA_TRY(launch_programmatic(users_to_bf16_kernel, (Bpad * c->dim + 255) / 256, 256, 0, c->stream, users_dev, c->users_bf, B, Bpad, c->dim,
                                     c->counts), c->err);
  }
  return PHX_OK;
}

// The end of a call: flag and status follow its kernels into pinned memory, so that the wait for the call is all a check needs
// (with two blocking copies of four bytes behind it one query over 1 M rows took 131 us, with one asynchronous copy 106), by a kernel
// of the call's chain: a copy starts 4 to 8 us after the last kernel.
phx_status close_call(phx_corpus* c) {
  if (c->state_wanted) PHX_CUDA_TRY(launch_programmatic(publish_state_kernel, 1, 32, 0, c->stream, (const int*)c->err_flag, (volatile int*)c->state_host), c->err);
  PHX_CUDA_TRY(cudaEventRecord(c->ev1, c->stream), c->err);
  c->state_fresh = c->state_wanted;
  return PHX_OK;
}

// The top-k of a window without any estimate: per user, bisection on the 64-bit key (bf16 score, then lower row) for a
// threshold that at least k and at most `cap` rows reach, each step one counting scan of the window; then one collect
// scan and the usual select.  Keys are unique, so the bisection always ends (at the latest with exactly k rows), whatever
// the scores look like: many equal scores, clustered rows, a corpus of copies.  Host-driven and synchronous between
// steps; a few tens of scans, for the calls the sampled pivot cannot serve.
phx_status topk_exact(phx_corpus* c, ScanArgs a, int B, int k, float* scores_dev, long long* ids_dev, int ostride = 0) {
  dispatch_note(DK_TOPK_EXACT);
  const long long n_tiles = (a.rows + TILE_ROWS - 1) / TILE_ROWS;
  const int grid = (int)(n_tiles < c->num_sms * 2 ? n_tiles : c->num_sms * 2);
  a.Bpad = B <= 16 ? 16 : (B <= 64 ? 64 : 256);
  a.thr = c->thr;
  { phx_status cs = convert_users(c, c->last.users, B, a.Bpad); if (cs) return cs; }
  std::vector<unsigned long long> lo(B, 0ull), hi(B, ~0ull), thr(B, 0ull);   // count(key >= lo) >= k > count(key >= hi)
  std::vector<int> cnt(B, 0);
  std::vector<char> done(B, 0);
  for (int it = 0; it < 66; ++it) {
    bool all = true;
    for (int u = 0; u < B; ++u) {
      if (!done[u]) { thr[u] = lo[u] + (hi[u] - lo[u]) / 2; all = false; }
    }
    if (all) break;
    PHX_CUDA_TRY(cudaMemcpyAsync(c->thr, thr.data(), (size_t)B * 8, cudaMemcpyHostToDevice, c->stream), c->err);
    PHX_CUDA_TRY(cudaMemsetAsync(c->counts, 0, 256 * 4, c->stream), c->err);
    phx_status s = run_scan(c, a, 2, grid);
    if (s) return s;
    PHX_CUDA_TRY(cudaMemcpyAsync(cnt.data(), c->counts, (size_t)B * 4, cudaMemcpyDeviceToHost, c->stream), c->err);
    PHX_CUDA_TRY(cudaStreamSynchronize(c->stream), c->err);
    for (int u = 0; u < B; ++u) {
      if (done[u]) continue;
      if (cnt[u] >= k) { lo[u] = thr[u]; if (cnt[u] <= c->cap) done[u] = 1; }
      else hi[u] = thr[u];
      if (!done[u] && hi[u] - lo[u] <= 1) { thr[u] = lo[u]; done[u] = 1; }   // lo is the k-th largest key itself
    }
  }
  for (int u = 0; u < B; ++u) if (!done[u]) { c->err = "topk: the exact passes did not converge"; return PHX_E_CAPACITY; }
  PHX_CUDA_TRY(cudaMemcpyAsync(c->thr, thr.data(), (size_t)B * 8, cudaMemcpyHostToDevice, c->stream), c->err);
  PHX_CUDA_TRY(cudaMemsetAsync(c->counts, 0, 256 * 4, c->stream), c->err);
  PHX_CUDA_TRY(cudaMemsetAsync(c->status, 0, 4, c->stream), c->err);
  phx_status s = run_scan(c, a, 3, grid);
  if (s) return s;
  const int kp2 = next_pow2(k);
  select_kernel<<<B, SEL_THREADS, (size_t)sel_room(kp2) * 8, c->stream>>>(c->surv, c->counts, 0, c->cap, k, kp2, scores_dev, ids_dev,
                                                               c->status, c->keys_out, ostride);
  PHX_CUDA_TRY(cudaGetLastError(), c->err);
  PHX_CUDA_TRY(cudaStreamSynchronize(c->stream), c->err);   // the host vectors above were the copies' sources
  c->exact_runs++;
  return PHX_OK;
}

}  // namespace

extern "C" {

phx_status phx_corpus_create(int32_t device, int64_t rows, int32_t dim, int64_t row_offset, int32_t max_queries,
                             int32_t max_k, phx_corpus** out) {
  if (!out || rows <= 0 || dim <= 0 || dim % 16 != 0 || dim > 512 || max_queries <= 0 || max_queries > 256 ||
      max_k <= 0 || max_k > 4096 || row_offset < 0 || rows + row_offset > 0xFFFFFFFFll) {
    set_global_error("phx_corpus_create: bad argument (dim % 16 == 0, <= 256 queries, k <= 4096, global rows < 2^32)");
    return PHX_E_ARG;
  }
  phx_corpus* c = new phx_corpus();
  c->device = device; c->rows = rows; c->dim = dim; c->row_offset = row_offset; c->max_queries = max_queries; c->max_k = max_k;
  c->cap = 64 * max_k > 32768 ? 64 * max_k : 32768;
  auto fail = [&](const std::string& m) { set_global_error(m); phx_corpus_destroy(c); return PHX_E_CUDA; };
  if (cudaSetDevice(device) != cudaSuccess) return fail("cudaSetDevice failed");
  cudaDeviceProp prop;
  if (cudaGetDeviceProperties(&prop, device) != cudaSuccess) return fail("cudaGetDeviceProperties failed");
  c->num_sms = prop.multiProcessorCount;
#define CU(x) do { cudaError_t _e = (x); if (_e != cudaSuccess) return fail(std::string(#x) + ": " + cudaGetErrorString(_e)); } while (0)
  CU(cudaStreamCreateWithFlags(&c->own_stream, cudaStreamNonBlocking));
  c->stream = c->own_stream;
  CU(cudaEventCreate(&c->ev0)); CU(cudaEventCreate(&c->ev1));
  CU(cudaMalloc(&c->data, (size_t)rows * dim * 2));
  CU(cudaMalloc(&c->users_bf, (size_t)256 * dim * 2));
  const long long n_tiles = (rows + TILE_ROWS - 1) / TILE_ROWS;
  c->gmax_elems = (long long)max_queries * n_tiles * 4;  // stride 1 worst case
  // the sample never needs more than ~ (64 * j) groups; bound the buffer at 64M floats
  if (c->gmax_elems > (64ll << 20)) c->gmax_elems = 64ll << 20;
  CU(cudaMalloc(&c->gmax, (size_t)c->gmax_elems * 4));
  CU(cudaMalloc(&c->pivot, 256 * 4));
  CU(cudaMalloc(&c->surv, (size_t)max_queries * c->cap * 8));
  CU(cudaMalloc(&c->counts, 256 * 4));
  CU(cudaMalloc(&c->thr, 256 * 8));
  CU(cudaMalloc(&c->err_flag, 16));   // [0] flag, [1] wait limit in microseconds (0 = default), [2] status
  CU(cudaMemset(c->err_flag, 0, 16));
  c->status = c->err_flag + 2;
  CU(cudaMallocHost(&c->state_host, 16));
#undef CU
  {
    const char* force = getenv("PHX_TOPK");
    const bool tc = prop.major == 10 && !(force && strcmp(force, "simt") == 0);
    c->use_tc = tc && tc_scan_supported(dim * 2);
    c->use_tc_i8 = tc && tc_scan_supported(dim);
    if (c->use_tc) {
      std::string err;
      phx_status s = tc_scan_make_maps(&c->map_corpus, &c->map_users, c->data, rows, dim * 2, c->users_bf, err);
      if (s) { set_global_error(err); phx_corpus_destroy(c); return s; }
    }
  }
  *out = c;
  return PHX_OK;
}

void phx_corpus_destroy(phx_corpus* c) {
  if (!c) return;
  cudaSetDevice(c->device);
  if (c->stream) cudaStreamSynchronize(c->stream);
  auto fr = [](void* p) { if (p) cudaFree(p); };
  fr(c->data); fr(c->users_bf); fr(c->gmax); fr(c->pivot); fr(c->surv); fr(c->merge_keys); fr(c->counts); fr(c->err_flag); fr(c->mask); fr(c->thr); fr(c->pad_rows); fr(c->q8); fr(c->row_scale); fr(c->user_scale);
  if (c->ev0) cudaEventDestroy(c->ev0);
  if (c->ev1) cudaEventDestroy(c->ev1);
  if (c->state_host) cudaFreeHost(c->state_host);
  if (c->own_stream) cudaStreamDestroy(c->own_stream);
  delete c;
}

const char* phx_corpus_last_error(const phx_corpus* c) { return c ? c->err.c_str() : phx_global_error(); }

phx_status phx_corpus_upload(phx_corpus* c, int64_t row0, int64_t nrows, const uint16_t* host_bf16) {
  if (!c || !host_bf16 || row0 < 0 || nrows < 0 || row0 + nrows > c->rows) { if (c) c->err = "phx_corpus_upload: range"; return PHX_E_ARG; }
  cudaSetDevice(c->device);
  PHX_CUDA_TRY(cudaMemcpy(c->data + row0 * c->dim, host_bf16, (size_t)nrows * c->dim * 2, cudaMemcpyHostToDevice), c->err);
  return PHX_OK;
}

phx_status phx_corpus_read_device(phx_corpus* c, int64_t row0, int64_t nrows, uint16_t* out_dev) {
  if (!c || !out_dev || row0 < 0 || nrows < 0 || row0 + nrows > c->rows) { if (c) c->err = "phx_corpus_read_device: range"; return PHX_E_ARG; }
  cudaSetDevice(c->device);
  PHX_CUDA_TRY(cudaMemcpyAsync(out_dev, c->data + row0 * c->dim, (size_t)nrows * c->dim * 2, cudaMemcpyDeviceToDevice, c->stream), c->err);
  PHX_CUDA_TRY(cudaStreamSynchronize(c->stream), c->err);
  return PHX_OK;
}

phx_status phx_corpus_fill_synthetic(phx_corpus* c, uint32_t seed) {
  if (!c) return PHX_E_ARG;
  cudaSetDevice(c->device);
  phx_status s = corpus_fill_launch(c->data, c->row_offset, c->rows, c->dim, seed, c->stream, c->err);
  if (s) return s;
  PHX_CUDA_TRY(cudaStreamSynchronize(c->stream), c->err);
  return PHX_OK;
}

namespace {
phx_status ensure_int8_buffers(phx_corpus* c) {
  if (c->dim % 32 != 0) { c->err = "int8 corpus: dim must be a multiple of 32"; return PHX_E_ARG; }
  if (!c->q8) PHX_CUDA_TRY(cudaMalloc(&c->q8, (size_t)c->rows * c->dim), c->err);
  if (!c->row_scale) PHX_CUDA_TRY(cudaMalloc(&c->row_scale, (size_t)c->rows * 4), c->err);
  if (!c->user_scale) PHX_CUDA_TRY(cudaMalloc(&c->user_scale, 256 * 4), c->err);
  if (c->use_tc_i8) return tc_scan_make_maps(&c->map_corpus_i8, &c->map_users_i8, c->q8, c->rows, c->dim, c->users_bf, c->err);
  return PHX_OK;
}
}  // namespace

phx_status phx_corpus_upload_int8(phx_corpus* c, int64_t row0, int64_t nrows, const int8_t* host_q8, const float* host_scales) {
  if (!c || !host_q8 || !host_scales || row0 < 0 || nrows < 0 || row0 + nrows > c->rows) { if (c) c->err = "phx_corpus_upload_int8: range"; return PHX_E_ARG; }
  cudaSetDevice(c->device);
  phx_status s = ensure_int8_buffers(c);
  if (s) return s;
  PHX_CUDA_TRY(cudaMemcpy(c->q8 + row0 * c->dim, host_q8, (size_t)nrows * c->dim, cudaMemcpyHostToDevice), c->err);
  for (int64_t i = 0; i < nrows; ++i) {
    const bool neg = host_scales[i] < 0.f;
    if (neg && c->negative.empty()) c->negative.assign((size_t)c->rows, false);
    if (c->negative.empty() || c->negative[row0 + i] == neg) continue;
    c->negative[row0 + i] = neg;
    c->n_negative += neg ? 1 : -1;
  }
  PHX_CUDA_TRY(cudaMemcpy(c->row_scale + row0, host_scales, (size_t)nrows * 4, cudaMemcpyHostToDevice), c->err);
  return PHX_OK;
}

phx_status phx_corpus_quantize_int8(phx_corpus* c) {
  if (!c) return PHX_E_ARG;
  cudaSetDevice(c->device);
  phx_status s = ensure_int8_buffers(c);
  if (s) return s;
  std::vector<bool>().swap(c->negative);      // the kernel's scales are at least 1e-12
  c->n_negative = 0;
  quantize_rows_int8_kernel<bf16><<<(unsigned)((c->rows + 7) / 8), 256, 0, c->stream>>>(c->data, c->rows, c->rows, c->dim, c->q8, c->row_scale, nullptr);
  PHX_CUDA_TRY(cudaGetLastError(), c->err);
  PHX_CUDA_TRY(cudaStreamSynchronize(c->stream), c->err);
  return PHX_OK;
}

phx_status phx_corpus_set_int8(phx_corpus* c, int32_t on) {
  if (!c) return PHX_E_ARG;
  if (on && !c->q8) { c->err = "phx_corpus_set_int8: no int8 rows (phx_corpus_upload_int8 / phx_corpus_quantize_int8)"; return PHX_E_STATE; }
  cudaSetDevice(c->device);
  PHX_CUDA_TRY(cudaStreamSynchronize(c->stream), c->err);
  c->int8 = on != 0;
  c->last.valid = false;
  return PHX_OK;
}

phx_status phx_corpus_read_int8_device(phx_corpus* c, int64_t row0, int64_t nrows, int8_t* q8_dev, float* scales_dev) {
  if (!c || !q8_dev || !scales_dev || !c->q8 || row0 < 0 || nrows < 0 || row0 + nrows > c->rows) { if (c) c->err = "phx_corpus_read_int8_device: range or no int8 rows"; return PHX_E_ARG; }
  cudaSetDevice(c->device);
  PHX_CUDA_TRY(cudaMemcpyAsync(q8_dev, c->q8 + row0 * c->dim, (size_t)nrows * c->dim, cudaMemcpyDeviceToDevice, c->stream), c->err);
  PHX_CUDA_TRY(cudaMemcpyAsync(scales_dev, c->row_scale + row0, (size_t)nrows * 4, cudaMemcpyDeviceToDevice, c->stream), c->err);
  PHX_CUDA_TRY(cudaStreamSynchronize(c->stream), c->err);
  return PHX_OK;
}

phx_status phx_corpus_set_mask(phx_corpus* c, const uint32_t* host_bits) {
  if (!c) return PHX_E_ARG;
  cudaSetDevice(c->device);
  PHX_CUDA_TRY(cudaStreamSynchronize(c->stream), c->err);   // no scan may be reading the old bits
  c->elig_begin = c->elig_end = -1;
  c->pad_begin = c->pad_end = -1;
  if (!host_bits) {
    if (c->mask) cudaFree(c->mask);
    c->mask = nullptr; c->mask_host.clear();
    return PHX_OK;
  }
  const size_t words = (size_t)((c->rows + 31) / 32);
  c->mask_host.assign(host_bits, host_bits + words);
  if (c->rows & 31) c->mask_host[words - 1] &= (1u << (c->rows & 31)) - 1u;   // bits past the last row do not count
  if (!c->mask) PHX_CUDA_TRY(cudaMalloc(&c->mask, words * 4), c->err);
  PHX_CUDA_TRY(cudaMemcpy(c->mask, c->mask_host.data(), words * 4, cudaMemcpyHostToDevice), c->err);
  return PHX_OK;
}

phx_status phx_corpus_topk_window_device(phx_corpus* c, const float* users_dev, int32_t B, int32_t k, int64_t row_begin,
                                         int64_t row_end, float* scores_dev, int64_t* ids_dev) {
  if (!c || !users_dev || ((!scores_dev || !ids_dev) && !c->keys_out)) return PHX_E_ARG;
  if (B <= 0 || B > c->max_queries || k <= 0 || k > c->max_k) { c->err = "topk: B or k exceeds what the corpus was created for"; return PHX_E_CAPACITY; }
  if (row_begin < 0 || row_end > c->rows || row_begin >= row_end) { c->err = "topk: window outside the shard's rows"; return PHX_E_ARG; }
  // the window [row_begin, row_end) of the shard scanned as a corpus of its own: rows, first row and global id of row 0
  const long long rows = row_end - row_begin, roff = c->row_offset + row_begin;
  const bool tc = c->int8 ? c->use_tc_i8 : c->use_tc;
  const int row_bytes = c->int8 ? c->dim : c->dim * 2;
  const bf16* data = c->int8 ? reinterpret_cast<const bf16*>(c->q8 + row_begin * (long long)c->dim) : c->data + row_begin * (long long)c->dim;
  if (k > rows) { c->err = "topk: k exceeds the rows of the window"; return PHX_E_ARG; }
  if (c->mask) {
    // eligible rows of the window (counted once per window on the host copy of the mask)
    if (c->elig_begin != row_begin || c->elig_end != row_end) {
      long long n = 0;
      for (long long r = row_begin; r < row_end;) {
        if ((r & 31) == 0 && r + 32 <= row_end) { n += __builtin_popcount(c->mask_host[r >> 5]); r += 32; }
        else { n += (c->mask_host[r >> 5] >> (r & 31)) & 1u; ++r; }
      }
      c->elig_begin = row_begin; c->elig_end = row_end; c->elig_count = n;
    }
  }
  // k_real entries come from the scan; a window with fewer eligible rows than k is completed with its first masked
  // rows at the bf16 minimum, as the reference's top-k over masked scores does
  const int k_real = (c->mask && k > c->elig_count) ? (int)c->elig_count : k;
  const int n_pad = k - k_real;
  if (n_pad > 0) {
    if (c->pad_begin != row_begin || c->pad_end != row_end || c->pad_have < n_pad) {
      std::vector<long long> rows_h;
      rows_h.reserve(n_pad);
      for (long long r = row_begin; r < row_end && (int)rows_h.size() < n_pad; ++r)
        if (!((c->mask_host[r >> 5] >> (r & 31)) & 1u)) rows_h.push_back(c->row_offset + r);
      if (!c->pad_rows) PHX_CUDA_TRY(cudaMalloc(&c->pad_rows, (size_t)c->max_k * sizeof(long long)), c->err);
      cudaSetDevice(c->device);
      PHX_CUDA_TRY(cudaMemcpyAsync(c->pad_rows, rows_h.data(), rows_h.size() * sizeof(long long), cudaMemcpyHostToDevice, c->stream), c->err);
      PHX_CUDA_TRY(cudaStreamSynchronize(c->stream), c->err);   // rows_h goes out of scope
      c->pad_begin = row_begin; c->pad_end = row_end; c->pad_have = n_pad;
    }
  }
  cudaSetDevice(c->device);
  const CUtensorMap* map_corpus = c->int8 ? &c->map_corpus_i8 : &c->map_corpus;
  const CUtensorMap& map_users = c->int8 ? c->map_users_i8 : c->map_users;
  if (tc && (row_begin != 0 || row_end != c->rows)) {
    if (c->win_begin != row_begin || c->win_end != row_end || c->win_i8 != c->int8) {
      CUtensorMap users_unused;
      phx_status ms = tc_scan_make_maps(&c->map_window, &users_unused, data, rows, row_bytes, c->users_bf, c->err);
      if (ms) return ms;
      c->win_begin = row_begin; c->win_end = row_end; c->win_i8 = c->int8;
    }
    map_corpus = &c->map_window;
  }
  const int Bpad = tc ? 256 : (B <= 16 ? 16 : (B <= 64 ? 64 : 256));
  auto pad_tail = [&]() -> phx_status {
    if (n_pad == 0) return PHX_OK;
    pad_masked_kernel<<<(B * n_pad + 255) / 256, 256, 0, c->stream>>>(c->pad_rows, n_pad, k_real, k, B, scores_dev, (long long*)ids_dev, c->keys_out);
    PHX_CUDA_TRY(cudaGetLastError(), c->err);
    return PHX_OK;
  };
  c->last.valid = true; c->last.users = users_dev; c->last.B = B; c->last.k = k; c->last.row_begin = row_begin;
  c->last.row_end = row_end; c->last.scores = scores_dev; c->last.ids = (long long*)ids_dev; c->last.keys = c->keys_out;
  c->last.sparse = false;
  c->state_fresh = false;
  PHX_CUDA_TRY(cudaEventRecord(c->ev0, c->stream), c->err);
  if (c->exact) {
    ScanArgs xa;
    xa.corpus = data; xa.users = c->users_bf; xa.rows = rows; xa.row_offset = roff; xa.dim = c->dim; xa.B = B; xa.Bpad = Bpad;
    xa.stride = 1; xa.gmax = c->gmax; xa.n_groups = 0; xa.pivot = c->pivot; xa.surv = c->surv; xa.counts = c->counts; xa.cap = c->cap;
    xa.mask = c->mask; xa.mask_row0 = row_begin;
    xa.i8 = c->int8 ? 1 : 0; xa.user_scale = c->user_scale; xa.row_scale = c->int8 ? c->row_scale + row_begin : nullptr;
    if (k_real > 0) {
      phx_status xs = topk_exact(c, xa, B, k_real, scores_dev, (long long*)ids_dev, k);
      if (xs) return xs;
    }
    { phx_status ps = pad_tail(); if (ps) return ps; }
    return close_call(c);
  }
  if (k_real == 0) {   // nothing eligible in the window: the list is all padding
    phx_status ps = pad_tail();
    if (ps) return ps;
    return close_call(c);
  }
  { phx_status cs = convert_users(c, users_dev, B, Bpad); if (cs) return cs; }

  // geometry of the scan in use: tile rows, rows per maximum group
  const int tile_rows = tc ? 128 : TILE_ROWS;
  const double group_rows = tc ? 32.0 : 16.0;
  ScanArgs a;
  a.corpus = data; a.users = c->users_bf; a.rows = rows; a.row_offset = roff; a.dim = c->dim; a.B = B; a.Bpad = Bpad;
  a.stride = 1; a.gmax = c->gmax; a.n_groups = 0; a.pivot = c->pivot; a.surv = c->surv; a.counts = c->counts; a.cap = c->cap;
  a.mask = c->mask; a.mask_row0 = row_begin;
  a.i8 = c->int8 ? 1 : 0; a.user_scale = c->user_scale; a.row_scale = c->int8 ? c->row_scale + row_begin : nullptr;
  TcScanArgs ta;
  ta.mask = c->mask; ta.mask_row0 = row_begin;
  if (c->int8) { ta.user_scale = c->user_scale; ta.row_scale = c->row_scale + row_begin; ta.scales_negative = c->n_negative > 0 ? 1 : 0; }
  ta.rows = rows; ta.row_offset = roff; ta.row_bytes = row_bytes; ta.B = B; ta.stride = 1; ta.gmax = c->gmax; ta.n_groups = 0;
  ta.pivot = c->pivot; ta.surv = c->surv; ta.counts = c->counts; ta.cap = c->cap;
  const long long n_tiles = (rows + tile_rows - 1) / tile_rows;
  int j = 0;
  double expected = c->mask ? (double)c->elig_count : (double)rows;    // rows of a query's list before the select
  // a window whose eligible rows all fit the survivor buffer needs no pivot: every eligible row is collected
  if (rows > c->cap && !(c->mask && c->elig_count <= c->cap)) {
    // Rows wanted at or above the pivot, and how many of them (`picks`) the sample is to hold: every (want / picks)-th tile is scored for
    // it.  3k and 48 serve every list; a list of 10 has every tile scored twice that way.  A short list may want more rows: a wanted row costs
    // about 0.14 ns a query in the collect pass and the select, a sampled tile as much as a collected one, and the more rows a list
    // has to spare the fewer picks keep it from running short: with want = r k and j picks that is the chance of a sum of j exponential
    // variables below j / r, at most exp(-j (1 / r - 1 + ln r)) (Chernoff), here e^-14 a query, and a call that missed is done again.
    // Where the good rows stand together - a topic uploaded in a row, a mask that leaves one range - a block of L rows shows in
    // L picks / (group_rows want) groups of the sample, and with fewer of them than the picks the pivot falls below the block: want is
    // bounded so that a block as long as the survivor buffer has half as many again.
    // Whole calls, us, 3k rows and 48 picks / up to 3000 rows and 48 picks / this rule: k = 10: 12.5 M rows, 256 queries 1466 / 726 / 680, one query
    // 1139 / 497 / 504, 3 M rows 336 / 162 / 162, 700 k rows, 16 queries 143 / 86 / 79; k = 100, 256 queries 983 / 765 / 683; k = 200, 10 queries
    // 572 / 519 / 523; 1.2 M rows with one block of 40 k 168 / 1337 / 81.
    const double limit = c->dense ? 0.0 : (double)c->cap / (1.5 * group_rows), unit = 17.5 * (double)rows / (double)B;
    double want = 3.0 * k_real, picks = 48.0, cost = want + unit / want;
    for (double w = want; w < limit;) {
      w = fmin(1.25 * w, limit);
      const double r = w / k_real, j = fmin(48.0, fmax(16.0, 14.0 / (1.0 / r - 1.0 + log(r)))), t = w + unit * (j / 48.0) / w;
      if (t < cost) { want = w; picks = j; cost = t; }
    }
    c->last.sparse = want > 3.0 * k_real;
    expected = want;
    long long stride = (long long)(want / picks);
    if (stride < 1) stride = 1;
    long long sampled_tiles = (n_tiles + stride - 1) / stride;
    while (sampled_tiles * 4 * (long long)B > c->gmax_elems) { stride *= 2; sampled_tiles = (n_tiles + stride - 1) / stride; }
    a.stride = ta.stride = (int)stride;
    a.n_groups = ta.n_groups = sampled_tiles * 4;
    // per-row tail fraction f = want / rows; a group of g rows exceeds the level with 1 - (1-f)^g
    const double f = want / (double)rows;
    const double qg = 1.0 - pow(1.0 - (f < 0.5 ? f : 0.5), group_rows);
    j = (int)ceil(qg * (double)a.n_groups);
    if (j < 1) j = 1;
    phx_status s;
    dispatch_note(tc ? DK_SCAN_TC : DK_SCAN_MMA);
    if (tc) s = tc_scan_launch(*map_corpus, map_users, ta, 0, expected, c->num_sms, c->err_flag, c->stream, c->err);
    else s = run_scan(c, a, 0, (int)(sampled_tiles < c->num_sms * 2 ? sampled_tiles : c->num_sms * 2));
    if (s) return s;
  }
  PHX_CUDA_TRY(launch_programmatic(pivot_kernel, B, SEL_THREADS, 0, c->stream, c->gmax, a.n_groups, j, c->pivot), c->err);
  {
    phx_status s;
    dispatch_note(tc ? DK_SCAN_TC : DK_SCAN_MMA);
    if (tc) s = tc_scan_launch(*map_corpus, map_users, ta, 1, expected, c->num_sms, c->err_flag, c->stream, c->err);
    else s = run_scan(c, a, 1, (int)(n_tiles < c->num_sms * 2 ? n_tiles : c->num_sms * 2));
    if (s) return s;
  }
  const int kp2 = next_pow2(k_real);
  // In plain stream order: a CTA that comes up beside the scan's is left with the L1 that the scan's shared memory leaves over, and
  // reads a long list up to eight times (30 k rows, all of them survivors, the digits alone: 164 us a call instead of 142).
  select_kernel<<<B, SEL_THREADS, (size_t)sel_room(kp2) * 8, c->stream>>>(c->surv, c->counts, 0, c->cap, k_real, kp2, scores_dev,
                                                               (long long*)ids_dev, c->status, c->keys_out, k);
  PHX_CUDA_TRY(cudaGetLastError(), c->err);
  { phx_status ps = pad_tail(); if (ps) return ps; }
  return close_call(c);
}

phx_status phx_corpus_topk_device(phx_corpus* c, const float* users_dev, int32_t B, int32_t k, float* scores_dev,
                                  int64_t* ids_dev) {
  if (!c) return PHX_E_ARG;
  if (k > c->rows) { c->err = "topk: k exceeds the shard's rows"; return PHX_E_ARG; }
  return phx_corpus_topk_window_device(c, users_dev, B, k, 0, c->rows, scores_dev, ids_dev);
}

phx_status phx_corpus_topk_keys_device(phx_corpus* c, const float* users_dev, int32_t B, int32_t k, uint64_t* keys_dev) {
  if (!c || !keys_dev) return PHX_E_ARG;
  if (k > c->rows) { c->err = "topk: k exceeds the shard's rows"; return PHX_E_ARG; }
  c->keys_out = (unsigned long long*)keys_dev;
  const phx_status s = phx_corpus_topk_window_device(c, users_dev, B, k, 0, c->rows, nullptr, nullptr);
  c->keys_out = nullptr;
  return s;
}

phx_status phx_topk_merge_keys_device(phx_corpus* c, const uint64_t* keys_dev, int32_t P, int32_t B, int32_t k,
                                      float* out_scores_dev, int64_t* out_ids_dev) {
  if (!c || !keys_dev || !out_scores_dev || !out_ids_dev || P <= 0 || B <= 0 || k <= 0 || k > 4096) return PHX_E_ARG;
  cudaSetDevice(c->device);
  const size_t need = (size_t)P * B * k;
  c->state_fresh = false;
  if (need > c->merge_keys_elems) {
    if (c->merge_keys) cudaFree(c->merge_keys);
    c->merge_keys = nullptr;
    PHX_CUDA_TRY(cudaMalloc(&c->merge_keys, need * 8), c->err);
    c->merge_keys_elems = need;
  }
  regroup_keys_kernel<<<(unsigned)((need + 255) / 256), 256, 0, c->stream>>>((const unsigned long long*)keys_dev, P, B, k, c->merge_keys);
  PHX_CUDA_TRY(cudaGetLastError(), c->err);
  const int kp2 = next_pow2(k);
  select_kernel<<<B, SEL_THREADS, (size_t)sel_room(kp2) * 8, c->stream>>>(c->merge_keys, nullptr, P * k, P * k, k, kp2, out_scores_dev,
                                                               (long long*)out_ids_dev, c->status);
  PHX_CUDA_TRY(cudaGetLastError(), c->err);
  return close_call(c);
}

phx_status phx_retrieve_topk(phx_comm* cm, phx_corpus* c, const float* users_dev, int32_t B, int32_t k, float* scores_dev,
                             int64_t* ids_dev, void* stream) {
  if (!cm || !c || !users_dev || !scores_dev || !ids_dev) { set_global_error("phx_retrieve_topk: null argument"); return PHX_E_ARG; }
  if (B <= 0 || B > c->max_queries || k <= 0 || k > c->max_k) { c->err = cm->err = "phx_retrieve_topk: B or k exceeds what the shard was created for"; return PHX_E_CAPACITY; }
  if (k > c->rows) { c->err = cm->err = "phx_retrieve_topk: k exceeds the shard's rows"; return PHX_E_ARG; }
  if (cm->device != c->device) { c->err = cm->err = "phx_retrieve_topk: communicator and shard live on different devices"; return PHX_E_ARG; }
  cudaSetDevice(c->device);
  const int W = cm->world;
  const size_t per = (size_t)B * k;
  if (per > cm->keys_cap) {
    if (cm->keys_local) cudaFree(cm->keys_local);
    if (cm->keys_all) cudaFree(cm->keys_all);
    cm->keys_local = cm->keys_all = nullptr; cm->keys_cap = 0;
    PHX_CUDA_TRY(cudaMalloc(&cm->keys_local, per * 8), cm->err);
    PHX_CUDA_TRY(cudaMalloc(&cm->keys_all, per * 8 * W), cm->err);
    cm->keys_cap = per;
  }
  cudaStream_t st = (cudaStream_t)stream;
  cudaStream_t saved = c->stream;
  c->stream = st;
  c->state_wanted = false;
  struct Restore {
    phx_corpus* c; cudaStream_t s;
    ~Restore() { c->stream = s; c->keys_out = nullptr; c->exact = c->dense = c->state_fresh = false; c->state_wanted = true; }
  } restore{c, saved};
  int* my_word = cm->status_all + PHX_MAX_SHARDS;
  auto shard_list = [&]() -> phx_status {
    c->keys_out = cm->keys_local;
    const phx_status s = phx_corpus_topk_window_device(c, users_dev, B, k, 0, c->rows, nullptr, nullptr);
    c->keys_out = nullptr;
    return s;
  };
  auto gather_and_merge = [&]() -> phx_status {
    pack_status_kernel<<<1, 1, 0, st>>>(c->status, c->err_flag, my_word);
    PHX_CUDA_TRY(cudaGetLastError(), cm->err);
    phx_status s;
    if ((s = comm_check(cm, cm->api->GroupStart(), "ncclGroupStart"))) return s;
    if ((s = comm_check(cm, cm->api->AllGather(cm->keys_local, cm->keys_all, per, ncclUint64, cm->comm, st), "ncclAllGather (lists)"))) return s;
    if ((s = comm_check(cm, cm->api->AllGather(my_word, cm->status_all, 1, ncclInt32, cm->comm, st), "ncclAllGather (status)"))) return s;
    if ((s = comm_check(cm, cm->api->GroupEnd(), "ncclGroupEnd"))) return s;
    if ((s = phx_topk_merge_keys_device(c, (const uint64_t*)cm->keys_all, W, B, k, scores_dev, ids_dev))) { cm->err = c->err; return s; }
    PHX_CUDA_TRY(cudaMemcpyAsync(cm->status_host, cm->status_all, (size_t)W * sizeof(int), cudaMemcpyDeviceToHost, st), cm->err);
    PHX_CUDA_TRY(cudaStreamSynchronize(st), cm->err);
    return PHX_OK;
  };
  phx_status s;
  if ((s = shard_list())) { cm->err = c->err; return s; }
  // Where the sampled pivot missed on some shard, that shard takes its list again - a short list first with a pivot for 3k rows, then by the
  // exact passes - and every rank gathers and merges again (all ranks hold the same status words, so all take the same turns together)
  const bool sparse = c->last.sparse;
  for (int turn = 0;; ++turn) {
    if ((s = gather_and_merge())) return s;
    int any = 0;
    for (int r = 0; r < W; ++r) any |= cm->status_host[r];
    if (any & 0x100) {
      cudaMemsetAsync(c->err_flag, 0, sizeof(int), st);
      c->err = cm->err = "phx_retrieve_topk: a bounded device-side wait ran out on some rank (scan pipeline)";
      return PHX_E_TIMEOUT;
    }
    if (!(any & 3)) return PHX_OK;
    if (turn == 2) { c->err = cm->err = "phx_retrieve_topk: a shard's exact passes left a status behind"; return PHX_E_CAPACITY; }
    if (cm->status_host[cm->rank] & 3) {
      PHX_CUDA_TRY(cudaMemsetAsync(c->status, 0, sizeof(int), st), cm->err);
      (turn == 0 && sparse ? c->dense : c->exact) = true;
      s = shard_list();
      c->exact = c->dense = false;
      if (s) { cm->err = c->err; return s; }
    }
  }
}

phx_status phx_corpus_set_stream(phx_corpus* c, void* stream, int32_t use_own) {
  if (!c) return PHX_E_ARG;
  c->stream = use_own ? c->own_stream : (cudaStream_t)stream;   // a NULL caller stream is the default stream
  return PHX_OK;
}

phx_status phx_topk_merge_device(phx_corpus* c, const float* scores_dev, const int64_t* ids_dev, int32_t P, int32_t B,
                                 int32_t k, float* out_scores_dev, int64_t* out_ids_dev) {
  if (!c || !scores_dev || !ids_dev || !out_scores_dev || !out_ids_dev || P <= 0 || B <= 0 || k <= 0 || k > 4096) return PHX_E_ARG;
  cudaSetDevice(c->device);
  const size_t need = (size_t)P * B * k;
  c->state_fresh = false;
  if (need > c->merge_keys_elems) {
    if (c->merge_keys) cudaFree(c->merge_keys);
    c->merge_keys = nullptr;
    PHX_CUDA_TRY(cudaMalloc(&c->merge_keys, need * 8), c->err);
    c->merge_keys_elems = need;
  }
  merge_keys_kernel<<<(unsigned)((need + 255) / 256), 256, 0, c->stream>>>(scores_dev, (const long long*)ids_dev, P, B, k, c->merge_keys, c->status);
  PHX_CUDA_TRY(cudaGetLastError(), c->err);
  const int kp2 = next_pow2(k);
  select_kernel<<<B, SEL_THREADS, (size_t)sel_room(kp2) * 8, c->stream>>>(c->merge_keys, nullptr, P * k, P * k, k, kp2, out_scores_dev,
                                                               (long long*)out_ids_dev, c->status);
  PHX_CUDA_TRY(cudaGetLastError(), c->err);
  return close_call(c);
}

// ---- merge without any allocation ---------------------------------------------------------------------
// Scratch for phx_topk_merge_static: the 64-bit sort keys of one merge and its status word live in
// device memory that belongs to the loaded library image, not to an allocator.  Every device that
// loads the library carries these 16 MiB until the process exits.
#define PHX_STATIC_MERGE_MAX_KEYS (1 << 21)
static __device__ __align__(256) unsigned long long g_static_merge_keys[PHX_STATIC_MERGE_MAX_KEYS];
static __device__ __align__(256) int g_static_merge_status[64];

namespace {
struct StaticScratch { unsigned long long* keys = nullptr; int* status = nullptr; bool ready = false; };
StaticScratch g_static_scratch[64];  // by device ordinal
std::mutex g_static_mu;

// In host code `g_static_merge_keys` only names the symbol; the address a kernel may use has to be asked
// for, per device, while that device is current.
phx_status static_scratch_for(int device, StaticScratch** out, std::string& err) {
  if (device < 0 || device >= 64) { err = "phx_topk_merge_static: device ordinal out of range"; return PHX_E_ARG; }
  std::lock_guard<std::mutex> lk(g_static_mu);
  StaticScratch& sc = g_static_scratch[device];
  if (!sc.ready) {
    void* pk = nullptr; void* ps = nullptr;
    PHX_CUDA_TRY(cudaGetSymbolAddress(&pk, g_static_merge_keys), err);
    PHX_CUDA_TRY(cudaGetSymbolAddress(&ps, g_static_merge_status), err);
    sc.keys = static_cast<unsigned long long*>(pk);
    sc.status = static_cast<int*>(ps);
    sc.ready = true;
  }
  *out = &sc;
  return PHX_OK;
}
struct DeviceGuard {
  int prev = -1; bool ok = false;
  explicit DeviceGuard(int device) {
    if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
    ok = cudaSetDevice(device) == cudaSuccess;
  }
  ~DeviceGuard() { if (prev >= 0) cudaSetDevice(prev); }
};
}  // namespace

phx_status phx_topk_merge_static_status(int32_t device, void* stream, int32_t* status_out) {
  if (!status_out) { set_global_error("phx_topk_merge_static_status: null argument"); return PHX_E_ARG; }
  DeviceGuard guard(device);
  if (!guard.ok) { set_global_error("phx_topk_merge_static_status: cudaSetDevice failed"); return PHX_E_CUDA; }
  std::string err;
  StaticScratch* sc = nullptr;
  phx_status s = static_scratch_for(device, &sc, err);
  if (s) { set_global_error(err); return s; }
  cudaError_t ce = cudaStreamSynchronize(static_cast<cudaStream_t>(stream));
  int v = 0;
  if (ce == cudaSuccess) ce = cudaMemcpy(&v, sc->status, sizeof(int), cudaMemcpyDeviceToHost);
  if (ce != cudaSuccess) { set_global_error(std::string("phx_topk_merge_static_status: ") + cudaGetErrorString(ce)); return PHX_E_CUDA; }
  *status_out = v;
  return PHX_OK;
}

phx_status phx_topk_merge_static(int32_t device, const float* scores_dev, const int64_t* ids_dev, int32_t P, int32_t B,
                                 int32_t k, float* out_scores_dev, int64_t* out_ids_dev, void* stream) {
  std::string err;
  if (!scores_dev || !ids_dev || !out_scores_dev || !out_ids_dev || P <= 0 || B <= 0 || k <= 0 || k > 4096) {
    set_global_error("phx_topk_merge_static: bad argument (P, B, k > 0, k <= 4096, non-null buffers)");
    return PHX_E_ARG;
  }
  const unsigned long long need = (unsigned long long)P * (unsigned long long)B * (unsigned long long)k;
  if (need > (unsigned long long)PHX_STATIC_MERGE_MAX_KEYS) {
    set_global_error("phx_topk_merge_static: P*B*k = " + std::to_string(need) + " exceeds the built-in scratch of " +
                     std::to_string((long long)PHX_STATIC_MERGE_MAX_KEYS) + " keys; use phx_topk_merge_device");
    return PHX_E_CAPACITY;
  }
  DeviceGuard guard(device);   // the caller's current device is put back on return
  if (!guard.ok) { set_global_error("phx_topk_merge_static: cudaSetDevice failed"); return PHX_E_CUDA; }
  StaticScratch* sc = nullptr;
  phx_status s = static_scratch_for(device, &sc, err);
  if (s) { set_global_error(err); return s; }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // the array keeps the previous call's contents: the status word must start at zero, the keys in
  // [0, need) are all rewritten by the first kernel
  cudaError_t ce = cudaMemsetAsync(sc->status, 0, sizeof(int), st);
  if (ce != cudaSuccess) { set_global_error(std::string("phx_topk_merge_static: ") + cudaGetErrorString(ce)); return PHX_E_CUDA; }
  merge_keys_kernel<<<(unsigned)((need + 255) / 256), 256, 0, st>>>(scores_dev, (const long long*)ids_dev, P, B, k, sc->keys, sc->status);
  const int kp2 = next_pow2(k);
  select_kernel<<<B, SEL_THREADS, (size_t)sel_room(kp2) * 8, st>>>(sc->keys, nullptr, P * k, P * k, k, kp2, out_scores_dev,
                                                         (long long*)out_ids_dev, sc->status);
  ce = cudaGetLastError();
  if (ce != cudaSuccess) { set_global_error(std::string("phx_topk_merge_static: ") + cudaGetErrorString(ce)); return PHX_E_CUDA; }
  return PHX_OK;
}

phx_status phx_corpus_sync(phx_corpus* c) {
  if (!c) return PHX_E_ARG;
  cudaSetDevice(c->device);
  // the last top-k / merge may have been enqueued on a caller's stream that is no longer the current one
  // (phx_corpus_set_stream): wait for the event recorded behind it as well
  PHX_CUDA_TRY(cudaEventSynchronize(c->ev1), c->err);
  PHX_CUDA_TRY(cudaStreamSynchronize(c->stream), c->err);
  int state[3] = {0, 0, 0};
  if (c->state_fresh) memcpy(state, c->state_host, sizeof(state));
  else PHX_CUDA_TRY(cudaMemcpy(state, c->err_flag, sizeof(state), cudaMemcpyDeviceToHost), c->err);
  c->state_fresh = false;
  const int ef = state[0];
  int st = state[2];
  auto wait_ran_out = [&]() {
    cudaMemset(c->err_flag, 0, 4);
    c->err = "topk: a bounded device-side wait ran out (scan pipeline)";
    return PHX_E_TIMEOUT;
  };
  if (ef != 0) return wait_ran_out();
  if (st & 4) {
    cudaMemset(c->status, 0, 4);
    c->err = "topk merge: an id does not fit 32 bits; the entry was left out";
    return PHX_E_ARG;
  }
  if (st != 0 && c->last.valid && !c->exact) {
    // The sampled pivot missed for some query (fewer than k rows, or more than the survivor buffer holds, reached it):
    // the call is done again into the same output buffers before this sync returns, a short list first with a pivot for 3k rows (many
    // rows a few bf16 steps apart, 300 k of them in 1.2 M rows, k = 10: 1512 us a call by the exact passes, 294 so), then with exact
    // thresholds.  The queries must still be where the call read them.
    const phx_corpus::LastCall call = c->last;
    for (int exact = call.sparse ? 0 : 1; exact < 2 && st != 0; ++exact) {
      PHX_CUDA_TRY(cudaMemsetAsync(c->status, 0, 4, c->stream), c->err);
      (exact ? c->exact : c->dense) = true;
      c->keys_out = call.keys;
      const phx_status xs = phx_corpus_topk_window_device(c, call.users, call.B, call.k, call.row_begin, call.row_end, call.scores,
                                                          (int64_t*)call.ids);
      c->keys_out = nullptr;
      c->exact = c->dense = false;
      c->state_fresh = false;
      if (xs) return xs;
      c->reran = 1;
      PHX_CUDA_TRY(cudaEventSynchronize(c->ev1), c->err);      // behind the re-run's last kernel and its state (close_call)
      if (c->state_host[0]) return wait_ran_out();
      st = c->state_host[2];
    }
  }
  if (st != 0) {
    cudaMemset(c->status, 0, 4);
    c->err = std::string("topk: survivor list ") + ((st & 2) ? "overflowed its capacity" : "held fewer than k rows") +
             " (pivot estimate off for this corpus); result withheld";
    return PHX_E_CAPACITY;
  }
  return PHX_OK;
}

phx_status phx_corpus_finish(phx_corpus* c, int32_t* reran_out) {
  if (!c) return PHX_E_ARG;
  c->reran = 0;
  const phx_status s = phx_corpus_sync(c);
  if (reran_out) *reran_out = c->reran;
  return s;
}

phx_status phx_corpus_set_exact(phx_corpus* c, int32_t on) {
  if (!c) return PHX_E_ARG;
  c->exact = on != 0;
  return PHX_OK;
}

phx_status phx_corpus_exact_runs(phx_corpus* c, int64_t* n) {
  if (!c || !n) return PHX_E_ARG;
  *n = c->exact_runs;
  return PHX_OK;
}

phx_status phx_corpus_last_device_ms(phx_corpus* c, float* ms) {
  if (!c || !ms) return PHX_E_ARG;
  PHX_CUDA_TRY(cudaEventSynchronize(c->ev1), c->err);
  PHX_CUDA_TRY(cudaEventElapsedTime(ms, c->ev0, c->ev1), c->err);
  return PHX_OK;
}

}  // extern "C"
