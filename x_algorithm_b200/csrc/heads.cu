// Final RMSNorm of the candidate rows, the action and continuous heads, the server's log-sigmoid
// and the value-model blend in one pass (phoenix/xrex/models/recsys_model.py:4792-4843, 3557-3560,
// 3756-3846, 712-733; phoenix/xrex/inference/model_runner.py:4474; xai-value-model/scoring.rs:67-73,
// 112-120, 282-291).  One warp per candidate row; the (V+NC) x D head matrix sits in shared memory.
// Also the user-tower pooling (recsys_two_tower_model.py:2187-2200).
#include <stdlib.h>
#include <string.h>

#include "common.cuh"

namespace phx {
namespace {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

constexpr int MAX_OUT = 32;  // V + NC
constexpr size_t POOL_SMEM = 72 * 1024;   // three CTAs of the pooling kernel an SM

__global__ void __launch_bounds__(256) heads_kernel(HeadsArgs a) {
  extern __shared__ __align__(16) uint8_t hsm[];
  bf16* sw = reinterpret_cast<bf16*>(hsm);  // [(V+NC), D]
  const int NO = a.V + a.NC;
  for (int i = threadIdx.x * 8; i < NO * a.D; i += blockDim.x * 8)
    *reinterpret_cast<uint4*>(sw + i) = *reinterpret_cast<const uint4*>(a.unembed_t + i);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const long long nrows = a.out_index ? a.rows : (long long)a.B * a.C;
  for (long long r = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < nrows;
       r += (long long)gridDim.x * (blockDim.x >> 5)) {
    const int b = (int)(r / a.C), c = (int)(r % a.C);
    // packed rows: candidate rows back to back, each answering the output slot out_index[r]
    const bf16* xr = a.out_index ? a.x + r * a.D : a.x + ((long long)b * a.T + a.S + c) * a.D;
    const long long orow = a.out_index ? a.out_index[r] : r;
    float ss = 0.f;
    for (int k = lane * 8; k < a.D; k += 256) {
      uint4 u = *reinterpret_cast<const uint4*>(xr + k);
      float2 p0 = unpack_bf2(u.x), p1 = unpack_bf2(u.y), p2 = unpack_bf2(u.z), p3 = unpack_bf2(u.w);
      ss += p0.x * p0.x + p0.y * p0.y + p1.x * p1.x + p1.y * p1.y + p2.x * p2.x + p2.y * p2.y + p3.x * p3.x + p3.y * p3.y;
    }
    ss = warp_sum(ss);
    const float rstd = rsqrtf(ss / (float)a.D + a.eps);
    float acc[MAX_OUT];
#pragma unroll
    for (int j = 0; j < MAX_OUT; ++j) acc[j] = 0.f;
    for (int k = lane * 8; k < a.D; k += 256) {
      uint4 u = *reinterpret_cast<const uint4*>(xr + k);
      float xv[8];
      float2 p0 = unpack_bf2(u.x), p1 = unpack_bf2(u.y), p2 = unpack_bf2(u.z), p3 = unpack_bf2(u.w);
      xv[0] = p0.x; xv[1] = p0.y; xv[2] = p1.x; xv[3] = p1.y; xv[4] = p2.x; xv[5] = p2.y; xv[6] = p3.x; xv[7] = p3.y;
#pragma unroll
      for (int i = 0; i < 8; ++i) xv[i] = round_bf(xv[i] * rstd * a.final_gain[k + i]);  // normed row is bf16
#pragma unroll
      for (int j = 0; j < MAX_OUT; ++j) {
        if (j < NO) {
          uint4 w = *reinterpret_cast<const uint4*>(sw + j * a.D + k);
          float2 w0 = unpack_bf2(w.x), w1 = unpack_bf2(w.y), w2 = unpack_bf2(w.z), w3 = unpack_bf2(w.w);
          acc[j] += xv[0] * w0.x + xv[1] * w0.y + xv[2] * w1.x + xv[3] * w1.y + xv[4] * w2.x + xv[5] * w2.y + xv[6] * w3.x + xv[7] * w3.y;
        }
      }
    }
    // butterfly: 31 shuffles leave the total of output j on lane j (instead of 5 shuffles per output)
#pragma unroll
    for (int step = 16; step >= 1; step >>= 1) {
      const bool upper = (lane & step) != 0;
#pragma unroll
      for (int i = 0; i < step; ++i) {
        const float send = upper ? acc[i] : acc[i + step];
        const float keep = upper ? acc[i + step] : acc[i];
        acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, step);
      }
    }
    const float mine = acc[0];
    float value = 0.f;  // probability (f32 log-prob kept separately) or continuous prediction
    float logp = 0.f;
    if (lane < a.V) {
      float lg = round_bf(round_bf(mine) * a.output_scale);
      if (a.final_logit_cap > 0.f) lg = round_bf(a.final_logit_cap * tanhf(lg / a.final_logit_cap));
      logp = fminf(lg, 0.f) - log1pf(expf(-fabsf(lg)));  // log_sigmoid in fp32
      if (a.log_probs) a.log_probs[orow * a.V + lane] = logp;
    } else if (lane < NO) {
      float cl = round_bf(mine);
      float sg = round_bf(1.0f / (1.0f + expf(-cl)));
      value = round_bf(sg * a.dwell_norm_scale);
      if (a.continuous) a.continuous[orow * a.NC + (lane - a.V)] = value;
    }
    if (a.has_blend && a.scores) {
      // exp(ln p as f32 -> f64) like the client side; terms summed left to right in f64 by lane 0
      double col = (lane < a.V) ? exp((double)logp) : (double)value;
      double s = 0.0;
      for (int i = 0; i < a.blend.num_terms; ++i) {
        const int src = a.blend.src[i];
        double cv = __shfl_sync(0xffffffffu, col, src);
        s = s + cv * a.blend.weight[i];
      }
      if (lane == 0) {
        double out;
        if (a.blend.total_sum == 0.0) out = s > 0.0 ? s : 0.0;
        else if (s < 0.0) out = (s + a.blend.negative_sum) / a.blend.total_sum * 0.001;
        else out = s + 0.001;
        a.scores[orow] = out;
      }
    }
  }
}


// ---- tensor-core variant (D a multiple of 32) -----------------------------------------------------------------------
// A strip = 16 candidate rows.  The head matrix product runs on mma.sync m16n8k16: within every group of 32 columns
// the k index is permuted so that a thread's A fragments for two k-steps are one 16-byte load of its row (columns
// 8*t4 .. 8*t4+7 of the group) and its B fragments one 16-byte read of the head matrix row in shared memory.  Rows are
// normalised exactly like the scalar kernel (x * rstd * gain rounded to bf16) on their way into the fragments; the
// sums of squares come from a first pass over the same rows.  The per-output transcendental work is spread over all
// lanes ((row, output) items), the f64 blend runs one row per lane in the spec's term order.
constexpr int HM_WARPS = 8;
constexpr int HM_WPAD = 32;   // elements of padding per head-matrix row: rows g and g+1 fall into different bank halves

__device__ __forceinline__ void mma_bf16_16816_h(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Row r of the call: candidate r % C of request r / C, or (packed) the r-th candidate row.  Rows fit 31 bits.
__device__ __forceinline__ const bf16* head_row(const HeadsArgs& a, long long r, long long nrows) {
  if (r >= nrows) r = nrows - 1;
  if (a.out_index) return a.x + r * (long long)a.D;
  const unsigned b = (unsigned)r / (unsigned)a.C, c = (unsigned)r - b * (unsigned)a.C;
  return a.x + ((long long)b * a.T + a.S + c) * (long long)a.D;
}
// One (row, output) pair: the result, and its value for the blend.
__device__ __forceinline__ double head_item(const HeadsArgs& a, float mine, long long r, long long nrows, int oo) {
  const long long orow = (a.out_index && r < nrows) ? a.out_index[r] : r;   // packed rows: the output slot this row answers
  if (oo < a.V) {
    float lg = round_bf(round_bf(mine) * a.output_scale);
    if (a.final_logit_cap > 0.f) lg = round_bf(a.final_logit_cap * tanhf(lg / a.final_logit_cap));
    const float logp = fminf(lg, 0.f) - log1pf(expf(-fabsf(lg)));  // log_sigmoid in fp32
    if (a.log_probs && r < nrows) a.log_probs[orow * a.V + oo] = logp;
    return a.has_blend ? exp((double)logp) : 0.0;   // exp(ln p as f32 -> f64) like the client side
  }
  const float cl = round_bf(mine);
  const float sg = round_bf(1.0f / (1.0f + expf(-cl)));
  const float value = round_bf(sg * a.dwell_norm_scale);
  if (a.continuous && r < nrows) a.continuous[orow * a.NC + (oo - a.V)] = value;
  return (double)value;
}
__device__ __forceinline__ void head_blend(const HeadsArgs& a, const double* cols, long long r) {
  double s = 0.0;   // terms summed left to right in f64
#pragma unroll 4
  for (int i = 0; i < a.blend.num_terms; ++i) s = s + cols[a.blend.src[i]] * a.blend.weight[i];
  double out;
  if (a.blend.total_sum == 0.0) out = s > 0.0 ? s : 0.0;
  else if (s < 0.0) out = (s + a.blend.negative_sum) / a.blend.total_sum * 0.001;
  else out = s + 0.001;
  a.scores[a.out_index ? a.out_index[r] : r] = out;
}
__device__ __forceinline__ float square_sum(uint4 u) {
  const float2 p0 = unpack_bf2(u.x), p1 = unpack_bf2(u.y), p2 = unpack_bf2(u.z), p3 = unpack_bf2(u.w);
  return (p0.x * p0.x + p0.y * p0.y) + (p1.x * p1.x + p1.y * p1.y) + (p2.x * p2.x + p2.y * p2.y) + (p3.x * p3.x + p3.y * p3.y);
}
// the head matrix and the norm's gain, staged while the last GEMM of the trunk drains
template <int NT>
__device__ __forceinline__ void stage_parameters(const HeadsArgs& a, bf16* sw, float* sgain) {
  const int D = a.D, NO = a.V + a.NC, WLD = D + HM_WPAD;
#pragma unroll 4
  for (int i = threadIdx.x; i < NT * 8 * (D / 8); i += blockDim.x) {
    const int n = i / (D / 8), ch = i % (D / 8);
    uint4 w = make_uint4(0u, 0u, 0u, 0u);
    if (n < NO) w = *reinterpret_cast<const uint4*>(a.unembed_t + (long long)n * D + ch * 8);
    *reinterpret_cast<uint4*>(sw + n * WLD + ch * 8) = w;
  }
  for (int i = threadIdx.x; i < D; i += blockDim.x) sgain[i] = a.final_gain[i];
}

// NT: n-tiles of 8 outputs, V + NC <= 8 * NT.  A strip of 16 rows is a chain of latencies - a round trip to its rows, sums of squares in a
// fixed order, products, logarithms and f64 exponentials, the blend.  In a small call sixteen warps take it together: the rows arrive in
// shared memory by one round of copies, two warps form the sums of squares (a quad a row), all of them normalise, a warp per n-tile
// multiplies, and every (row, output) pair has a thread.  Where eight warps each went through the whole strip, 512 rows of 512 columns with 20
// outputs took 2.1 us for the rows, 1.2 + 2.6 for sums and products, 1.1 and 0.7 for the rest.
constexpr int HS_WARPS = 16;
template <int NT>
__global__ void __launch_bounds__(HS_WARPS * 32, 3) heads_strip_kernel(HeadsArgs a) {
  extern __shared__ __align__(16) uint8_t hsm[];
  const int D = a.D, NO = a.V + a.NC, WLD = D + HM_WPAD, per_row = D / 8, groups = D / 32;
  bf16* sw = reinterpret_cast<bf16*>(hsm);                                   // [NT*8][WLD], rows >= NO are zero
  float* sgain = reinterpret_cast<float*>(sw + NT * 8 * WLD);                // [D]
  float* sC = sgain + D;                                                     // [16][NT*8] fp32 sums
  double* sD = reinterpret_cast<double*>(sC + 16 * NT * 8);                  // [16][NT*8] blend inputs
  float* srstd = reinterpret_cast<float*>(sD + 16 * NT * 8);                 // [16]
  bf16* sX = reinterpret_cast<bf16*>(srstd + 16);                            // [16][WLD] the strip's rows, normalised in place
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const long long nrows = a.out_index ? a.rows : (long long)a.B * a.C, r0 = (long long)blockIdx.x * 16;
  stage_parameters<NT>(a, sw, sgain);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  for (int i = threadIdx.x; i < 16 * per_row; i += HS_WARPS * 32) {
    const int rr = i / per_row, ch = i - rr * per_row;
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(sX + rr * WLD + ch * 8);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(head_row(a, r0 + rr, nrows) + ch * 8) : "memory");
  }
  asm volatile("cp.async.commit_group;\n cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  if (warp < 2) {    // sums of squares: a row's 32-column groups are spread over the 4 lanes of its quad
    const bf16* xr = sX + (warp * 8 + g) * WLD + 8 * t4;
    float ss = 0.f;
#pragma unroll 8
    for (int gr = 0; gr < groups; ++gr) ss += square_sum(*reinterpret_cast<const uint4*>(xr + gr * 32));
    ss += __shfl_xor_sync(0xffffffffu, ss, 1);
    ss += __shfl_xor_sync(0xffffffffu, ss, 2);
    if (t4 == 0) srstd[warp * 8 + g] = rsqrtf(ss / (float)D + a.eps);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 16 * per_row; i += HS_WARPS * 32) {   // the normed row is bf16
    const int rr = i / per_row, ch = i - rr * per_row;
    uint4* const at = reinterpret_cast<uint4*>(sX + rr * WLD + ch * 8);
    const float4 ga = *reinterpret_cast<const float4*>(sgain + ch * 8), gb = *reinterpret_cast<const float4*>(sgain + ch * 8 + 4);
    const float rstd = srstd[rr];
    const uint4 u = *at;
    const float2 p0 = unpack_bf2(u.x), p1 = unpack_bf2(u.y), p2 = unpack_bf2(u.z), p3 = unpack_bf2(u.w);
    *at = make_uint4(pack_bf2(p0.x * rstd * ga.x, p0.y * rstd * ga.y), pack_bf2(p1.x * rstd * ga.z, p1.y * rstd * ga.w),
                     pack_bf2(p2.x * rstd * gb.x, p2.y * rstd * gb.y), pack_bf2(p3.x * rstd * gb.z, p3.y * rstd * gb.w));
  }
  __syncthreads();
  if (warp < NT) {
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int gr = 0; gr < groups; ++gr) {
      // k-step 0 uses pairs 0, 1 of each row's 8 columns, k-step 1 pairs 2, 3: fragment order [g][lo], [g+8][lo], [g][hi], [g+8][hi]
      const uint4 lo = *reinterpret_cast<const uint4*>(sX + g * WLD + gr * 32 + 8 * t4), hi = *reinterpret_cast<const uint4*>(sX + (g + 8) * WLD + gr * 32 + 8 * t4);
      const uint4 w = *reinterpret_cast<const uint4*>(sw + (warp * 8 + g) * WLD + gr * 32 + 8 * t4);
      const uint32_t a0[4] = {lo.x, hi.x, lo.y, hi.y}, a1[4] = {lo.z, hi.z, lo.w, hi.w};
      mma_bf16_16816_h(acc, a0, w.x, w.y);
      mma_bf16_16816_h(acc, a1, w.z, w.w);
    }
    *reinterpret_cast<float2*>(sC + g * (NT * 8) + warp * 8 + 2 * t4) = make_float2(acc[0], acc[1]);
    *reinterpret_cast<float2*>(sC + (g + 8) * (NT * 8) + warp * 8 + 2 * t4) = make_float2(acc[2], acc[3]);
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < 16 * NO; idx += HS_WARPS * 32) {
    const int rr = idx / NO, oo = idx - rr * NO;
    sD[rr * (NT * 8) + oo] = head_item(a, sC[rr * (NT * 8) + oo], r0 + rr, nrows, oo);
  }
  __syncthreads();
  if (a.has_blend && a.scores && threadIdx.x < 16 && r0 + threadIdx.x < nrows) head_blend(a, sD + threadIdx.x * (NT * 8), r0 + threadIdx.x);
}

// Many strips: every warp has its own (WPS = 1) and reads its rows where they are, once for the sums of squares, once for the products; the
// same arithmetic, the same bits.  Four warps share one in small calls of rows too wide to stand beside the head matrix in shared memory.
template <int NT, int WPS>
__global__ void __launch_bounds__((WPS == 1 ? HM_WARPS : WPS) * 32) heads_mma_kernel(HeadsArgs a) {
  constexpr int WARPS = WPS == 1 ? HM_WARPS : WPS;      // warps per CTA
  extern __shared__ __align__(16) uint8_t hsm[];
  const int D = a.D, NO = a.V + a.NC, WLD = D + HM_WPAD;
  bf16* sw = reinterpret_cast<bf16*>(hsm);                                   // [NT*8][WLD], rows >= NO are zero
  float* sgain = reinterpret_cast<float*>(sw + NT * 8 * WLD);                // [D]
  float* sC_all = sgain + D;                                                 // per warp [16][NT*8] fp32 sums
  double* sD_all = reinterpret_cast<double*>(sC_all + WARPS * 16 * NT * 8);   // per strip [16][NT*8] blend inputs
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  stage_parameters<NT>(a, sw, sgain);
  // programmatic dependent launch: the parameters above are staged while the last GEMM of the trunk drains; its
  // output is read only from here on
  asm volatile("griddepcontrol.wait;" ::: "memory");
  __syncthreads();
  float* sC = sC_all + warp * 16 * NT * 8;
  double* sD = sD_all + (WPS == 1 ? warp : 0) * 16 * NT * 8;
  const int part = WPS == 1 ? 0 : warp;                 // this warp's share of the strip's items
  const long long nrows = a.out_index ? a.rows : (long long)a.B * a.C;
  const long long n_strips = (nrows + 15) / 16;
  const int groups = D / 32;
  constexpr int CTA_STRIPS = WPS == 1 ? HM_WARPS : 1;
  for (long long strip = (long long)blockIdx.x * CTA_STRIPS + (WPS == 1 ? warp : 0); strip < n_strips; strip += (long long)gridDim.x * CTA_STRIPS) {
    const long long r0 = strip * 16;
    const bf16* xr[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) xr[i] = head_row(a, r0 + g + 8 * i, nrows) + 8 * t4;
    // pass 1: sums of squares (a row's 32-column groups are spread over the 4 lanes of its quad)
    float ss[2] = {0.f, 0.f};
#pragma unroll 8
    for (int gr = 0; gr < groups; ++gr) {
#pragma unroll
      for (int i = 0; i < 2; ++i) ss[i] += square_sum(*reinterpret_cast<const uint4*>(xr[i] + gr * 32));
    }
    float rstd[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], 1);
      ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], 2);
      rstd[i] = rsqrtf(ss[i] / (float)D + a.eps);
    }
    // pass 2: normalise into A fragments, multiply
    float acc[NT][4];
#pragma unroll
    for (int j = 0; j < NT; ++j) { acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f; }
#pragma unroll 4
    for (int gr = 0; gr < groups; ++gr) {
      const float4 ga = *reinterpret_cast<const float4*>(sgain + gr * 32 + 8 * t4);
      const float4 gb = *reinterpret_cast<const float4*>(sgain + gr * 32 + 8 * t4 + 4);
      uint32_t fr[2][4];   // per row: the four packed pairs of its 8 normalised columns
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const uint4 u = *reinterpret_cast<const uint4*>(xr[i] + gr * 32);
        const float2 p0 = unpack_bf2(u.x), p1 = unpack_bf2(u.y), p2 = unpack_bf2(u.z), p3 = unpack_bf2(u.w);
        fr[i][0] = pack_bf2(p0.x * rstd[i] * ga.x, p0.y * rstd[i] * ga.y);   // the normed row is bf16
        fr[i][1] = pack_bf2(p1.x * rstd[i] * ga.z, p1.y * rstd[i] * ga.w);
        fr[i][2] = pack_bf2(p2.x * rstd[i] * gb.x, p2.y * rstd[i] * gb.y);
        fr[i][3] = pack_bf2(p3.x * rstd[i] * gb.z, p3.y * rstd[i] * gb.w);
      }
      // k-step 0 uses pairs 0, 1 of each row, k-step 1 pairs 2, 3: fragment order [g][lo], [g+8][lo], [g][hi], [g+8][hi]
      const uint32_t a0[4] = {fr[0][0], fr[1][0], fr[0][1], fr[1][1]};
      const uint32_t a1[4] = {fr[0][2], fr[1][2], fr[0][3], fr[1][3]};
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        const uint4 w = *reinterpret_cast<const uint4*>(sw + (j * 8 + g) * WLD + gr * 32 + 8 * t4);
        mma_bf16_16816_h(acc[j], a0, w.x, w.y);
        mma_bf16_16816_h(acc[j], a1, w.z, w.w);
      }
    }
    // the strip's 16 x (8 NT) sums to shared memory
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      *reinterpret_cast<float2*>(sC + g * (NT * 8) + j * 8 + 2 * t4) = make_float2(acc[j][0], acc[j][1]);
      *reinterpret_cast<float2*>(sC + (g + 8) * (NT * 8) + j * 8 + 2 * t4) = make_float2(acc[j][2], acc[j][3]);
    }
    __syncwarp();
    for (int idx = lane + 32 * part; idx < 16 * NO; idx += 32 * WPS) {
      const int rr = idx / NO, oo = idx % NO;
      sD[rr * (NT * 8) + oo] = head_item(a, sC[rr * (NT * 8) + oo], r0 + rr, nrows, oo);
    }
    if (WPS == 1) __syncwarp(); else __syncthreads();
    if (a.has_blend && a.scores && part == 0 && lane < 16 && r0 + lane < nrows) head_blend(a, sD + lane * (NT * 8), r0 + lane);
    if (WPS == 1) __syncwarp(); else __syncthreads();
  }
}

constexpr size_t HEADS_SMEM_MAX = 200 * 1024;
// Launched programmatically: the kernel stages its parameters while the one in front drains, and waits before it reads the residual stream.
template <typename Kernel>
phx_status launch_heads(Kernel kern, SmemLimit& limit, const HeadsArgs& a, long long blocks, int threads, size_t smem, cudaStream_t stream, std::string& err) {
  if (smem > HEADS_SMEM_MAX) { err = "heads: head matrix does not fit shared memory"; return PHX_E_CAPACITY; }
  PHX_CUDA_TRY(limit.raise(kern, (int)HEADS_SMEM_MAX), err);
  PHX_CUDA_TRY(launch_programmatic(kern, dim3((unsigned)blocks), dim3(threads), smem, stream, a), err);
  return PHX_OK;
}
template <int NT>
phx_status launch_heads_mma(const HeadsArgs& a, long long rows, cudaStream_t stream, std::string& err) {
  const long long strips = (rows + 15) / 16;
  const size_t params = (size_t)NT * 8 * (a.D + HM_WPAD) * sizeof(bf16) + (size_t)a.D * sizeof(float);
  const size_t strip_smem = params + (size_t)16 * NT * 8 * (sizeof(float) + sizeof(double)) + 64 + (size_t)16 * (a.D + HM_WPAD) * sizeof(bf16);
  // Three CTAs of a strip each fit an SM's registers, of wide rows two or one its shared memory, so that the line below is one to three rounds of
  // them: each round takes less than a warp a strip, or four, take with all strips at once.  Kernel, us, sixteen warps / four / one, at 148, 296 and
  // 444 strips: D = 512, 20 outputs 12.6 / 18.9 / 20.9, 12.7 / 22.9 / 22.9, 14.8 / 23.0 / 22.9; D = 1024, 30 outputs 16.9 / 39.3 / 39.4, 18.9 / 39.4 / 39.4, 29.2 / 63.9 /
  // 39.4; D = 1280, 20 outputs 18.9 / 39.4 / 37.3, 20.9 / 39.4 / 39.3, 33.2 / 66.0 / 41.4; D = 1280, 30 outputs (one CTA an SM from here on) 20.9 / 45.5 /
  // 45.5, 29.1 / 47.6 / 45.5, 39.4 / 78.2 / 49.6; D = 1536 18.9 / 45.5 / 41.4, 29.1 / 47.6 / 41.4, 39.4 / 80.3 / 45.5; D = 2048 23.0 / 49.6 / 49.6, 37.3 / 90.4 /
  // 55.7, 51.7 / 131.6 / 57.8.  Beyond the line one warp a strip: D = 512, 20 outputs, sixteen / one: 768 strips 22.8 / 22.9, 2048 45.4 / 27.0, 8192 164 / 92.
  static SmemLimit limit16, limit4, limit1;
  const int sms = device_sms();
  if (strips <= 3LL * sms && strip_smem <= HEADS_SMEM_MAX)
    return launch_heads(heads_strip_kernel<NT>, limit16, a, strips, HS_WARPS * 32, strip_smem, stream, err);
  if (strips <= 2LL * sms)
    return launch_heads(heads_mma_kernel<NT, 4>, limit4, a, strips, 4 * 32, params + (size_t)16 * NT * 8 * (4 * sizeof(float) + sizeof(double)), stream, err);
  const long long blocks = (strips + HM_WARPS - 1) / HM_WARPS;
  return launch_heads(heads_mma_kernel<NT, 1>, limit1, a, blocks < 3LL * sms ? blocks : 3LL * sms, HM_WARPS * 32,
                      params + (size_t)16 * NT * 8 * HM_WARPS * (sizeof(float) + sizeof(double)), stream, err);
}

// users[b] = l2norm(mean over valid t of final_norm(x[b,t])), fp32; one CTA per user, one thread per column.  Two passes
// over the user's rows (row statistics, then the mean): a chain of latencies, so the rows are fetched once, all loads in
// flight together, and kept in shared memory (STAGED) where they fit beside those of two more CTAs.
// 128 rows of 256 columns: one user 20.0 -> 11.8 us, 256 users 24.3 -> 17.1.
template <bool F32, bool STAGED>   // F32: fp32 rows, nothing rounded (the full-precision path)
__global__ void tower_pool_kernel(const void* __restrict__ xv, const float* __restrict__ gain, const int* __restrict__ seg,
                                  int T, int D, float eps, float* __restrict__ users) {
  extern __shared__ __align__(16) float psm[];  // STAGED: [T][D] rows; [T] rstd (0 for invalid) + reduction scratch
  const int b = blockIdx.x;
  const char* rows = reinterpret_cast<const char*>(xv) + (long long)b * T * D * (F32 ? 4 : 2);
  float* rstd = psm;
  if (STAGED) {
    const int n = T * D * (F32 ? 4 : 2) / 16;    // 16-byte units
    rstd = psm + n * 4;
#pragma unroll 8
    for (int i = threadIdx.x; i < n; i += blockDim.x) reinterpret_cast<uint4*>(psm)[i] = reinterpret_cast<const uint4*>(rows)[i];
    rows = reinterpret_cast<const char*>(psm);
    __syncthreads();
  }
  auto ld = [&](long long i) { return F32 ? reinterpret_cast<const float*>(rows)[i] : bf2f(reinterpret_cast<const bf16*>(rows)[i]); };
  float* red = rstd + T;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  // Both passes keep several rows' loads in flight; the order of every sum is that of one row after the other
  constexpr int RU = 4;
  for (int t0 = warp * RU; t0 < T; t0 += nw * RU) {
    float ss[RU] = {0.f, 0.f, 0.f, 0.f};
    int ok[RU];
#pragma unroll
    for (int i = 0; i < RU; ++i) ok[i] = t0 + i < T ? seg[(long long)b * T + t0 + i] : 0;
    const long long r0 = (long long)t0 * D;
#pragma unroll 4
    for (int k = lane; k < D; k += 32) {
#pragma unroll
      for (int i = 0; i < RU; ++i) {
        const float v = t0 + i < T ? ld(r0 + (long long)i * D + k) : 0.f;
        ss[i] += v * v;
      }
    }
#pragma unroll
    for (int i = 0; i < RU; ++i) {
      const float s = warp_sum(ss[i]);
      if (lane == 0 && t0 + i < T) rstd[t0 + i] = ok[i] != 0 ? (F32 ? 1.0f / sqrtf(s / (float)D + eps) : rsqrtf(s / (float)D + eps)) : 0.f;
    }
  }
  __syncthreads();
  float cnt = 0.f;     // whole numbers: exact in any order
  for (int t = lane; t < T; t += 32) cnt += (rstd[t] != 0.f) ? 1.f : 0.f;
  cnt = warp_sum(cnt);
  float sq = 0.f;
  float vals[8];  // D <= 8 * blockDim.x
  int nv = 0;
  for (int k = threadIdx.x; k < D; k += blockDim.x, ++nv) {
    float acc = 0.f;
    const float gk = gain[k];
    constexpr int TU = 16;
    for (int t0 = 0; t0 < T; t0 += TU) {  // fixed order over positions
      float x[TU];
#pragma unroll
      for (int i = 0; i < TU; ++i) x[i] = t0 + i < T ? ld((long long)(t0 + i) * D + k) : 0.f;
#pragma unroll
      for (int i = 0; i < TU; ++i) {
        const float rs = t0 + i < T ? rstd[t0 + i] : 0.f;
        const float v = x[i] * rs * gk;
        if (rs != 0.f) acc = acc + (F32 ? v : round_bf(v));
      }
    }
    const float rep = acc / fmaxf(cnt, 1.0f);
    vals[nv] = rep;
    sq += rep * rep;
  }
  sq = warp_sum(sq);
  if (lane == 0) red[warp] = sq;
  __syncthreads();
  float tot = 0.f;
  for (int w = 0; w < nw; ++w) tot += red[w];
  const float inv = 1.0f / sqrtf(fmaxf(tot, 1e-12f));
  nv = 0;
  for (int k = threadIdx.x; k < D; k += blockDim.x, ++nv) users[(long long)b * D + k] = vals[nv] * inv;
}

}  // namespace

phx_status heads_launch(const HeadsArgs& a, cudaStream_t stream, std::string& err) {
  const int NO = a.V + a.NC;
  if (NO > MAX_OUT || a.D % 8 != 0) { err = "heads: V + NC must be <= 32 and D a multiple of 8"; return PHX_E_ARG; }
  if (a.has_blend) {
    for (int i = 0; i < a.blend.num_terms; ++i)
      if (a.blend.src[i] < 0 || a.blend.src[i] >= NO) { err = "heads: blend term source out of range"; return PHX_E_ARG; }
  }
  const long long rows = a.out_index ? a.rows : (long long)a.B * a.C;
  if (rows == 0) return PHX_OK;
  if (a.D % 32 == 0 && !(getenv("PHX_HEADS") && strcmp(getenv("PHX_HEADS"), "scalar") == 0)) {   // tensor-core path
    if (NO <= 8) return launch_heads_mma<1>(a, rows, stream, err);
    if (NO <= 16) return launch_heads_mma<2>(a, rows, stream, err);
    if (NO <= 24) return launch_heads_mma<3>(a, rows, stream, err);
    return launch_heads_mma<4>(a, rows, stream, err);
  }
  const size_t smem = (size_t)NO * a.D * sizeof(bf16);
  static SmemLimit limit;
  if (smem > 48 * 1024) PHX_CUDA_TRY(limit.raise(heads_kernel, 200 * 1024), err);
  if (smem > 200 * 1024) { err = "heads: head matrix does not fit shared memory"; return PHX_E_CAPACITY; }
  long long blocks = (rows + 7) / 8;
  if (blocks > 148 * 4) blocks = 148 * 4;
  heads_kernel<<<(unsigned)blocks, 256, smem, stream>>>(a);
  PHX_CUDA_TRY(cudaGetLastError(), err);
  return PHX_OK;
}

phx_status tower_pool_launch(const void* x, const float* final_gain, const int* seg, int B, int T, int D, float eps,
                             float* users, cudaStream_t stream, std::string& err, bool x_is_f32) {
  if (B == 0) return PHX_OK;
  int threads = 256;
  if (D > 8 * threads) { err = "tower_pool: D too large"; return PHX_E_CAPACITY; }
  const size_t small = (size_t)(T + 32) * sizeof(float), rows = (size_t)T * D * (x_is_f32 ? 4 : 2);
  const bool staged = rows % 16 == 0 && small + rows <= POOL_SMEM;
  const size_t smem = small + (staged ? rows : 0);
  static SmemLimit limit_bf16, limit_f32;
  if (staged && x_is_f32) {
    PHX_CUDA_TRY(limit_f32.raise(tower_pool_kernel<true, true>, (int)POOL_SMEM), err);
    tower_pool_kernel<true, true><<<B, threads, smem, stream>>>(x, final_gain, seg, T, D, eps, users);
  } else if (staged) {
    PHX_CUDA_TRY(limit_bf16.raise(tower_pool_kernel<false, true>, (int)POOL_SMEM), err);
    tower_pool_kernel<false, true><<<B, threads, smem, stream>>>(x, final_gain, seg, T, D, eps, users);
  } else if (x_is_f32) {
    tower_pool_kernel<true, false><<<B, threads, smem, stream>>>(x, final_gain, seg, T, D, eps, users);
  } else {
    tower_pool_kernel<false, false><<<B, threads, smem, stream>>>(x, final_gain, seg, T, D, eps, users);
  }
  PHX_CUDA_TRY(cudaGetLastError(), err);
  return PHX_OK;
}

}  // namespace phx
