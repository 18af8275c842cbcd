// Multi-hash id -> unified-table row (phoenix/xrex/models/recsys_embedding.py:154-172, 282-331),
// row gather (xai-recsys-engine/src/emb_table.rs:124-140) and the fixed-order fp32 combine of the
// gathered rows into one token.  HBM-bound: one warp per token, 16-byte loads per lane, rows of one
// token read back to back and summed in slot order so the result does not depend on the launch shape.
#include "common.cuh"

namespace phx {
namespace {

// n mod d for any unsigned 64-bit n, with magic = floor((2^64 - 1) / d): the quotient estimate mulhi(n, magic)
// is at most 2 short, so two conditional subtractions finish the job.  (A 64-bit '%' by a run-time value costs
// ~100 instructions; this path made the gather instruction-bound.)
__device__ __forceinline__ unsigned long long umod_magic(unsigned long long n, unsigned long long d, unsigned long long magic) {
  unsigned long long r = n - __umul64hi(n, magic) * d;
  if (r >= d) r -= d;
  if (r >= d) r -= d;
  return r;
}
// raw = (id*scale + bias) mod M, floored (non-negative); idx = 0 if id == 0 else raw mod (buckets-1) + 1
__device__ __forceinline__ int hash_one(long long id, long long scale, long long bias, const HashFamilyDev& f) {
  if (id == 0) return 0;
  // wrapping int64 arithmetic, as numba / Rust release builds do
  const long long raw = (long long)((unsigned long long)id * (unsigned long long)scale + (unsigned long long)bias);
  const unsigned long long m = (unsigned long long)f.modulus;
  unsigned long long r;
  if (raw >= 0) r = umod_magic((unsigned long long)raw, m, f.magic_mod);
  else r = m - 1 - umod_magic((unsigned long long)(~raw), m, f.magic_mod);   // floored: -(x+1) mod m = m-1-(x mod m)
  return (int)umod_magic(r, (unsigned long long)f.buckets_m1, f.magic_bkt) + 1 + f.offset;
}

__device__ __forceinline__ void acc_row(float (&acc)[8], const bf16* row, int col) {
  uint4 u = __ldg(reinterpret_cast<const uint4*>(row + col));
  float2 a = unpack_bf2(u.x), b = unpack_bf2(u.y), c = unpack_bf2(u.z), d = unpack_bf2(u.w);
  acc[0] += a.x; acc[1] += a.y; acc[2] += b.x; acc[3] += b.y;
  acc[4] += c.x; acc[5] += c.y; acc[6] += d.x; acc[7] += d.y;
}

// The action row of a history token, columns col..col+7, as packed bf16.  Single action: row `act` of the table.
// Action set (multi_hot_to_embeddings, recsys_model.py:3282-3312): the [D] vector, the chunk these columns lie in
// signed by 2 a_v - 1 (a sign-bit flip: exact), everything zero when the set is empty.
__device__ __forceinline__ uint4 action_chunk(const TokenBuildArgs& a, int act, int col, bool action_set) {
  if (!action_set) return __ldg(reinterpret_cast<const uint4*>(a.action_table + (long long)act * a.D + col));
  const unsigned live = (a.num_action_types >= 32) ? 0xffffffffu : ((1u << a.num_action_types) - 1u);
  const unsigned bits = (unsigned)act & live;
  if (bits == 0u) return make_uint4(0u, 0u, 0u, 0u);
  uint4 u = __ldg(reinterpret_cast<const uint4*>(a.action_table + col));
  const int v = col / (a.D / a.num_action_types);
  if (!((bits >> v) & 1u)) { u.x ^= 0x80008000u; u.y ^= 0x80008000u; u.z ^= 0x80008000u; u.w ^= 0x80008000u; }
  return u;
}
__device__ __forceinline__ void acc_chunk(float (&acc)[8], uint4 u) {
  float2 a = unpack_bf2(u.x), b = unpack_bf2(u.y), c = unpack_bf2(u.z), d = unpack_bf2(u.w);
  acc[0] += a.x; acc[1] += a.y; acc[2] += b.x; acc[3] += b.y;
  acc[4] += c.x; acc[5] += c.y; acc[6] += d.x; acc[7] += d.y;
}

// One warp per token.  History token slots: post h0.., author h0.., action row, surface row;
// candidate token slots: post h0.., author h0...  x = bf16(bf16(sum) * input_scale).
// This kernel carries every optional input and output (packed rows, pre-hashed rows, landing buffer, projected tokens, action
// sets, fp32 rows, debug taps, rows-only); the plain build has its own below.
// Continuous history actions (project_continuous_value_to_embedding, recsys_model.py:1850-1886).  Hidden activations
// of every configured column for one token, gelu(norm(v) * w1), into hid[c][0..hidden): the warp's scratch.
__device__ __forceinline__ void cont_hidden(const TokenBuildArgs& a, const float* __restrict__ vals, int lane, float (*hid)[64]) {
  for (int c = 0; c < a.n_cont; ++c) {
    float v = __ldg(vals + a.cont_index[c]);
    v = fminf(fmaxf(v, 0.f), a.cont_scale[c]);                                        // normalize_continuous_value, 1756-1765
    v = a.cont_log[c] ? log1pf(v) / log1pf(a.cont_scale[c]) : v / a.cont_scale[c];
    for (int j = lane; j < a.cont_hidden; j += 32) hid[c][j] = gelu_tanh_f(v * __bfloat162float(a.cont_w1[c][j]));
  }
  __syncwarp();
}
// tv[0..8) (columns col..col+7 of the token, bf16-valued) += bf16(hid[c] @ w2[c]) for every configured column, one
// rounding per addend.
__device__ __forceinline__ void cont_add(const TokenBuildArgs& a, const float (*hid)[64], int col, float (&tv)[8]) {
  for (int c = 0; c < a.n_cont; ++c) {
    float e[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int j = 0; j < a.cont_hidden; ++j) {
      const float h = hid[c][j];
      const uint4 u = __ldg(reinterpret_cast<const uint4*>(a.cont_w2[c] + (long long)j * a.D + col));
      const float2 p0 = unpack_bf2(u.x), p1 = unpack_bf2(u.y), p2 = unpack_bf2(u.z), p3 = unpack_bf2(u.w);
      e[0] = fmaf(h, p0.x, e[0]); e[1] = fmaf(h, p0.y, e[1]); e[2] = fmaf(h, p1.x, e[2]); e[3] = fmaf(h, p1.y, e[3]);
      e[4] = fmaf(h, p2.x, e[4]); e[5] = fmaf(h, p2.y, e[5]); e[6] = fmaf(h, p3.x, e[6]); e[7] = fmaf(h, p3.y, e[7]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) tv[i] = round_bf(tv[i] + round_bf(e[i]));
  }
}

// A row's statistics for the first fused RMSNorm: its sum of squares in slot 0, zero in the others (D / 64 slots, more than 32 of them from D = 2112 on)
__device__ __forceinline__ void store_row_ss(float* slots, int n, int lane, float ss) {
  for (int i = lane; i < n; i += 32) slots[i] = i == 0 ? ss : 0.f;
}

__global__ void __launch_bounds__(256, 3) build_tokens_kernel(TokenBuildArgs a) {
  // (no early launch signal here: the GEMM behind this kernel would park its CTAs - registers and all - on the SMs
  // while this bandwidth-bound kernel still needs every warp slot it can get)
  __shared__ float hid_s[8][PHX_MAX_HIST_CONT][64];
  const int T = a.S + a.C;
  const long long tok = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (tok >= (long long)a.B * T) return;
  // request and slot by 32-bit division (the launcher refuses B * T >= 2^31): a 64-bit '/' and '%' here cost more
  // instructions than the rest of the warp's prologue
  const int b = (int)((unsigned)tok / (unsigned)T), t = (int)((unsigned)tok - (unsigned)b * (unsigned)T);
  const int P = a.P;
  const bool is_front = t < a.S;              // rows in front of the candidates: user prefix + history
  const bool is_user = t < P;
  const bool is_hist = is_front && !is_user;
  const int Sh = a.S - P;                     // history slots of the input arrays
  const int H = a.item.num_hashes;
  const long long slot = is_user ? (long long)b : is_hist ? (long long)b * Sh + (t - P) : (long long)b * a.C + (t - a.S);
  long long orow;   // where this token's row goes
  if (a.pack.on() && !a.rows_only) {
    // packed rows: slots past the request's counts are not built at all (one token per warp: the whole warp leaves)
    if (is_front ? t >= a.pack.hist_cnt(b) : (t - a.S) >= a.pack.cand_cnt(b)) return;
    orow = is_front ? (long long)a.pack.hist_off[b] + t : a.pack.cand_base + a.pack.cand_off[b] + (t - a.S);
  } else {
    orow = token_row(a.split, a.B, a.S, T, b, t);
  }
  // lanes 0..H-1 hold the post rows, lanes H..2H-1 the author rows: hashed here, or taken as given; the user token
  // holds its user rows in lanes 0..Hu-1 and its IP rows behind them
  const int n_ip = (a.user_ip_hashes) ? a.Hip : 0;
  const int nrow = is_user ? a.Hu + n_ip : 2 * H;
  int my_idx = 0;
  if (is_user) {
    if (lane < a.Hu) my_idx = a.user_hashes[(long long)b * a.Hu + lane];
    else if (lane < nrow) my_idx = a.user_ip_hashes[(long long)b * a.Hip + (lane - a.Hu)];
  } else if (a.pre_hist_post) {
    if (lane < H) my_idx = (is_hist ? a.pre_hist_post : a.pre_cand_post)[slot * H + lane];
    else if (lane < 2 * H) my_idx = (is_hist ? a.pre_hist_author : a.pre_cand_author)[slot * H + (lane - H)];
  } else {
    const long long post_id = is_hist ? a.hist_post[slot] : a.cand_post[slot];
    const long long auth_id = is_hist ? a.hist_author[slot] : a.cand_author[slot];
    if (lane < H) my_idx = hash_one(post_id, a.item.scales[lane], a.item.biases[lane], a.item);
    else if (lane < 2 * H) {
      const int j = lane - H;
      my_idx = hash_one(auth_id, a.author.scales[j], a.author.biases[j], a.author);
    }
  }
  if (a.hashes && lane < 2 * H) a.hashes[tok * (2 * H) + lane] = my_idx;
  if (a.rows_only) return;   // uniform over the grid: the caller only wants the rows (exchange outside the kernel)
  const int first_hash = __shfl_sync(0xffffffffu, my_idx, 0);
  if (lane == 0) a.seg[orow] = (first_hash != 0) ? (is_front ? 1 : -1) : 0;
  int act = 0, srf = 0;
  if (is_hist) {
    if (a.hist_actions_bool) {   // the action set as the batch-prep hands it over: one byte per flag
      const unsigned char* f = a.hist_actions_bool + slot * a.num_action_types;
      act = (int)__ballot_sync(0xffffffffu, lane < a.num_action_types && f[lane] != 0);
    } else {
      act = a.hist_actions[slot];
    }
    srf = a.hist_surfaces[slot];
    if (!(a.action_multi_hot)) act = act < 0 ? 0 : (act > a.num_action_types ? a.num_action_types : act);
  } else if (!is_front && a.cand_surfaces) {
    srf = a.cand_surfaces[slot];
  }
  srf = srf < 0 ? 0 : (srf > a.num_surfaces ? a.num_surfaces : srf);
  const bool has_srf = is_hist || (!is_front && a.cand_surfaces);
  const bool has_cont = is_hist && a.n_cont > 0;
  float (*hid)[64] = hid_s[threadIdx.x >> 5];
  if (has_cont && !a.concat_hist) cont_hidden(a, a.hist_cont + slot * PHX_PREP_CONTINUOUS, lane, hid);
  // every lane takes part in these shuffles (lanes whose column chunk lies past D skip the loop below, so a
  // shuffle inside the loop would leave the warp split across two different shuffle instructions)
  const bf16* rowp[2 * PHX_MAX_HASHES];
  int my_pos = 0;   // exchanged rows: where slot `lane` of this token sits in the landing buffer
  if (a.landing && lane < 2 * H) my_pos = a.pos[tok * (2 * H) + lane];
#pragma unroll
  for (int j = 0; j < 2 * PHX_MAX_HASHES; ++j) {
    const int jj = j < nrow ? j : 0;
    const int idx = __shfl_sync(0xffffffffu, my_idx, jj);
    const int ps = __shfl_sync(0xffffffffu, my_pos, jj);
    rowp[j] = (a.landing) ? a.landing + (long long)ps * a.D : a.table.row_ptr(idx, a.D);
  }
  if (a.concat_hist) {
    // projected tokens: the gathered rows side by side - post rows, author rows, then the action and surface rows
    // (history) or the surface row (candidates that carry one); the user rows alone for the user token - as one GEMM
    // operand row (recsys_model.py:1903-1918, 2190-2221, 2307-2329); the projection, the addends, the scaling and
    // the row statistics follow in their own launches
    const int ngat = is_user ? a.Hu : 2 * H;
    const int nslot = ngat + (is_hist ? 2 : has_srf ? 1 : 0);
    bf16* dst = (is_user ? a.concat_user : is_hist ? a.concat_hist : a.concat_cand) + slot * (long long)nslot * a.D;
    for (int col = lane * 8; col < a.D; col += 256) {
#pragma unroll
      for (int j = 0; j < 2 * PHX_MAX_HASHES; ++j)
        if (j < ngat) *reinterpret_cast<uint4*>(dst + (long long)j * a.D + col) = __ldg(reinterpret_cast<const uint4*>(rowp[j] + col));
      if (is_hist)
        *reinterpret_cast<uint4*>(dst + (long long)ngat * a.D + col) = action_chunk(a, act, col, a.action_multi_hot);
      if (has_srf)
        *reinterpret_cast<uint4*>(dst + (long long)(nslot - 1) * a.D + col) =
            __ldg(reinterpret_cast<const uint4*>(a.surface_table + (long long)srf * a.D + col));
    }
    return;
  }
  float row_ss = 0.f;
  for (int col = lane * 8; col < a.D; col += 256) {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 2 * PHX_MAX_HASHES; ++j)
      if (j < nrow) acc_row(acc, rowp[j], col);
    if (is_hist) acc_chunk(acc, action_chunk(a, act, col, a.action_multi_hot));
    if (has_srf) acc_row(acc, a.surface_table + (long long)srf * a.D, col);
    float tv[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) tv[i] = round_bf(acc[i]);
    if (has_cont) cont_add(a, hid, col, tv);
    uint4 o;
    if (a.tokens) {
      o.x = pack_bf2(tv[0], tv[1]); o.y = pack_bf2(tv[2], tv[3]); o.z = pack_bf2(tv[4], tv[5]); o.w = pack_bf2(tv[6], tv[7]);
      *reinterpret_cast<uint4*>(a.tokens + tok * a.D + col) = o;
    }
    if (a.x32) {   // full-precision path: the token is the bf16 sum, its scaled value stays fp32
      float* dst = a.x32 + orow * a.D + col;
#pragma unroll
      for (int i = 0; i < 8; ++i) dst[i] = tv[i] * a.input_scale;
      continue;
    }
    float s[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) { s[i] = round_bf(tv[i] * a.input_scale); row_ss += s[i] * s[i]; }
    o.x = pack_bf2(s[0], s[1]); o.y = pack_bf2(s[2], s[3]); o.z = pack_bf2(s[4], s[5]); o.w = pack_bf2(s[6], s[7]);
    *reinterpret_cast<uint4*>(a.x + orow * a.D + col) = o;
  }
  if (a.row_ss) {   // statistics of the bf16 row for the first fused RMSNorm
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) row_ss += __shfl_xor_sync(0xffffffffu, row_ss, o);
    store_row_ss(a.row_ss + orow * a.ss_slots, a.ss_slots, lane, row_ss);
  }
}

// The plain token build (ids in, bf16 rows out; packed rows or not) for calls of many tokens.  The kernel above spends most of its
// instructions on the hash of one token - 64-bit multiplications and remainders on 2H lanes while the others wait - and
// on its prologue.  Here a warp takes TPW tokens: lane l hashes slot l % SL of token l / SL (SL = 2H rounded up to a power of
// two), then the warp walks over (token, 256 columns) pairs, the rows of two pairs in flight.  Same order of additions and
// roundings: the same bits.  The kernel above without its options, as it stood here before / this one with the tokens a warp that the
// launcher chooses: 640 tokens of 512 columns 7.7 / 5.6 us, 10240: 19.9 / 13.7, 81920: 103.5 / 56.9 (419 MB of rows, ids and
// results, part of them from L2); 32768 of 256 columns 35.8 / 22.1; a ragged batch of 48 packed requests 44.6 / 20.9.
template <int SL, int TPW>
__global__ void __launch_bounds__(256, SL == 8 ? 2 : 3) build_tokens_bulk_kernel(TokenBuildArgs a) {
  static_assert(SL * TPW <= 32, "a lane per hash");
  const int lane = threadIdx.x & 31, H = a.item.num_hashes;
  const unsigned T = (unsigned)(a.S + a.C), n_tok = (unsigned)a.B * T;      // the launcher refuses B * T >= 2^31
  const unsigned tok0 = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * TPW;
  if (tok0 >= n_tok) return;
  // ---- lane (k, slot): token k's facts and one of its hashes ----
  const int slot = lane % SL;
  const unsigned tok = tok0 + lane / SL;
  int orow = -1, aux = 0;            // where the token's row goes (-1: nowhere); its action (slot 0) and surface (slot 1)
  bool front = false;
  unsigned long long rowp = reinterpret_cast<unsigned long long>(a.table.base[0]);
  if (lane < SL * TPW && tok < n_tok) {
    const unsigned b = tok / T, t = tok - b * T;
    front = t < (unsigned)a.S;
    if (!a.pack.on()) orow = (int)token_row(a.split, a.B, a.S, (int)T, (int)b, (int)t);
    else if (front) orow = (int)t < a.pack.hist_cnt(b) ? a.pack.hist_off[b] + (int)t : -1;
    else orow = (int)(t - a.S) < a.pack.cand_cnt(b) ? (int)a.pack.cand_base + a.pack.cand_off[b] + (int)(t - a.S) : -1;
    if (orow >= 0) {
      const long long s = front ? (long long)b * a.S + t : (long long)b * a.C + (t - a.S);
      int idx = 0;
      if (slot < 2 * H) {
        const bool post = slot < H;
        const HashFamilyDev& f = post ? a.item : a.author;
        const long long id = __ldg((post ? (front ? a.hist_post : a.cand_post) : (front ? a.hist_author : a.cand_author)) + s);
        const int j = post ? slot : slot - H;
        idx = hash_one(id, f.scales[j], f.biases[j], f);
        rowp = reinterpret_cast<unsigned long long>(a.table.row_ptr(idx, a.D));
      }
      if (slot == 0) a.seg[orow] = idx != 0 ? (front ? 1 : -1) : 0;
      if (front && slot < 2) {
        aux = __ldg((slot == 0 ? a.hist_actions : a.hist_surfaces) + s);
        const int top = slot == 0 ? a.num_action_types : a.num_surfaces;
        aux = aux < 0 ? 0 : (aux > top ? top : aux);
      }
    }
  }
  __syncwarp();
  // ---- (token, 256 columns) pairs, two at a time; `on` and `hist` are uniform over the warp ----
  struct Pair { uint4 r[SL + 2]; int row; bool on, hist; };
  auto request = [&](int k, int col, bool there, Pair& p) {
    const int l0 = (k * SL) & 31;
    p.row = __shfl_sync(0xffffffffu, orow, l0);
    p.on = there && p.row >= 0;
    p.hist = __shfl_sync(0xffffffffu, (int)front, l0) != 0;
    const int act = __shfl_sync(0xffffffffu, aux, l0), srf = __shfl_sync(0xffffffffu, aux, l0 + 1);
#pragma unroll
    for (int j = 0; j < SL; ++j) {
      const bf16* src = reinterpret_cast<const bf16*>(__shfl_sync(0xffffffffu, rowp, l0 + j));
      if (p.on && j < 2 * H && col < a.D) p.r[j] = __ldg(reinterpret_cast<const uint4*>(src + col));
    }
    if (p.on && p.hist && col < a.D) {
      p.r[SL] = __ldg(reinterpret_cast<const uint4*>(a.action_table + (long long)act * a.D + col));
      p.r[SL + 1] = __ldg(reinterpret_cast<const uint4*>(a.surface_table + (long long)srf * a.D + col));
    }
  };
  auto add = [](float2 (&acc)[4], const uint4& u) {
    acc[0] = __fadd2_rn(acc[0], unpack_bf2(u.x)); acc[1] = __fadd2_rn(acc[1], unpack_bf2(u.y));
    acc[2] = __fadd2_rn(acc[2], unpack_bf2(u.z)); acc[3] = __fadd2_rn(acc[3], unpack_bf2(u.w));
  };
  float row_ss = 0.f;
  const float2 scale = make_float2(a.input_scale, a.input_scale);
  auto finish = [&](int col, bool first, bool last, const Pair& p) {
    if (!p.on) return;
    if (first) row_ss = 0.f;
    if (col < a.D) {
      float2 acc[4] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
      for (int j = 0; j < SL; ++j)
        if (j < 2 * H) add(acc, p.r[j]);
      if (p.hist) { add(acc, p.r[SL]); add(acc, p.r[SL + 1]); }
      uint32_t o[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {       // the token is rounded, then scaled and rounded again
        const float2 s = __fmul2_rn(unpack_bf2(pack_bf2(acc[i].x, acc[i].y)), scale);
        o[i] = pack_bf2(s.x, s.y);
        const float2 v = unpack_bf2(o[i]);
        row_ss += v.x * v.x; row_ss += v.y * v.y;
      }
      *reinterpret_cast<uint4*>(a.x + (long long)p.row * a.D + col) = make_uint4(o[0], o[1], o[2], o[3]);
    }
    if (last && a.row_ss) {               // statistics of the bf16 row for the first fused RMSNorm
      float ss = row_ss;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      store_row_ss(a.row_ss + (long long)p.row * a.ss_slots, a.ss_slots, lane, ss);
    }
  };
  const int span = (a.D + 255) & ~255;    // columns of a token's walk
  int k0 = 0, c0 = 0;
  while (k0 < TPW) {
    int k1 = k0, c1 = c0 + 256;
    if (c1 == span) { c1 = 0; ++k1; }
    Pair p0, p1;
    request(k0, c0 + lane * 8, true, p0);
    request(k1, c1 + lane * 8, k1 < TPW, p1);
    finish(c0 + lane * 8, c0 == 0, c0 + 256 == span, p0);
    finish(c1 + lane * 8, c1 == 0, c1 + 256 == span, p1);
    k0 = k1; c0 = c1 + 256;
    if (c0 == span) { c0 = 0; ++k0; }
  }
}
template <int TPW>
void build_tokens_bulk(const TokenBuildArgs& a, long long toks, cudaStream_t stream) {
  const unsigned grid = (unsigned)((toks + 8 * TPW - 1) / (8 * TPW));
  if (a.item.num_hashes == 1) build_tokens_bulk_kernel<2, TPW><<<grid, 256, 0, stream>>>(a);
  else if (a.item.num_hashes == 2) build_tokens_bulk_kernel<4, TPW><<<grid, 256, 0, stream>>>(a);
  else if constexpr (TPW <= 4) build_tokens_bulk_kernel<8, TPW><<<grid, 256, 0, stream>>>(a);
}

// Projected tokens, last step: x = bf16(token * input_scale) at the token's row of the residual stream (plain or
// split layout) with the row statistics of the first fused RMSNorm; tok_user [B, D], tok_hist [B*(S-P), D] and
// tok_cand [B*C, D] are the outputs of the projection GEMMs.  The addends of the reference's blocks that follow their
// projection are applied here: the sum of the IP rows on the user token (recsys_model.py:1920-1923) and the
// continuous-action embeddings on the history tokens (2249-2271).  One warp per token.
__global__ void __launch_bounds__(256) finish_tokens_kernel(const bf16* __restrict__ tok_user, const bf16* __restrict__ tok_hist,
                                                            const bf16* __restrict__ tok_cand, TokenBuildArgs a) {
  __shared__ float hid_s[8][PHX_MAX_HIST_CONT][64];
  const int T = a.S + a.C;
  const long long tok = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (tok >= (long long)a.B * T) return;
  // request and slot by 32-bit division (the launcher refuses B * T >= 2^31): a 64-bit '/' and '%' here cost more
  // instructions than the rest of the warp's prologue
  const int b = (int)((unsigned)tok / (unsigned)T), t = (int)((unsigned)tok - (unsigned)b * (unsigned)T);
  const int Sh = a.S - a.P;
  const bool is_user = t < a.P, is_hist = !is_user && t < a.S;
  const bf16* src = is_user ? tok_user + (long long)b * a.D
                  : is_hist ? tok_hist + ((long long)b * Sh + (t - a.P)) * a.D : tok_cand + ((long long)b * a.C + (t - a.S)) * a.D;
  long long orow;
  if (a.pack.on()) {
    if (t < a.S ? t >= a.pack.hist_cnt(b) : (t - a.S) >= a.pack.cand_cnt(b)) return;
    orow = t < a.S ? (long long)a.pack.hist_off[b] + t : a.pack.cand_base + a.pack.cand_off[b] + (t - a.S);
  } else {
    orow = token_row(a.split, a.B, a.S, T, b, t);
  }
  const bool has_cont = is_hist && a.n_cont > 0;
  const int n_ip = (is_user && a.user_ip_hashes) ? a.Hip : 0;
  float (*hid)[64] = hid_s[threadIdx.x >> 5];
  if (has_cont) cont_hidden(a, a.hist_cont + ((long long)b * Sh + (t - a.P)) * PHX_PREP_CONTINUOUS, lane, hid);
  float row_ss = 0.f;
  for (int col = lane * 8; col < a.D; col += 256) {
    uint4 u = *reinterpret_cast<const uint4*>(src + col);
    const float2 p0 = unpack_bf2(u.x), p1 = unpack_bf2(u.y), p2 = unpack_bf2(u.z), p3 = unpack_bf2(u.w);
    float s[8] = {p0.x, p0.y, p1.x, p1.y, p2.x, p2.y, p3.x, p3.y};
    if (n_ip > 0) {
      float ip[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      for (int j = 0; j < n_ip; ++j) acc_row(ip, a.table.row_ptr(__ldg(a.user_ip_hashes + (long long)b * a.Hip + j), a.D), col);
#pragma unroll
      for (int i = 0; i < 8; ++i) s[i] = round_bf(s[i] + round_bf(ip[i]));
    }
    if (has_cont) cont_add(a, hid, col, s);
    if (n_ip > 0 || has_cont) { u.x = pack_bf2(s[0], s[1]); u.y = pack_bf2(s[2], s[3]); u.z = pack_bf2(s[4], s[5]); u.w = pack_bf2(s[6], s[7]); }
    if (a.tokens) *reinterpret_cast<uint4*>(a.tokens + tok * a.D + col) = u;
#pragma unroll
    for (int i = 0; i < 8; ++i) { s[i] = round_bf(s[i] * a.input_scale); row_ss += s[i] * s[i]; }
    uint4 o;
    o.x = pack_bf2(s[0], s[1]); o.y = pack_bf2(s[2], s[3]); o.z = pack_bf2(s[4], s[5]); o.w = pack_bf2(s[6], s[7]);
    *reinterpret_cast<uint4*>(a.x + orow * a.D + col) = o;
  }
  if (a.row_ss) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) row_ss += __shfl_xor_sync(0xffffffffu, row_ss, o);
    store_row_ss(a.row_ss + orow * a.ss_slots, a.ss_slots, lane, row_ss);
  }
}

// Packed rows: the position of every packed row (RoPE) and, for the candidate rows, the slot of the [B, C] output
// arrays each one answers.  One thread per (request, slot).  Offsets in host memory are copied on the way (T >= 2: threads enough).
__global__ void pack_plan_kernel(PackMap pk, int B, int S, int C, int* __restrict__ pos_rows, int* __restrict__ out_index,
                                 int* __restrict__ hist_copy, int* __restrict__ cand_copy) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int T = S + C;
  if (i >= (long long)B * T) return;
  if (hist_copy && i <= B) { hist_copy[i] = pk.hist_off[i]; cand_copy[i] = pk.cand_off[i]; }
  const int b = (int)(i / T), t = (int)(i % T);
  if (t < S) {
    if (t < pk.hist_cnt(b)) pos_rows[pk.hist_off[b] + t] = t;
  } else if (t - S < pk.cand_cnt(b)) {
    const int r = pk.cand_off[b] + (t - S);
    pos_rows[pk.cand_base + r] = S;               // every candidate sits at the first position after the history
    out_index[r] = b * C + (t - S);
  }
}

__global__ void hash_ids_kernel(HashFamilyDev fam, const long long* __restrict__ ids, long long n, int* __restrict__ out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n * fam.num_hashes) return;
  const long long t = i / fam.num_hashes;
  const int j = (int)(i % fam.num_hashes);
  out[i] = hash_one(ids[t], fam.scales[j], fam.biases[j], fam);
}

// Stand-alone gather-sum: out[i] = bf16(sum_j table[hash_j(id_i)]) in hash order.  LANES lanes per id
// (LANES * 8 >= D or a loop), several ids per warp for narrow rows.
template <int LANES>
__global__ void __launch_bounds__(256) gather_sum_kernel(HashFamilyDev fam, TableView table, int D,
                                                         const long long* __restrict__ ids,
                                                         long long n, bf16* __restrict__ out) {
  const long long gid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / LANES;
  const int sub = threadIdx.x % LANES;
  const bool valid = gid < n;   // no early return: the shuffles below need every lane of the warp
  const long long id = valid ? __ldg(ids + gid) : 0;
  // lane j of the id's lane group computes hash j; the group shares the results by shuffle
  int mine = 0;
  if (sub < fam.num_hashes) {
    mine = hash_one(id, fam.scales[sub], fam.biases[sub], fam);
  }
  const bf16* rowp[PHX_MAX_HASHES];
#pragma unroll
  for (int j = 0; j < PHX_MAX_HASHES; ++j) rowp[j] = table.row_ptr(__shfl_sync(0xffffffffu, mine, j, LANES), D);
  for (int col = sub * 8; col < D && valid; col += LANES * 8) {
    uint4 u[PHX_MAX_HASHES];
#pragma unroll
    for (int j = 0; j < PHX_MAX_HASHES; ++j)
      if (j < fam.num_hashes) u[j] = __ldg(reinterpret_cast<const uint4*>(rowp[j] + col));
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int j = 0; j < PHX_MAX_HASHES; ++j) {
      if (j < fam.num_hashes) {
        float2 a = unpack_bf2(u[j].x), b = unpack_bf2(u[j].y), c = unpack_bf2(u[j].z), d = unpack_bf2(u[j].w);
        acc[0] += a.x; acc[1] += a.y; acc[2] += b.x; acc[3] += b.y;
        acc[4] += c.x; acc[5] += c.y; acc[6] += d.x; acc[7] += d.y;
      }
    }
    uint4 o;
    o.x = pack_bf2(acc[0], acc[1]); o.y = pack_bf2(acc[2], acc[3]); o.z = pack_bf2(acc[4], acc[5]); o.w = pack_bf2(acc[6], acc[7]);
    __stcs(reinterpret_cast<uint4*>(out + gid * D + col), o);
  }
}

// The same for many ids: a warp takes 32 / H ids at a time (H = hash count rounded up to a power of two), lane l hashes slot
// l % H of id l / H - every lane one hash, where the kernel above has 32 lanes wait for 4 - and the rows of 16 / H ids per
// lane group are requested before the first is summed; the next ids are already on their way.  Same order of additions.
// Measured (256 columns, 4 hashes): 4 M Zipf ids 2095 -> 977 us, 256 k 143 -> 74, 16 k 18.4 -> 12.9, 4 k 11.5 -> 10.8.
template <int LANES, int H>
__global__ void __launch_bounds__(256, 2) gather_sum_bulk_kernel(HashFamilyDev fam, TableView table, int D,
                                                                 const long long* __restrict__ ids, long long n,
                                                                 bf16* __restrict__ out) {
  constexpr int PER = 32 / H;         // ids per warp and round
  constexpr int W = 32 / LANES;       // ids side by side in one load instruction
  constexpr int G = 16 / H;           // such loads in flight per hash slot
  const int lane = threadIdx.x & 31, sub = lane % LANES, side = lane / LANES, slot = lane % H;
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  long long r = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const long long rounds = (n + PER - 1) / PER;
  auto load_id = [&](long long round) {
    const long long i = round * PER + lane / H;
    return (round < rounds && i < n) ? __ldg(ids + i) : 0ll;
  };
  long long scale = fam.scales[0], bias = fam.biases[0];   // of this lane's hash
#pragma unroll
  for (int j = 1; j < H; ++j)
    if (slot == j) { scale = fam.scales[j]; bias = fam.biases[j]; }
  long long next_id = load_id(r);
  for (; r < rounds; r += warps) {
    const long long id = next_id;
    next_id = load_id(r + warps);
    int row = 0;
    if (slot < fam.num_hashes) row = hash_one(id, scale, bias, fam);
    const unsigned long long mine = reinterpret_cast<unsigned long long>(table.row_ptr(row, D));
    for (int l0 = 0; l0 < PER; l0 += G * W) {
      const long long first = r * PER + l0 + side;
      for (int c0 = 0; c0 < D; c0 += LANES * 8) {        // uniform trip count: the shuffles need every lane
        const int col = c0 + sub * 8;
        uint4 u[G][H];
#pragma unroll
        for (int g = 0; g < G; ++g) {
          const bool on = col < D && first + g * W < n;
#pragma unroll
          for (int j = 0; j < H; ++j) {
            const bf16* src = reinterpret_cast<const bf16*>(__shfl_sync(0xffffffffu, mine, (l0 + g * W + side) * H + j));
            u[g][j] = (on && j < fam.num_hashes) ? __ldg(reinterpret_cast<const uint4*>(src + col)) : make_uint4(0u, 0u, 0u, 0u);
          }
        }
#pragma unroll
        for (int g = 0; g < G; ++g) {
          float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int j = 0; j < H; ++j) {
            if (j < fam.num_hashes) {
              const float2 a = unpack_bf2(u[g][j].x), b = unpack_bf2(u[g][j].y), c = unpack_bf2(u[g][j].z), d = unpack_bf2(u[g][j].w);
              acc[0] += a.x; acc[1] += a.y; acc[2] += b.x; acc[3] += b.y;
              acc[4] += c.x; acc[5] += c.y; acc[6] += d.x; acc[7] += d.y;
            }
          }
          uint4 o;
          o.x = pack_bf2(acc[0], acc[1]); o.y = pack_bf2(acc[2], acc[3]); o.z = pack_bf2(acc[4], acc[5]); o.w = pack_bf2(acc[6], acc[7]);
          if (col < D && first + g * W < n) __stcs(reinterpret_cast<uint4*>(out + (first + g * W) * D + col), o);
        }
      }
    }
  }
}

// From how many ids on.  A round of a warp is 32 / H ids and a pass over its columns for every 256 of them: too few rounds
// leave SMs idle where the kernel above has a warp for every id or two.  Time of that kernel over this one's, Zipf ids:
//   1 hash:   256 columns 0.83 at 4 k ids, 1.00 at 8 k, 512 columns 0.81 at 8 k, 1.13 at 16 k, 1024 columns 0.83 at 16 k, 1.00 at 32 k;
//             64 and 128 columns 0.90-0.94 at 4 k, 1.12 at 8 k
//   2 hashes: 256 columns 0.91 at 2 k, 1.01 at 4 k, 512 columns 0.85 at 4 k, 1.10 at 8 k, 1024 columns 0.88 at 8 k, 1.13 at 16 k
//   4 hashes: 256 columns 1.06 at 4 k, 512 columns 0.90 at 4 k, 1.05 at 6 k, 1024 columns 0.85 at 6 k, 1.00 at 12 k
inline bool gather_in_bulk(int num_hashes, int D, long long n) {
  const int H = num_hashes <= 1 ? 1 : (num_hashes <= 2 ? 2 : 4);
  const long long per_column = H == 4 ? 12 : 32 / H;
  return n >= (H == 1 ? 8192 : 4096) && n >= per_column * D;
}

template <int LANES>
void gather_sum_bulk(const HashFamilyDev& fam, const TableView& table, int D, const long long* ids, long long n, bf16* out, cudaStream_t stream) {
  const int H = fam.num_hashes <= 1 ? 1 : (fam.num_hashes <= 2 ? 2 : 4);
  const long long blocks = ((n + 32 / H - 1) / (32 / H) + 7) / 8;
  const unsigned grid = (unsigned)(blocks < 148 * 2 ? blocks : 148 * 2);
  if (H == 1) gather_sum_bulk_kernel<LANES, 1><<<grid, 256, 0, stream>>>(fam, table, D, ids, n, out);
  else if (H == 2) gather_sum_bulk_kernel<LANES, 2><<<grid, 256, 0, stream>>>(fam, table, D, ids, n, out);
  else gather_sum_bulk_kernel<LANES, 4><<<grid, 256, 0, stream>>>(fam, table, D, ids, n, out);
}

__device__ __forceinline__ uint32_t mix32(uint32_t x) {
  x ^= x >> 16; x *= 0x7FEB352Du; x ^= x >> 15; x *= 0x846CA68Bu; x ^= x >> 16;
  return x;
}
__device__ __forceinline__ float synth_value(unsigned long long row, int col, int width, uint32_t seed, float scale) {
  uint32_t x = (uint32_t)((row * (unsigned long long)width + (unsigned long long)col) & 0xFFFFFFFFull) ^ seed;
  x = mix32(x);
  return ((float)(x >> 16) - 32768.0f) * scale;
}

__global__ void table_fill_kernel(bf16* table, long long row0, long long rows, int width, uint32_t seed, float scale) {
  const long long total = rows * (long long)(width / 8);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / (width / 8);
    const int c = (int)(i % (width / 8)) * 8;
    float v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = synth_value((unsigned long long)(row0 + r), c + k, width, seed, scale);
    uint4 o;
    o.x = pack_bf2(v[0], v[1]); o.y = pack_bf2(v[2], v[3]); o.z = pack_bf2(v[4], v[5]); o.w = pack_bf2(v[6], v[7]);
    *reinterpret_cast<uint4*>(table + r * width + c) = o;
  }
}

// corpus rows: synthetic values rounded to bf16, fixed-order fp32 sum of squares, scaled, rounded again
__global__ void corpus_fill_kernel(bf16* rows_ptr, long long global_row0, long long rows, int dim, uint32_t seed) {
  for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += (long long)gridDim.x * blockDim.x) {
    float acc = 0.f;
    for (int c = 0; c < dim; ++c) {
      float v = round_bf(synth_value((unsigned long long)(global_row0 + r), c, dim, seed, 1.0f / 32768.0f));
      acc = acc + v * v;
    }
    const float inv = 1.0f / sqrtf(fmaxf(acc, 1e-12f));
    for (int c = 0; c < dim; c += 8) {
      float v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k)
        v[k] = round_bf(synth_value((unsigned long long)(global_row0 + r), c + k, dim, seed, 1.0f / 32768.0f)) * inv;
      uint4 o;
      o.x = pack_bf2(v[0], v[1]); o.y = pack_bf2(v[2], v[3]); o.z = pack_bf2(v[4], v[5]); o.w = pack_bf2(v[6], v[7]);
      *reinterpret_cast<uint4*>(rows_ptr + r * dim + c) = o;
    }
  }
}

}  // namespace

namespace {
// Tokens a warp of the plain build takes.  Few tokens want a warp each (every warp is one round trip for ids and one for rows), many
// want the hash shared.  The bulk kernel with 1 / 2 / 4 / 8 tokens, us (2 hashes): D = 512: 2560 tokens 6.0 / 6.7 / 8.3 / 12.4, 5120: 8.8 / 8.4 / 9.5 /
// 13.6, 10240: 15.5 / 14.4 / 13.9 / 18.4, 20480: 25.9 / 21.3 / 21.3 / 21.8, 81920: 88 / 70 / 61 / 57; D = 256: 2048: 4.7 / 4.7 / 6.0 /
// 8.3, 8192: 11.0 / 9.8 / 7.7 / 9.3, 32768: 36.7 / 25.8 / 22.3 / 21.9; D = 1024: 8688: 21.1 / 21.3 / 19.8 / 28.0.
inline int tokens_per_warp(long long toks) { return toks < 4096 ? 1 : toks < 8192 ? 2 : toks < 32768 ? 4 : 8; }
}  // namespace

phx_status build_tokens_launch(const TokenBuildArgs& a, cudaStream_t stream, std::string& err) {
  if (a.D % 8 != 0 || a.item.num_hashes != a.author.num_hashes || 2 * a.item.num_hashes > 32) {
    err = "build_tokens: D must be a multiple of 8 and hash counts must match";
    return PHX_E_ARG;
  }
  const long long toks = (long long)a.B * (a.S + a.C);
  if (toks == 0) return PHX_OK;
  if (toks >= (1ll << 31)) { err = "build_tokens: more than 2^31 tokens in one call"; return PHX_E_CAPACITY; }
  const int warps = 8;
  if (a.P && (a.Hu <= 0 || a.Hu + a.Hip > 2 * PHX_MAX_HASHES || !a.user_hashes)) { err = "build_tokens: user-prefix arguments"; return PHX_E_ARG; }
  if (a.n_cont && (a.cont_hidden <= 0 || a.cont_hidden > 64 || !a.hist_cont)) { err = "build_tokens: continuous-action arguments"; return PHX_E_ARG; }
  const bool plain = !(a.pre_hist_post || a.landing || a.concat_hist || a.action_multi_hot || a.x32 || a.tokens || a.hashes || a.rows_only ||
                       a.P || a.hist_actions_bool || a.cand_surfaces || a.n_cont);
  const int H = a.item.num_hashes;
  int tpw = plain && H <= 4 ? tokens_per_warp(toks) : 0;
  if (tpw == 8 && H > 2) tpw = 4;        // 2H lanes a token
  if (tpw == 8) build_tokens_bulk<8>(a, toks, stream);
  else if (tpw == 4) build_tokens_bulk<4>(a, toks, stream);
  else if (tpw == 2) build_tokens_bulk<2>(a, toks, stream);
  else if (tpw == 1) build_tokens_bulk<1>(a, toks, stream);
  else build_tokens_kernel<<<(unsigned)((toks + warps - 1) / warps), warps * 32, 0, stream>>>(a);
  PHX_CUDA_TRY(cudaGetLastError(), err);
  return PHX_OK;
}

phx_status pack_plan_launch(const PackMap& pk, int B, int S, int C, int* pos_rows, int* out_index, int* hist_copy, int* cand_copy,
                            cudaStream_t stream, std::string& err) {
  const long long n = (long long)B * (S + C);
  if (n == 0) return PHX_OK;
  pack_plan_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(pk, B, S, C, pos_rows, out_index, hist_copy, cand_copy);
  PHX_CUDA_TRY(cudaGetLastError(), err);
  return PHX_OK;
}

phx_status finish_tokens_launch(const bf16* tok_user, const bf16* tok_hist, const bf16* tok_cand, const TokenBuildArgs& a,
                                cudaStream_t stream, std::string& err) {
  const long long toks = (long long)a.B * (a.S + a.C);
  if (toks == 0) return PHX_OK;
  if (toks >= (1ll << 31)) { err = "finish_tokens: more than 2^31 tokens in one call"; return PHX_E_CAPACITY; }
  finish_tokens_kernel<<<(unsigned)((toks + 7) / 8), 256, 0, stream>>>(tok_user, tok_hist, tok_cand, a);
  PHX_CUDA_TRY(cudaGetLastError(), err);
  return PHX_OK;
}

phx_status hash_ids_launch(const HashFamilyDev& fam, const long long* ids, long long n, int* out, cudaStream_t stream,
                           std::string& err) {
  const long long total = n * fam.num_hashes;
  if (total == 0) return PHX_OK;
  hash_ids_kernel<<<(unsigned)((total + 255) / 256), 256, 0, stream>>>(fam, ids, n, out);
  PHX_CUDA_TRY(cudaGetLastError(), err);
  return PHX_OK;
}

phx_status gather_sum_launch(const HashFamilyDev& fam, const TableView& table, int D,
                             const long long* ids, long long n, bf16* out, cudaStream_t stream, std::string& err) {
  if (D % 8 != 0) { err = "gather_sum: D must be a multiple of 8"; return PHX_E_ARG; }
  if (n == 0) return PHX_OK;
  const bool bulk = gather_in_bulk(fam.num_hashes, D, n);
  dispatch_note(bulk ? DK_GATHER_BULK : DK_GATHER);
  if (bulk) {
    if (D <= 128) gather_sum_bulk<16>(fam, table, D, ids, n, out, stream);
    else gather_sum_bulk<32>(fam, table, D, ids, n, out, stream);
  } else if (D <= 128) {
    gather_sum_kernel<16><<<(unsigned)((n * 16 + 255) / 256), 256, 0, stream>>>(fam, table, D, ids, n, out);
  } else {
    gather_sum_kernel<32><<<(unsigned)((n * 32 + 255) / 256), 256, 0, stream>>>(fam, table, D, ids, n, out);
  }
  PHX_CUDA_TRY(cudaGetLastError(), err);
  return PHX_OK;
}

phx_status table_fill_launch(bf16* table, long long row0, long long rows, int width, uint32_t seed, float amp,
                             cudaStream_t stream, std::string& err) {
  if (rows == 0) return PHX_OK;
  table_fill_kernel<<<148 * 8, 256, 0, stream>>>(table, row0, rows, width, seed, amp / 32768.0f);
  PHX_CUDA_TRY(cudaGetLastError(), err);
  return PHX_OK;
}

phx_status corpus_fill_launch(bf16* rows_ptr, long long global_row0, long long rows, int dim, uint32_t seed,
                              cudaStream_t stream, std::string& err) {
  if (rows == 0) return PHX_OK;
  corpus_fill_kernel<<<148 * 8, 256, 0, stream>>>(rows_ptr, global_row0, rows, dim, seed);
  PHX_CUDA_TRY(cudaGetLastError(), err);
  return PHX_OK;
}

}  // namespace phx
