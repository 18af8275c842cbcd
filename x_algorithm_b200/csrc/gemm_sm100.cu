// bf16 GEMM for the Linear layers of the Phoenix trunk (phoenix/xrex/models/linear_layer.py:52-91)
// on Blackwell tensor cores: C[M,N] = epilogue(A[M,K] @ Wt[N,K]^T), fp32 accumulation in TMEM.
//
// Persistent kernel, one CTA per SM, 64 + 128 x NG threads (NG = epilogue groups: 2 or 4):
//   warp 0      TMA producer: A tile 128x64 and W tile per k-step (bf16, 128-byte swizzle) into a ring of
//               shared-memory stages (cp.async.bulk.tensor + mbarrier tx count)
//   warp 1      MMA issuer: one lane issues tcgen05.mma (N=BN, K=16) x4 per stage into one of two TMEM
//               accumulators, tcgen05.commit releases the stage / publishes the tile
//   warps 2..   epilogue, NG groups of four warps: tcgen05.ld the finished accumulator (each warp its
//               32-lane quadrant) in 64-column slabs, fused op (store | +residual | GELU-tanh | RoPE | RMSNorm
//               scale), bf16 slab staged in swizzled shared memory and written by one TMA bulk store; the
//               residual slab is fetched by TMA ahead of its use; overlaps the next tile's main loop through
//               the second accumulator
// PAIR variant (cta_group::2): the two CTAs of a cluster work on one 256 x BN tile.  Each loads its own 128 rows of
// A and its own half of the W tile, the even CTA issues one MMA (M=256) that reads both shared memories and
// writes each CTA's 128 rows into that CTA's TMEM, and each CTA runs the epilogue on its own rows.  Operand bytes
// per CTA per k-step fall from 128+BN to 128+BN/2 rows: that fill, and the power it takes, is what a tile costs beside its MMAs.
// Every mbarrier wait is bounded by wall time; on expiry the kernel raises *err_flag and unwinds.
#include <stdlib.h>
#include <string.h>

#include <type_traits>

#include "common.cuh"
#include "sm100_ptx.cuh"

namespace phx {

namespace {

using namespace sm100;
constexpr int BM = 128;
// threads: TMA warp, MMA warp, NG epilogue groups of four warps
constexpr int gemm_threads(int ng) { return 64 + ng * 128; }

template <int BN, bool PAIR, int NG>
struct Cfg {
  static_assert(NG == 2 || (NG == 4 && PAIR), "four epilogue groups need the smaller stages of a CTA pair");
  static constexpr int STAGES = PAIR ? 5 : 4;
  // output slab buffers, NSLAB / NG per epilogue group
  static constexpr int NSLAB = NG == 4 ? 4 : (PAIR ? ((BN == 256) ? 4 : 6) : ((BN == 256) ? 2 : 6));
  static constexpr int B_ROWS = PAIR ? BN / 2 : BN;   // rows of the W tile this CTA loads
  static constexpr int A_BYTES = BM * BK * 2;
  static constexpr int B_BYTES = B_ROWS * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int BAR_BYTES = 256;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + NSLAB * (128 * 64 * 2) + BAR_BYTES + 1024;  // + slabs, +1024 alignment slack
  static constexpr int TMEM_COLS = 2 * BN;                                    // two accumulators
};

// ---- epilogue helpers -----------------------------------------------------------------------------
constexpr int SLAB_COLS = 64;                 // one output slab = 128 rows x 64 bf16 columns = 128-byte rows
constexpr int SLAB_BYTES = BM * SLAB_COLS * 2;

__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, uint32_t src, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(map), "r"(src), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// named barrier `id` over the 128 threads of one epilogue group, AND-reducing a per-thread flag: every thread
// always arrives, so a thread that gave up on a bounded wait can never leave the others parked here
__device__ __forceinline__ bool epi_barrier_and(bool ok, int id) {
  uint32_t out;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.u32 q, %1, 0;\n bar.red.and.pred p, %2, 128, q;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(out) : "r"((uint32_t)ok), "r"(id) : "memory");
  return out != 0;
}
__device__ __forceinline__ uint4 ld_shared_v4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint4 v) {
  asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// Epilogue arithmetic, two columns per instruction (packed fp32) and one conversion per pair: an epilogue thread's
// instruction stream is what a tile with a short K waits for.  Measured: 163840 x 1024, K = 256, GELU 114.6 -> 94.2 us; a
// forward of one request 384 -> 349 us; full batches, the user tower and ragged batches gain no more than runs differ.
// fp32 accumulators -> the Linear output, a bf16 pair: rounded once, kept in the form it is stored in
__device__ __forceinline__ uint32_t linear_bf2(uint32_t a0, uint32_t a1, float2 rstd2) {
  const float2 v = __fmul2_rn(make_float2(__uint_as_float(a0), __uint_as_float(a1)), rstd2);
  return pack_bf2(v.x, v.y);
}
__device__ __forceinline__ float2 bf2_to_f2(uint32_t b) { return make_float2(__uint_as_float(b << 16), __uint_as_float(b & 0xFFFF0000u)); }
// GELU, tanh form, of a bf16 pair (gelu_tanh_f's formula: sqrt(2/pi) (x + 0.044715 x^3) as x (c0 + c1 x^2)).  Rounded to bf16 the
// results equal gelu_tanh_f's for every bf16 value, but for the sign of zeros (negative x where tanh is -1); keeping that sign
// takes 163840 x 2048, K = 512 from 307 to 311 us (or'ed in) or 313 us (x (0.5 + 0.5 t)).
__device__ __forceinline__ uint32_t gelu_bf2(uint32_t b) {
  const float2 x = bf2_to_f2(b);
  const float2 p = __ffma2_rn(__fmul2_rn(x, x), make_float2(0.035677408136300125f, 0.035677408136300125f),
                              make_float2(0.7978845608028654f, 0.7978845608028654f));
  const float2 in = __fmul2_rn(x, p);
  float2 t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t.x) : "f"(in.x));
  asm("tanh.approx.f32 %0, %1;" : "=f"(t.y) : "f"(in.y));
  const float2 h = __fmul2_rn(x, make_float2(0.5f, 0.5f));
  const float2 g = __ffma2_rn(h, t, h);
  return pack_bf2(g.x, g.y);
}
// one RoPE pair of columns against its partner pair: (lo, hi) -> (lo c - hi s, hi c + lo s).  Which of the two products of a sum is
// rounded before the other goes into the fma shows in a few results per million: hi s and hi c, and with heads of 128
// lo s instead of hi c.
template <bool D128>
__device__ __forceinline__ void rope_bf2(uint32_t& lo, uint32_t& hi, float c0, float c1, float s0, float s1) {
  const float2 x1 = bf2_to_f2(lo), x2 = bf2_to_f2(hi), c = make_float2(c0, c1), sn = make_float2(s0, s1);
  const float2 a = __fmul2_rn(x2, sn);
  const float2 l = __ffma2_rn(x1, c, make_float2(-a.x, -a.y));
  const float2 h = D128 ? __ffma2_rn(x2, c, __fmul2_rn(x1, sn)) : __ffma2_rn(x1, sn, __fmul2_rn(x2, c));
  lo = pack_bf2(l.x, l.y); hi = pack_bf2(h.x, h.y);
}
// position of a token row: the row's slot in its request, at most pos_cap (GemmRope); token rows fit 31 bits
__device__ __forceinline__ int rope_pos(const GemmRope& rope, long long row, bool in) {
  if (rope.pos_rows) return in ? rope.pos_rows[row] : 0;
  if (rope.split_rows != 0 && row >= rope.split_rows) return rope.pos_cap;
  const int t = (int)((unsigned)row % (unsigned)rope.T);
  return t < rope.pos_cap ? t : rope.pos_cap;
}

// Column tiles of a QKV projection that nobody reads: of every `per` the first `skip`, in the first `m_tiles` row tiles.  Not part of GemmRope, which
// the kernels for few tiles take as well: with 24 bytes more in it (416 bytes of parameters in place of 392) each of their launches took
// 0.35 us longer on the host, the small tower's 22-launch forward 64 us in place of 58 (and 97.6 us on the device in place of 95.6).
struct GemmLeftOut { int m_tiles = 0, per = 1, skip = 0; };
static_assert(sizeof(GemmRope) <= 56 && sizeof(GemmNorm) <= 32, "parameters of gemm_small_kernel: measure the host time of a small call");
__host__ __device__ constexpr bool leaves_out(int bn, int epi, bool pair) { return epi == EPI_ROPE128 && pair && bn == 256; }

template <int BN, int EPI, bool PAIR, int NG>
__global__ void __launch_bounds__(gemm_threads(NG), 1)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                    const __grid_constant__ CUtensorMap map_c, const __grid_constant__ CUtensorMap map_r,
                    GemmRope rope, GemmNorm norm, long long M, int N, int K, int* err_flag,
                    unsigned long long* counters, GemmLeftOut out) {
  // C and R may be the same buffer (in-place residual update): a slab is fetched before it is written back,
  // and no other CTA touches the tile.
  using cfg = Cfg<BN, PAIR, NG>;
  // columns per epilogue work item: one 64-column slab, or a whole head of 128 whose halves RoPE rotates against each other
  constexpr int ITEM_COLS = (EPI == EPI_ROPE128) ? 128 : SLAB_COLS;
  constexpr int ITEM_SLABS = ITEM_COLS / SLAB_COLS;
  constexpr int SLABS = BN / ITEM_COLS;      // items per tile
  // epilogue threads that drain one accumulator (a tile with fewer slabs than groups is shared by SLABS groups)
  constexpr int DRAIN_THREADS = (SLABS < NG ? SLABS : NG) * 128 * (PAIR ? 2 : 1);
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;  // swizzle atoms need 1024-byte alignment
  const uint32_t slab_base = smem_base + cfg::STAGES * cfg::STAGE_BYTES;   // output slab buffers
  const uint32_t bars = slab_base + cfg::NSLAB * SLAB_BYTES;
  // barrier slots (8 bytes each): full[STAGES], empty[STAGES], tmem_full[2], tmem_empty[2], res[NSLAB]; then the TMEM slot
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (cfg::STAGES + s); };
  auto tfull_bar = [&](int a) { return bars + 8u * (2 * cfg::STAGES + a); };
  auto tempty_bar = [&](int a) { return bars + 8u * (2 * cfg::STAGES + 2 + a); };
  auto res_bar = [&](int b) { return bars + 8u * (2 * cfg::STAGES + 4 + b); };
  const uint32_t tmem_slot = bars + 8u * (2 * cfg::STAGES + 4 + cfg::NSLAB);
  uint32_t* tmem_slot_ptr = reinterpret_cast<uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));

  const int warp = warp_index(), lane = threadIdx.x & 31;
  if (counters && blockIdx.x == 0 && threadIdx.x == 0) counters[3] = globaltimer_ns();   // diagnostics: kernel entry
  constexpr int TILE_M = PAIR ? 2 * BM : BM;          // rows of one work tile (of the CTA pair)
  const uint32_t rank = PAIR ? cluster_ctarank() : 0u; // 0 = the CTA that issues the pair's MMAs
  const long long first_tile = PAIR ? (blockIdx.x >> 1) : blockIdx.x;
  const long long tile_step = PAIR ? (gridDim.x >> 1) : gridDim.x;
  const int n_tiles = (N + BN - 1) / BN;
  const long long m_tiles = (M + TILE_M - 1) / TILE_M;
  // work list: the row tiles whose q columns nobody reads, their other column tiles; then every column tile of the other rows
  constexpr bool KV = leaves_out(BN, EPI, PAIR);
  const int kept = out.per - out.skip, kv_n = KV ? n_tiles / out.per * kept : 1;      // column tiles of such a row tile
  const long long kv_tiles = KV ? (long long)out.m_tiles * kv_n : 0;
  const long long total_tiles = KV ? kv_tiles + (m_tiles - out.m_tiles) * n_tiles : m_tiles * n_tiles;
  auto place = [&](long long tile, long long& m_blk, int& n_blk) {
    if constexpr (KV) {
      if (tile < kv_tiles) {
        const int j = (int)(tile % kv_n);
        m_blk = tile / kv_n; n_blk = j / kept * out.per + out.skip + j % kept;
      } else {
        tile -= kv_tiles;
        m_blk = out.m_tiles + tile / n_tiles; n_blk = (int)(tile % n_tiles);
      }
    } else {
      m_blk = tile / n_tiles; n_blk = (int)(tile % n_tiles);
    }
  };
  const int k_blocks = (K + BK - 1) / BK;
  volatile int* verr = err_flag;

  if (threadIdx.x == 0) {
    *gave_up() = 0;
    prefetch_map(&map_a); prefetch_map(&map_b); prefetch_map(&map_c);
    if (EPI == EPI_RESIDUAL) prefetch_map(&map_r);
    for (int s = 0; s < cfg::STAGES; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    // a pair's accumulators are drained by the epilogue threads of both CTAs, counted on the issuing CTA
    for (int a = 0; a < 2; ++a) { mbar_init(tfull_bar(a), 1); mbar_init(tempty_bar(a), DRAIN_THREADS); }
    for (int a = 0; a < cfg::NSLAB; ++a) mbar_init(res_bar(a), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    if (PAIR) tmem_alloc_pair(tmem_slot, cfg::TMEM_COLS);
    else tmem_alloc(tmem_slot, cfg::TMEM_COLS);
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();   // the peer's barriers are initialised before anything signals them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;
  // Programmatic dependent launch: everything above (barriers, tensor memory, cluster hand-shake) touched no global
  // data, so it may run while the kernel in front of this one on the stream is still finishing.  From here on the
  // kernel reads what its predecessor wrote: wait for it (a no-op for a launch without the attribute), and let the
  // kernel behind start its own set-up.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (elect_one()) {
      int stage = 0; uint32_t phase = 0;
      bool ok = true;
      for (long long tile = first_tile; tile < total_tiles && ok; tile += tile_step) {
        int n_blk; long long m_blk;
        place(tile, m_blk, n_blk);
        for (int kb = 0; kb < k_blocks; ++kb) {
          if (!mbar_wait(empty_bar(stage), phase ^ 1, verr)) { ok = false; break; }
          const uint32_t a_dst = smem_base + stage * cfg::STAGE_BYTES;
          const uint32_t b_dst = a_dst + cfg::A_BYTES;
          if (PAIR) {
            // both CTAs' bytes are counted on the issuing CTA's barrier
            const uint32_t bar0 = mapa_shared(full_bar(stage), 0);
            if (rank == 0) mbar_expect_tx(full_bar(stage), 2 * cfg::STAGE_BYTES);
            tma_load_2d_pair(a_dst, &map_a, bar0, kb * BK, (int)(m_blk * TILE_M + rank * BM));
            tma_load_2d_pair(b_dst, &map_b, bar0, kb * BK, n_blk * BN + (int)rank * cfg::B_ROWS);
          } else {
            mbar_expect_tx(full_bar(stage), cfg::STAGE_BYTES);
            tma_load_2d(a_dst, &map_a, full_bar(stage), kb * BK, (int)(m_blk * BM));
            tma_load_2d(b_dst, &map_b, full_bar(stage), kb * BK, n_blk * BN);
          }
          if (++stage == cfg::STAGES) { stage = 0; phase ^= 1; }
        }
      }
      if (PAIR && ok) {
        // the issuing CTA releases stages in this CTA by remote arrivals: all of them must have landed before
        // this CTA may retire
        for (int s = 0; s < cfg::STAGES; ++s) {
          if (!mbar_wait(empty_bar(stage), phase ^ 1, verr)) break;
          if (++stage == cfg::STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    // One thread, and the pipe only stays fed if this loop is short: the thread shares its scheduler with four
    // epilogue warps, so every instruction here costs several cycles of wall time.  Stage addresses and descriptors
    // are carried as running values (no per-step address arithmetic), the wait counters exist only when asked for.
    if (rank == 0 && elect_one()) {
      constexpr uint32_t idesc = make_idesc(TILE_M, BN);
      constexpr uint64_t DESC_STEP = (uint64_t)(cfg::STAGE_BYTES >> 4);    // descriptor address field: bytes / 16
      const uint64_t adesc0 = make_smem_desc(smem_base);
      const uint64_t bdesc0 = make_smem_desc(smem_base + cfg::A_BYTES);
      uint64_t adesc = adesc0, bdesc = bdesc0;
      uint32_t full_addr = full_bar(0), empty_addr = empty_bar(0);
      int stage = 0; uint32_t phase = 0;
      uint32_t it = 0;
      bool ok = true;
      long long cnt_tempty = 0, cnt_full = 0;
      const bool timed = counters != nullptr;
      const long long t_start = timed ? clock64() : 0;
      if (timed && blockIdx.x == 0) counters[4] = globaltimer_ns();   // first MMA wait
      for (long long tile = first_tile; tile < total_tiles && ok; tile += tile_step, ++it) {
        const uint32_t acc = it & 1, acc_phase = (it >> 1) & 1;
        long long c0 = timed ? clock64() : 0;
        if (!mbar_wait(tempty_bar(acc), acc_phase ^ 1, verr)) { ok = false; break; }
        if (timed) cnt_tempty += clock64() - c0;
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + acc * BN;
        for (int kb = 0; kb < k_blocks; ++kb) {
          if (timed) c0 = clock64();
          if (!mbar_wait(full_addr, phase, verr)) { ok = false; break; }
          if (timed) cnt_full += clock64() - c0;
          tc_fence_after();
          // advancing 16 elements along K inside the 128-byte swizzle row = +32 bytes = +2 in the address field
          if (PAIR) {
            umma_bf16_pair(tmem_d, adesc, bdesc, idesc, kb != 0);
            umma_bf16_pair(tmem_d, adesc + 2, bdesc + 2, idesc, 1);
            umma_bf16_pair(tmem_d, adesc + 4, bdesc + 4, idesc, 1);
            umma_bf16_pair(tmem_d, adesc + 6, bdesc + 6, idesc, 1);
            umma_commit_pair(empty_addr, 3);   // stage reusable (in both CTAs) once these MMAs have read it
          } else {
            umma_bf16(tmem_d, adesc, bdesc, idesc, kb != 0);
            umma_bf16(tmem_d, adesc + 2, bdesc + 2, idesc, 1);
            umma_bf16(tmem_d, adesc + 4, bdesc + 4, idesc, 1);
            umma_bf16(tmem_d, adesc + 6, bdesc + 6, idesc, 1);
            umma_commit(empty_addr);
          }
          adesc += DESC_STEP; bdesc += DESC_STEP; full_addr += 8; empty_addr += 8;
          if (++stage == cfg::STAGES) {
            stage = 0; phase ^= 1;
            adesc = adesc0; bdesc = bdesc0; full_addr = full_bar(0); empty_addr = empty_bar(0);
          }
        }
        if (ok) {  // accumulator complete
          if (PAIR) umma_commit_pair(tfull_bar(acc), 3); else umma_commit(tfull_bar(acc));
        }
      }
      if (timed) {   // diagnostic: where the MMA issuer spent its time (cycles summed over CTAs)
        atomicAdd(&counters[0], (unsigned long long)(clock64() - t_start));
        atomicAdd(&counters[1], (unsigned long long)cnt_full);
        atomicAdd(&counters[2], (unsigned long long)cnt_tempty);
        if (blockIdx.x == 0) counters[5] = globaltimer_ns();   // last MMA issued
      }
    }
  } else {
    // ---------------- epilogue (warps 2..: NG groups of four warps) ----------------
    // Work item = one 64-column slab of a tile; group gidx takes the items with q % NG == gidx and owns NB
    // slab buffers, an issuing thread and named barrier 1 + gidx.  Per item: TMEM -> registers -> fused op
    // -> swizzled shared-memory slab -> one TMA bulk store.  The residual slab arrives by TMA into the same
    // buffer (up to NB - 1 items ahead, at least one) and is updated in place.
    constexpr int NB = cfg::NSLAB / NG / ITEM_SLABS;    // item buffers per group
    static_assert(NB >= 1, "an item needs its slab buffers");
    constexpr bool RES = (EPI == EPI_RESIDUAL);
    constexpr int DIST = NB - 1;                        // residual prefetch distance (items of this group)
    const int ew = warp - 2;
    const int gidx = ew >> 2;
    const int quad = warp & 3;                          // TMEM lane quadrant this warp may read
    const int row_in_tile = quad * 32 + lane;
    const bool issuer_warp = (ew & 3) == 0;             // one lane of it issues the group's copies
    const long long my_tiles = (total_tiles > first_tile) ? (total_tiles - first_tile + tile_step - 1) / tile_step : 0;
    // the accumulator-drained signal goes to the CTA that issues the MMAs
    const uint32_t tempty0 = PAIR ? mapa_shared(tempty_bar(0), 0) : tempty_bar(0);
    const uint32_t tempty1 = PAIR ? mapa_shared(tempty_bar(1), 0) : tempty_bar(1);
    auto release_acc = [&](uint32_t a) {
      tc_fence_before();
      if (PAIR) mbar_arrive_cluster(a ? tempty1 : tempty0);
      else mbar_arrive(a ? tempty1 : tempty0);
    };
    const long long total_items = my_tiles * SLABS;
    const long long my_items = (total_items > gidx) ? (total_items - gidx + NG - 1) / NG : 0;
    const uint32_t gslab = slab_base + gidx * NB * ITEM_SLABS * SLAB_BYTES;
    auto coords = [&](long long i, long long& m0, int& c0) {   // i = item index inside this group
      const long long q = (long long)NG * i + gidx;
      const long long tile = first_tile + (q / SLABS) * tile_step;
      int n_blk;
      place(tile, m0, n_blk);
      m0 = m0 * TILE_M + rank * BM;
      c0 = n_blk * BN + (int)(q % SLABS) * ITEM_COLS;
    };
    auto issue_res = [&](long long i) {
      long long m1; int c1; coords(i, m1, c1);
      const int bi = (int)(i % NB);
      mbar_expect_tx(res_bar(gidx * NB + bi), SLAB_BYTES);
      tma_load_2d(gslab + bi * SLAB_BYTES, &map_r, res_bar(gidx * NB + bi), c1, (int)m1);
    };
    if (RES && issuer_warp && elect_one()) {
      for (int i = 0; i < DIST && i < my_items; ++i) issue_res(i);
    }
    float rstd = 1.0f;   // 1/rms of this thread's row, refreshed at each tile
    for (long long i = 0; i < my_items; ++i) {
      const long long q = (long long)NG * i + gidx;
      const int s = (int)(q % SLABS);
      const uint32_t it = (uint32_t)(q / SLABS), acc = it & 1, acc_phase = (it >> 1) & 1;
      const int bi = (int)(i % NB);
      const uint32_t slab = gslab + bi * ITEM_SLABS * SLAB_BYTES;
      long long m0; int c0; coords(i, m0, c0);
      const bool first_of_tile = (s < NG);              // this group's first slab of the tile
      // RMSNorm folded into this GEMM: the row's 1/rms comes from the sum of squares its producer left behind
      // (partials in fixed slots, summed in slot order: deterministic), the gain is folded into the weights.
      // Read once per tile, before the wait on the accumulator, so the loads hide behind it.
      float4 ssa = make_float4(0.f, 0.f, 0.f, 0.f), ssb = ssa;   // up to 8 partials, summed after the wait below
      float ss_rest = 0.f;
      const bool need_rstd = !RES && norm.ss_in != nullptr && first_of_tile;
      if (need_rstd) {
        const long long row = m0 + row_in_tile;
        if (row < M) {
          const float* sp = norm.ss_in + row * norm.slots_in;
          if (norm.slots_in == 8) {
            ssa = __ldg(reinterpret_cast<const float4*>(sp));
            ssb = __ldg(reinterpret_cast<const float4*>(sp + 4));
          } else if (norm.slots_in == 4) {
            ssa = __ldg(reinterpret_cast<const float4*>(sp));
          } else {
            for (int t = 0; t < norm.slots_in; ++t) ss_rest += __ldg(sp + t);
          }
        }
      }
      const bool last_of_tile = (s + NG >= SLABS);      // ... and its last
      // RoPE: whether this item is rotated (q and k parts are), the row's position, and the first pass' angles, all before
      // the wait on the accumulator
      constexpr bool ROPE = EPI == EPI_ROPE || EPI == EPI_ROPE128, D128 = EPI == EPI_ROPE128;
      const bool d64 = ROPE && !D128 && rope.dh == 64;
      // A thread is a row.  With one table row per position every lane of a load touched a cache line of its own, 32 tag
      // look-ups an instruction and 5.5 k cycles a 256-column tile, which is what the tile waited for; with positions
      // as the fast index a load touches four or five lines (more where a warp's rows cross a request).  User tower (32768 rows, K = 256, four layers) 517 -> 489 us,
      // two layers of 8 x 1086 rows with heads of 128 455 -> 449 us; full batches (K = 512) gain no more than runs differ.
      float4 ang[8];
      const float4* ang_col = nullptr;
      auto part_rotated = [&](int p) {
        const int part = D128 ? (c0 >> 7) : d64 ? (c0 >> 6) : (c0 >> 5) + p;
        return part % rope.group <= rope.g;
      };
      auto load_angles = [&](int p) {
#pragma unroll
        for (int t = 0; t < 8; ++t) ang[t] = __ldg(ang_col + (((D128 || d64) ? 8 * p : 0) + t) * rope.n_pos);
      };
      if (ROPE) {
        const long long row = m0 + row_in_tile;
        ang_col = rope.angles + rope_pos(rope, row + rope.row_offset, row < M);
        if (part_rotated(0)) load_angles(0);
      }
      if (RES && issuer_warp && i + DIST < my_items && elect_one()) {
        // the buffer of item i + DIST was last used by item i - 1: its store must have drained
        bulk_wait_read<0>();
        issue_res(i + DIST);
      }
      bool ok = true;
      if (first_of_tile) ok = mbar_wait(tfull_bar(acc), acc_phase, verr);
      if (RES && ok) ok = mbar_wait(res_bar(gidx * NB + bi), (uint32_t)((i / NB) & 1), verr);
      ok = __all_sync(0xffffffffu, ok);
      if (need_rstd) {   // slot order: deterministic
        float ss = ss_rest;
        ss += ssa.x; ss += ssa.y; ss += ssa.z; ss += ssa.w; ss += ssb.x; ss += ssb.y; ss += ssb.z; ss += ssb.w;
        rstd = rsqrtf(ss * norm.inv_d + norm.eps);
      }
      const uint32_t row_addr = slab + row_in_tile * 128;
      const int sw = row_in_tile & 7;
      const uint32_t taddr = tmem_base + acc * BN + ((uint32_t)(quad * 32) << 16) + s * ITEM_COLS;
      if (!RES) {
        // the store that last read this buffer (item i - NB of this group) must have drained before it is rewritten
        if (issuer_warp && elect_one()) bulk_wait_read<NB - 1>();
        ok = epi_barrier_and(ok, 1 + gidx);
      }
      if (ok) {
        tc_fence_after();
        const float2 rstd2 = make_float2(rstd, rstd);
        if (ROPE) {
          // RoPE on the q / k head parts of this item (layers.py:52-67, 784-788), pairs (j, j + dh/2), in
          // passes of 16 pairs so that only 32 values are live: head dim 64 = one part per slab, pass p rotates
          // columns [16p, 16p+16) against [32+16p, 48+16p); head dim 32 = pass p is the slab's p-th part; head dim 128 =
          // four passes, [16p, 16p+16) of the item's first slab against the same columns of its second.
#pragma unroll
          for (int p = 0; p < (D128 ? 4 : 2); ++p) {
            const int lo_col = (D128 || d64) ? 16 * p : 32 * p;
            const int hi_col = D128 ? 64 + 16 * p : d64 ? 32 + 16 * p : 32 * p + 16;
            uint32_t rl[16], rh[16];
            tmem_ld16_nowait(taddr + lo_col, rl);
            tmem_ld16_nowait(taddr + hi_col, rh);
            tmem_ld_wait();
            if (p == (D128 ? 3 : 1) && last_of_tile) release_acc(acc);
            uint32_t lo[8], hi[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              lo[k] = linear_bf2(rl[2 * k], rl[2 * k + 1], rstd2);
              hi[k] = linear_bf2(rh[2 * k], rh[2 * k + 1], rstd2);
            }
            if (part_rotated(p)) {   // v parts pass through
#pragma unroll
              for (int t = 0; t < 8; ++t) rope_bf2<D128>(lo[t], hi[t], ang[t].x, ang[t].y, ang[t].z, ang[t].w);
            }
            if (p + 1 < (D128 ? 4 : 2) && part_rotated(p + 1)) load_angles(p + 1);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              st_shared_v4(row_addr + ((uint32_t)(((lo_col >> 3) + h) ^ sw) << 4), make_uint4(lo[4 * h], lo[4 * h + 1], lo[4 * h + 2], lo[4 * h + 3]));
              const uint32_t hi_addr = D128 ? row_addr + SLAB_BYTES + ((uint32_t)(((lo_col >> 3) + h) ^ sw) << 4)
                                            : row_addr + ((uint32_t)(((hi_col >> 3) + h) ^ sw) << 4);
              st_shared_v4(hi_addr, make_uint4(hi[4 * h], hi[4 * h + 1], hi[4 * h + 2], hi[4 * h + 3]));
            }
          }
        } else {
          float ss_out = 0.f;
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {              // two 32-column halves keep the register footprint low
            uint32_t r[32];
            tmem_ld32(taddr + hh * 32, r);
            if (hh == 1 && last_of_tile) release_acc(acc);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const uint32_t addr = row_addr + ((uint32_t)((hh * 4 + c) ^ sw) << 4);
              uint32_t o[4];
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                o[k] = linear_bf2(r[c * 8 + 2 * k], r[c * 8 + 2 * k + 1], rstd2);
                if (EPI == EPI_GELU) o[k] = gelu_bf2(o[k]);
              }
              if (RES) {
                const uint4 rr = ld_shared_v4(addr);
                const uint32_t rb[4] = {rr.x, rr.y, rr.z, rr.w};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                  const float2 v = __fadd2_rn(bf2_to_f2(o[k]), bf2_to_f2(rb[k]));
                  ss_out += v.x * v.x; ss_out += v.y * v.y;          // statistics of the fp32 sums (pre-rounding)
                  o[k] = pack_bf2(v.x, v.y);
                }
              }
              st_shared_v4(addr, make_uint4(o[0], o[1], o[2], o[3]));
            }
          }
          if (RES && norm.ss_out != nullptr && m0 + row_in_tile < M && c0 < N)
            norm.ss_out[(m0 + row_in_tile) * (long long)(N / SLAB_COLS) + c0 / SLAB_COLS] = ss_out;
        }
        fence_async_smem();
      }
      if (!epi_barrier_and(ok, 1 + gidx)) break;        // uniform over the group's 128 threads
      if (issuer_warp && c0 < N && m0 < M && elect_one()) {
        tma_store_2d(&map_c, slab, c0, (int)m0);
        if (ITEM_SLABS == 2) tma_store_2d(&map_c, slab + SLAB_BYTES, c0 + SLAB_COLS, (int)m0);
        bulk_commit();
      }
    }
    if (issuer_warp && elect_one()) bulk_wait_read<0>();   // the slabs have been read; their writes land before the grid counts as done
  }

  // ---------------- teardown ----------------
  settle();
  if (PAIR) cluster_sync_all();   // neither CTA retires (or frees tensor memory) while the other may still signal or read it
  if (warp == 1) {
    tc_fence_after();
    if (PAIR) tmem_dealloc_pair(tmem_base, cfg::TMEM_COLS);
    else tmem_dealloc(tmem_base, cfg::TMEM_COLS);
  }
  if (counters && blockIdx.x == 0 && threadIdx.x == 0) counters[6] = globaltimer_ns();   // CTA 0 done
}

template <int BN, int EPI, bool PAIR>
phx_status launch_t(const GemmPlan& p, const GemmRope& rope, const GemmNorm& norm, int64_t M, int* err_flag, int num_sms,
                    cudaStream_t stream, std::string& err, const GemmLeftOut& out = {}) {
  // the residual epilogues are fed by TMA prefetch and keep up with two groups; the others (RoPE, GELU, norm
  // scaling) are bound by the latency of each thread's instruction stream and get four groups where a pair's
  // smaller stages leave room for the slab buffers
  // (heads of 128: two groups, each with the two slab buffers of its item)
  constexpr int NG = (PAIR && EPI != EPI_RESIDUAL && EPI != EPI_ROPE128) ? 4 : 2;
  using cfg = Cfg<BN, PAIR, NG>;
  auto kern = gemm_tcgen05_kernel<BN, EPI, PAIR, NG>;
  static OncePerDevice once;
  static std::atomic<int> pairs_of[LAUNCH_MAX_DEVICES];
  int max_pairs = 0;
  cudaLaunchConfig_t lc;
  memset(&lc, 0, sizeof(lc));
  cudaLaunchAttribute attr[2];
  lc.blockDim = dim3(gemm_threads(NG));
  lc.dynamicSmemBytes = cfg::SMEM_BYTES;
  lc.stream = stream;
  lc.attrs = attr; lc.numAttrs = 0;
  if (PAIR) {
    attr[lc.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[lc.numAttrs].val.clusterDim.x = 2; attr[lc.numAttrs].val.clusterDim.y = 1; attr[lc.numAttrs].val.clusterDim.z = 1;
    lc.numAttrs++;
  }
  const int attrs_for_query = lc.numAttrs;
  // the kernel's set-up may overlap the tail of the kernel in front of it (it waits before it reads global data);
  // PHX_PDL=0 keeps plain stream order
  static const bool pdl = !(getenv("PHX_PDL") && getenv("PHX_PDL")[0] == '0');
  if (pdl) {
    attr[lc.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[lc.numAttrs].val.programmaticStreamSerializationAllowed = 1;
    lc.numAttrs++;
  }
  int dev = 0;
  PHX_CUDA_TRY(cudaGetDevice(&dev), err);
  PHX_CUDA_TRY(once.run([&](int d) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, cfg::SMEM_BYTES);
    if (PAIR && e == cudaSuccess) {   // how many CTA pairs the device can hold at once (pairs need two SMs of one cluster-capable group)
      lc.gridDim = dim3(2 * (num_sms / 2));
      int n = 0;
      const int all_attrs = lc.numAttrs;
      lc.numAttrs = attrs_for_query;   // the occupancy query takes the cluster shape only
      e = cudaOccupancyMaxActiveClusters(&n, kern, &lc);
      lc.numAttrs = all_attrs;
      max_pairs = n < num_sms / 2 ? n : num_sms / 2;
      if (d >= 0 && d < LAUNCH_MAX_DEVICES) pairs_of[d].store(max_pairs, std::memory_order_relaxed);
    }
    return e;
  }), err);
  if (PAIR && max_pairs == 0 && dev >= 0 && dev < LAUNCH_MAX_DEVICES) max_pairs = pairs_of[dev].load(std::memory_order_relaxed);
  if (PAIR && max_pairs <= 0) { err = "gemm: the device cannot hold a CTA pair of this kernel"; return PHX_E_CUDA; }
  constexpr int TILE_M = PAIR ? 2 * BM : BM;
  const int n_tiles = (p.N + BN - 1) / BN;
  long long tiles = (M + TILE_M - 1) / TILE_M * n_tiles;
  if (leaves_out(BN, EPI, PAIR)) tiles -= (long long)out.m_tiles * (n_tiles / out.per * out.skip);
  const int slots = PAIR ? max_pairs : num_sms;
  const int units = (int)(tiles < slots ? tiles : slots);
  if (units <= 0) return PHX_OK;
  lc.gridDim = dim3(PAIR ? 2 * units : units);
  const CUtensorMap& mr = (EPI == EPI_RESIDUAL) ? p.map_r : p.map_c;
  long long Mll = M;
  int N = p.N, K = p.K;
  unsigned long long* counters = p.counters;
  PHX_CUDA_TRY(cudaLaunchKernelEx(&lc, kern, p.map_a, p.map_b, p.map_c, mr, rope, norm, Mll, N, K, err_flag, counters, out), err);
  return PHX_OK;
}

template <int BN, bool PAIR>
phx_status launch_e(const GemmPlan& p, int epilogue, const GemmRope& rp, const GemmNorm& nm, int64_t M, int* err_flag,
                    int num_sms, cudaStream_t stream, std::string& err, const GemmLeftOut& out = {}) {
  switch (epilogue) {
    case EPI_STORE: return launch_t<BN, EPI_STORE, PAIR>(p, rp, nm, M, err_flag, num_sms, stream, err);
    case EPI_RESIDUAL: return launch_t<BN, EPI_RESIDUAL, PAIR>(p, rp, nm, M, err_flag, num_sms, stream, err);
    case EPI_GELU: return launch_t<BN, EPI_GELU, PAIR>(p, rp, nm, M, err_flag, num_sms, stream, err);
    case EPI_ROPE:
      if (rp.dh == 128) {   // a single CTA's 256-column tiles leave no room for the item buffers: gemm_launch takes narrow ones
        if constexpr (PAIR || BN == 128) return launch_t<BN, EPI_ROPE128, PAIR>(p, rp, nm, M, err_flag, num_sms, stream, err, out);
        break;
      }
      return launch_t<BN, EPI_ROPE, PAIR>(p, rp, nm, M, err_flag, num_sms, stream, err);
  }
  err = "gemm: unknown epilogue";
  return PHX_E_ARG;
}

// ---- small problems: one TM x BN tile per CTA ------------------------------------------------------------------------
// For calls whose 128 x BN tiles (BN = 64 or 128) do not outnumber the SMs: one request, or a few.  Such a GEMM is a chain of
// latencies - launch, first operand bytes, k-steps, epilogue, last store - and the pair kernel above pays most of them on
// a dozen CTA pairs.  Here every tile (128 rows, or 64: low_tiles) has a CTA of its own and there is no cluster hand-shake.  Two CTAs with
// shallow rings fit an SM, so that the next kernel's set up (and, for weights that nothing rewrites, fetch the W half of their ring) under the
// tail of this one; a CTA with a deep ring has an SM to itself (deep_ring).  Each epilogue thread owns half a row's slab, has its residual / statistics loads in flight under the main loop and
// stores its 64 bytes straight to global memory.
//   warp 0 TMA producer, warp 1 MMA issuer, then BN / 32 epilogue groups of four warps: group g takes the half g & 1 of
//   64-column slab g >> 1 (RoPE: the column pairs of pass g & 1)
// Measured: a forward of one request (640 rows, 8 layers) 492 -> 431 us, 16 small requests through two layers 155 -> 143 us.
// The arithmetic per element, the order of the row statistics included, is the pair kernel's: results are the same bits.
template <int TM, int BN, bool DEEP>
struct SmallCfg {
  static constexpr int NG = BN / 32;
  static constexpr int THREADS = 64 + NG * 128;
  static constexpr int A_BYTES = TM * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + BN * BK * 2;
  static constexpr int STAGES = (DEEP ? 196608 : 98304) / STAGE_BYTES;   // ring: 4 (BN = 64) or 3 (BN = 128) k-steps, deep 8 or 6, of low tiles 12
  static constexpr int BAR_BYTES = (2 * STAGES + 2) * 8;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + (BN / 64) * TM * 4 + BAR_BYTES + 1024;   // + partial row sums, barriers, alignment
};

template <int TM, int BN, int EPI, bool DEEP>
__global__ void __launch_bounds__(SmallCfg<TM, BN, DEEP>::THREADS, 1)
gemm_small_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, bf16* C, const bf16* R,
                  GemmRope rope, GemmNorm norm, long long M, int N, int K, int early_w, int* err_flag) {
  using cfg = SmallCfg<TM, BN, DEEP>;
  constexpr bool RES = (EPI == EPI_RESIDUAL);
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t ss_base = smem_base + cfg::STAGES * cfg::STAGE_BYTES;     // [slab][TM] first halves of the row sums
  const uint32_t bars = ss_base + (BN / 64) * TM * 4;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (cfg::STAGES + s); };
  const uint32_t tfull_bar = bars + 8u * (2 * cfg::STAGES);
  const uint32_t tmem_slot = tfull_bar + 8u;
  uint32_t* tmem_slot_ptr = reinterpret_cast<uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int n_tiles = (N + BN - 1) / BN;
  const int n0 = ((int)blockIdx.x % n_tiles) * BN;
  const long long m0 = (long long)((int)blockIdx.x / n_tiles) * TM;
  const int k_blocks = (K + BK - 1) / BK;
  volatile int* verr = err_flag;

  if (threadIdx.x == 0) {
    *gave_up() = 0;
    prefetch_map(&map_a); prefetch_map(&map_b);
    for (int s = 0; s < cfg::STAGES; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    mbar_init(tfull_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tmem_slot, BN);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_d = *tmem_slot_ptr;

  auto load_w = [&](int kb, int stage) {
    const uint32_t dst = smem_base + stage * cfg::STAGE_BYTES + cfg::A_BYTES;
    for (int c = 0; c < BN / 64; ++c) tma_load_2d(dst + c * 64 * BK * 2, &map_b, full_bar(stage), kb * BK, n0 + c * 64);
  };
  const int ahead = k_blocks < cfg::STAGES ? k_blocks : cfg::STAGES;
  if (warp == 0 && early_w && elect_one()) {
    // weights that no kernel writes while forwards run need not wait for the kernel in front
    for (int kb = 0; kb < ahead; ++kb) { mbar_expect_tx(full_bar(kb), cfg::STAGE_BYTES); load_w(kb, kb); }
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0; uint32_t phase = 0;
      for (int kb = 0; kb < k_blocks; ++kb) {
        if (kb >= ahead || !early_w) {
          if (!mbar_wait(empty_bar(stage), phase ^ 1, verr)) break;
          mbar_expect_tx(full_bar(stage), cfg::STAGE_BYTES);
          load_w(kb, stage);
        }
        tma_load_2d(smem_base + stage * cfg::STAGE_BYTES, &map_a, full_bar(stage), kb * BK, (int)m0);
        if (++stage == cfg::STAGES) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc(TM, BN);
      int stage = 0; uint32_t phase = 0;
      bool ok = true;
      for (int kb = 0; kb < k_blocks; ++kb) {
        if (!mbar_wait(full_bar(stage), phase, verr)) { ok = false; break; }
        tc_fence_after();
        const uint64_t adesc = make_smem_desc(smem_base + stage * cfg::STAGE_BYTES);
        const uint64_t bdesc = make_smem_desc(smem_base + stage * cfg::STAGE_BYTES + cfg::A_BYTES);
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_bf16(tmem_d, adesc + (uint64_t)(2 * k), bdesc + (uint64_t)(2 * k), idesc, (kb | k) != 0);
        umma_commit(empty_bar(stage));
        if (++stage == cfg::STAGES) { stage = 0; phase ^= 1; }
      }
      if (ok) umma_commit(tfull_bar);
    }
  } else {
    // heads of 128 columns (BN = 128 only): the tile is one head, group p takes pass p of its four
    const bool d128 = EPI == EPI_ROPE && BN == 128 && rope.dh == 128;
    const int gidx = (warp - 2) >> 2, slab = d128 ? 0 : gidx >> 1, p = d128 ? gidx : gidx & 1;
    const int quad = warp & 3;
    // a tile of 64 rows lies in the first 16 lanes of each quadrant of tensor memory
    const bool has_row = TM == 128 || lane < 16;
    const int r = quad * (TM / 4) + (TM == 128 ? lane : lane & 15);
    const long long row = m0 + r;
    const bool in = has_row && row < M;
    const int c0 = n0 + slab * 64;                       // first column of the slab
    // two runs of 16 columns: neighbours, or (RoPE) the halves of a head that are rotated against each other
    const bool d64 = EPI == EPI_ROPE && rope.dh == 64;
    const int lo_col = (d64 || d128) ? 16 * p : 32 * p, hi_col = d128 ? 64 + 16 * p : d64 ? 32 + 16 * p : 32 * p + 16;
    // ---- everything that does not need the accumulator ----
    uint4 res[4];
    if (RES) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int col = c0 + (c < 2 ? lo_col : hi_col) + (c & 1) * 8;
        res[c] = (in && col < N) ? *reinterpret_cast<const uint4*>(R + row * N + col) : make_uint4(0u, 0u, 0u, 0u);
      }
    }
    float rstd = 1.0f;
    if (!RES && norm.ss_in != nullptr) {                 // partials summed in slot order
      float ss = 0.f;
      if (in) {
        const float* sp = norm.ss_in + row * norm.slots_in;
        if (norm.slots_in == 8) {
          const float4 a = __ldg(reinterpret_cast<const float4*>(sp)), b = __ldg(reinterpret_cast<const float4*>(sp + 4));
          ss += a.x; ss += a.y; ss += a.z; ss += a.w; ss += b.x; ss += b.y; ss += b.z; ss += b.w;
        } else {
          for (int t = 0; t < norm.slots_in; ++t) ss += __ldg(sp + t);
        }
      }
      rstd = rsqrtf(ss * norm.inv_d + norm.eps);
    }
    float4 ang[8];
    bool rotate = false;
    if (EPI == EPI_ROPE) {
      const int pos = rope_pos(rope, row + rope.row_offset, in);
      const int kind = d128 ? (c0 >> 7) % rope.group : d64 ? (c0 >> 6) % rope.group : ((c0 >> 5) + p) % rope.group;
      rotate = kind <= rope.g;
      if (rotate) {
        const float4* col = rope.angles + pos + ((d64 || d128) ? 8 * p : 0) * rope.n_pos;
#pragma unroll
        for (int t = 0; t < 8; ++t) ang[t] = __ldg(col + t * rope.n_pos);
      }
    }
    bool ok = mbar_wait(tfull_bar, 0, verr);
    ok = __all_sync(0xffffffffu, ok);
    if (ok) {
      tc_fence_after();
      const uint32_t taddr = tmem_d + ((uint32_t)(quad * 32) << 16) + slab * 64;
      uint32_t raw[32];
      tmem_ld16_nowait(taddr + lo_col, raw);
      tmem_ld16_nowait(taddr + hi_col, raw + 16);
      tmem_ld_wait();
      const float2 rstd2 = make_float2(rstd, rstd);
      uint32_t o[16];                                                 // column pairs: 8 of the low run, 8 of the high run
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        o[k] = linear_bf2(raw[2 * k], raw[2 * k + 1], rstd2);
        if (EPI == EPI_GELU) o[k] = gelu_bf2(o[k]);
      }
      if (EPI == EPI_ROPE && rotate) {
        auto rotate_all = [&](auto wide) {
#pragma unroll
          for (int t = 0; t < 8; ++t) rope_bf2<wide.value>(o[t], o[8 + t], ang[t].x, ang[t].y, ang[t].z, ang[t].w);
        };
        if (BN == 128 && d128) rotate_all(std::true_type()); else rotate_all(std::false_type());
      }
      float2 v[RES ? 16 : 1];
      if (RES) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint32_t rb[4] = {res[c].x, res[c].y, res[c].z, res[c].w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float2 x = __fadd2_rn(bf2_to_f2(o[4 * c + k]), bf2_to_f2(rb[k]));
            v[RES ? 4 * c + k : 0] = x;
            o[4 * c + k] = pack_bf2(x.x, x.y);
          }
        }
      }
      if (in) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int col = c0 + (c < 2 ? lo_col : hi_col) + (c & 1) * 8;
          if (col < N) *reinterpret_cast<uint4*>(C + row * N + col) = make_uint4(o[4 * c], o[4 * c + 1], o[4 * c + 2], o[4 * c + 3]);
        }
      }
      if (RES && norm.ss_out != nullptr) {
        // statistics of the fp32 sums, one chain over the slab's 64 columns: the second half's thread goes on from where
        // the first half's stopped
        const uint32_t slot = ss_base + (slab * TM + r) * 4;
        float ss = 0.f;
        if (p == 0) {
#pragma unroll
          for (int k = 0; k < (RES ? 16 : 1); ++k) { ss += v[k].x * v[k].x; ss += v[k].y * v[k].y; }
          if (has_row) asm volatile("st.shared.f32 [%0], %1;" ::"r"(slot), "f"(ss) : "memory");
        }
        asm volatile("bar.sync %0, 256;" ::"r"(1 + slab) : "memory");
        if (p == 1) {
          asm volatile("ld.shared.f32 %0, [%1];" : "=f"(ss) : "r"(slot) : "memory");
#pragma unroll
          for (int k = 0; k < (RES ? 16 : 1); ++k) { ss += v[k].x * v[k].x; ss += v[k].y * v[k].y; }
          if (in && c0 < N) norm.ss_out[row * (long long)(N / SLAB_COLS) + c0 / SLAB_COLS] = ss;
        }
      }
    } else if (RES && norm.ss_out != nullptr) {
      asm volatile("bar.sync %0, 256;" ::"r"(1 + slab) : "memory");    // a warp that gave up never leaves the others parked
    }
  }

  // ---------------- teardown ----------------
  settle();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_d, BN);
  }
}

template <int TM, int BN, int EPI, bool DEEP>
phx_status launch_small_d(const GemmPlan& p, const CUtensorMap& map_b64, bf16* C, const bf16* R, const GemmRope& rope,
                          const GemmNorm& norm, int64_t M, int* err_flag, cudaStream_t stream, std::string& err) {
  using cfg = SmallCfg<TM, BN, DEEP>;
  auto kern = gemm_small_kernel<TM, BN, EPI, DEEP>;
  static SmemLimit limit;
  PHX_CUDA_TRY(limit.raise(kern, cfg::SMEM_BYTES), err);
  cudaLaunchConfig_t lc;
  memset(&lc, 0, sizeof(lc));
  cudaLaunchAttribute attr[1];
  static const bool pdl = !(getenv("PHX_PDL") && getenv("PHX_PDL")[0] == '0');
  if (pdl) {
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = attr; lc.numAttrs = 1;
  }
  lc.gridDim = dim3((unsigned)(((M + TM - 1) / TM) * ((p.N + BN - 1) / BN)));
  lc.blockDim = dim3(cfg::THREADS);
  lc.dynamicSmemBytes = cfg::SMEM_BYTES;
  lc.stream = stream;
  long long Mll = M;
  int N = p.N, K = p.K, early = p.w_stable ? 1 : 0;
  PHX_CUDA_TRY(cudaLaunchKernelEx(&lc, kern, TM == 64 ? p.map_a_low : p.map_a, map_b64, C, R, rope, norm, Mll, N, K, early, err_flag), err);
  return PHX_OK;
}
// A deep ring has its SM for itself; a shallow one leaves room for a CTA of the kernel behind.  Deep from K = 1024 on, and from 512 where the
// kernel behind finds SMs free anyway or has few CTAs.  Forwards of 1 to 16 requests on the device, us, shallow / deep from K = 1024 / from 512 /
// as here: eight layers of D = 512 and 106 rows a request, one 248 / 222 / 216 / 216, three 242 / 219 / 213 / 213, 118 rows, 16 requests 383 / 336 /
// 324 / 324; 640 rows, one request 276 / 251 / 254 / 250; D = 1024, two layers of 275 rows, six requests 210 / 168.  (The shallow figures are of
// kernels that still read the error flag as their last act, 0.5 us each - see gave_up.)
bool deep_ring(int K, int epilogue, long long tiles, int num_sms) {
  return K >= 1024 || (K >= 512 && (epilogue == EPI_RESIDUAL || 3 * tiles <= 2 * num_sms));
}
// Tiles of 64 rows where those find an SM each: a k-step is paced by the rows its copies bring in (1.6 to 1.9 cycles a row of 128 bytes,
// however deep the ring), 128 in place of 192.  The forwards above: one request of 172 rows 216 -> 203 us, three of 106 213 -> 197, one of 640
// 250 -> 240 (from K = 1024 on alone: 213, 206, 244).
bool low_tiles(int64_t M, int N, int K, int num_sms) { return K >= 512 && ((M + 63) / 64) * ((N + 63) / 64) <= num_sms; }
template <int BN, int EPI>
phx_status launch_small_t(const GemmPlan& p, const CUtensorMap& map_b64, bf16* C, const bf16* R, const GemmRope& rope,
                          const GemmNorm& norm, int64_t M, int num_sms, int* err_flag, cudaStream_t stream, std::string& err) {
  if (BN == 64 && low_tiles(M, p.N, p.K, num_sms)) {
    dispatch_note(DK_FORM_GEMM_LOW);
    return launch_small_d<64, 64, EPI, true>(p, map_b64, C, R, rope, norm, M, err_flag, stream, err);
  }
  const long long tiles = ((M + BM - 1) / BM) * ((p.N + BN - 1) / BN);
  if (!deep_ring(p.K, EPI, tiles, num_sms)) return launch_small_d<BM, BN, EPI, false>(p, map_b64, C, R, rope, norm, M, err_flag, stream, err);
  dispatch_note(DK_FORM_GEMM_DEEP);
  return launch_small_d<BM, BN, EPI, true>(p, map_b64, C, R, rope, norm, M, err_flag, stream, err);
}
template <int BN>
phx_status launch_small(const GemmPlan& p, const CUtensorMap& map_b64, bf16* C, const bf16* R, int epilogue, const GemmRope& rp,
                        const GemmNorm& nm, int64_t M, int num_sms, int* err_flag, cudaStream_t stream, std::string& err) {
  switch (epilogue) {
    case EPI_STORE: return launch_small_t<BN, EPI_STORE>(p, map_b64, C, R, rp, nm, M, num_sms, err_flag, stream, err);
    case EPI_RESIDUAL: return launch_small_t<BN, EPI_RESIDUAL>(p, map_b64, C, R, rp, nm, M, num_sms, err_flag, stream, err);
    case EPI_GELU: return launch_small_t<BN, EPI_GELU>(p, map_b64, C, R, rp, nm, M, num_sms, err_flag, stream, err);
    case EPI_ROPE: return launch_small_t<BN, EPI_ROPE>(p, map_b64, C, R, rp, nm, M, num_sms, err_flag, stream, err);
  }
  err = "gemm: unknown epilogue";
  return PHX_E_ARG;
}

// ---- SIMT cross-check GEMM --------------------------------------------------------------------------
template <int EPI>
__global__ void gemm_simt_kernel(const bf16* __restrict__ A, const bf16* __restrict__ Wt, bf16* C,
                                 const bf16* R, long long M, int N, int K) {
  __shared__ float sa[32][33];
  __shared__ float sb[32][33];
  const int tx = threadIdx.x, ty = threadIdx.y;
  const long long row = (long long)blockIdx.y * 32 + ty;
  const int col = blockIdx.x * 32 + tx;
  float acc = 0.f;
  for (int k0 = 0; k0 < K; k0 += 32) {
    sa[ty][tx] = (row < M && k0 + tx < K) ? bf2f(A[row * K + k0 + tx]) : 0.f;
    const int wr = blockIdx.x * 32 + ty;
    sb[ty][tx] = (wr < N && k0 + tx < K) ? bf2f(Wt[(long long)wr * K + k0 + tx]) : 0.f;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 32; ++k) acc += sa[ty][k] * sb[tx][k];
    __syncthreads();
  }
  if (row < M && col < N) {
    float v = round_bf(acc);
    if (EPI == EPI_RESIDUAL) v += bf2f(R[row * N + col]);
    else if (EPI == EPI_GELU) v = gelu_tanh_f(v);
    C[row * N + col] = f2bf(v);
  }
}

}  // namespace

phx_status gemm_plan_create(GemmPlan* plan, const bf16* A, const bf16* Wt, int64_t rows_max, int N, int K,
                            bool narrow_tiles, std::string& err, int pair) {
  if (N % 8 != 0 || K % 8 != 0 || N <= 0 || K <= 0 || rows_max <= 0) {
    err = "gemm: N and K must be positive multiples of 8";
    return PHX_E_ARG;
  }
  plan->A = A; plan->Wt = Wt; plan->rows_max = rows_max; plan->a_rows = rows_max; plan->N = N; plan->K = K;
  // 128-wide tiles leave room for six output slabs: deep residual prefetch for the HBM-bound short-K GEMMs
  { const char* t = getenv("PHX_GEMM_TILES");   // diagnostics: wide | narrow overrides the caller's choice
    if (t && strcmp(t, "wide") == 0) narrow_tiles = false;
    if (t && strcmp(t, "narrow") == 0) narrow_tiles = true; }
  // CTA pairs, and one tile per CTA for few tiles, by default; for comparison PHX_GEMM=pair takes pairs at every size and
  // PHX_GEMM=cta1 the persistent kernel with single CTAs
  const char* mode = getenv("PHX_GEMM");
  plan->pair = pair >= 0 ? (pair != 0) : !(mode && strcmp(mode, "cta1") == 0);
  plan->small_ok = plan->pair && !(mode && strcmp(mode, "pair") == 0);
  // a pair fills 128 + BN/2 operand rows per CTA and k-step: the wide tile is the cheaper one per FLOP there
  // (out-projection, N = K = 512: 0.100 ms wide against 0.146 ms narrow)
  if (plan->pair && !(getenv("PHX_GEMM_TILES") && strcmp(getenv("PHX_GEMM_TILES"), "narrow") == 0)) narrow_tiles = false;
  plan->BN = (N % 256 == 0 && !narrow_tiles) ? 256 : 128;
  plan->low_A = nullptr;
  phx_status s = make_map(&plan->map_a, A, rows_max, K, BM, err);
  if (s != PHX_OK) return s;
  s = make_map(&plan->map_b, Wt, N, K, plan->pair ? plan->BN / 2 : plan->BN, err);
  if (s != PHX_OK) return s;
  if (plan->BN == 256) {   // the narrow tiles' W box: one tile per CTA, and single CTAs in gemm_launch's latency regime
    s = make_map(&plan->map_b_narrow, Wt, N, K, plan->pair ? 64 : 128, err);
    if (s != PHX_OK) return s;
  }
  plan->ready = true;
  return PHX_OK;
}

phx_status gemm_launch(GemmPlan& p, const bf16* A, bf16* C, const bf16* R, int64_t M, int epilogue, const GemmRope* rope,
                       const GemmNorm* norm, int* err_flag, int num_sms, cudaStream_t stream, std::string& err, int64_t kv_rows) {
  if (!p.ready || M > p.rows_max) { err = "gemm: plan not ready or M exceeds plan rows"; return PHX_E_ARG; }
  if (epilogue == EPI_RESIDUAL && R == nullptr) { err = "gemm: residual epilogue needs R"; return PHX_E_ARG; }
  GemmRope rp;
  GemmLeftOut out;
  memset(&rp, 0, sizeof(rp));
  GemmNorm nm;
  memset(&nm, 0, sizeof(nm));
  if (norm) nm = *norm;
  if (nm.ss_out && (epilogue != EPI_RESIDUAL || p.N % SLAB_COLS != 0)) { err = "gemm: row statistics are produced by the residual epilogue only"; return PHX_E_ARG; }
  if (A != p.A || (p.a_rows != M && p.a_rows != p.rows_max)) {
    // the activation buffer moved (double-buffered residual stream, or a block of rows inside it): re-encode its
    // map over exactly the M rows of this call, so that no tile reads past them
    phx_status s = make_map(&p.map_a, A, M, p.K, BM, err);
    if (s != PHX_OK) return s;
    p.A = A; p.a_rows = M;
  }
  if (epilogue == EPI_ROPE) {
    if (!rope || (rope->dh != 32 && rope->dh != 64 && rope->dh != 128) || rope->T <= 0 || p.N % rope->dh != 0) {
      err = "gemm: the RoPE epilogue needs head dim 32, 64 or 128";
      return PHX_E_ARG;
    }
    rp = *rope;
    // pairs of CTAs on 256 columns and heads of 128: the q heads of a group that fill whole tiles (where four share a key head, four of the
    // twelve column tiles of 16 heads are left: 8 x (1022 + 64) rows 42.4 -> 23.1 us)
    const int width = rp.group * rp.dh, q_tiles = rp.g * rp.dh / 256;
    if (rp.dh == 128 && p.pair && p.BN == 256 && kv_rows > 0 && width % 256 == 0 && p.N % width == 0 && q_tiles > 0) {
      out.m_tiles = (int)(kv_rows / (2 * BM)); out.per = width / 256; out.skip = q_tiles;
    }
  }
  // output / residual maps are [M, N] with 128 x 64 boxes; rows past M are clipped by the TMA unit
  if (p.c_ptr != C || p.c_rows != M) {
    phx_status s = make_map(&p.map_c, C, M, p.N, BM, err);
    if (s != PHX_OK) return s;
    p.c_ptr = C; p.c_rows = M;
  }
  if (epilogue == EPI_RESIDUAL && (p.r_ptr != R || p.r_rows != M)) {
    phx_status s = make_map(&p.map_r, R, M, p.N, BM, err);
    if (s != PHX_OK) return s;
    p.r_ptr = R; p.r_rows = M;
  }
  if (p.small_ok) {
    // Few tiles: one 128 x 64 (else 128 x 128) tile per CTA while they do not outnumber the SMs.  Beyond that a CTA would have
    // a second tile with nothing overlapped, and the pair kernel's wide tiles fetch fewer operand bytes.  Pair time over this
    // kernel's, each alone: 8-40 tiles of 64 columns (128 and 640 rows, N = 512) 1.28-1.30; 144-148 tiles of 128: N = 2048 1.11-1.15,
    // N = 1024 1.12-1.18 up to K = 4096, N = 512 1.02 at K = 512 and 1.11-1.13 at 2048 and 4096, N = 128 0.97-1.00.  Three-layer
    // forwards: D = 512, 640 rows a request 1.31 with one, 1.04 with four, 0.99 with eight (only the last layer's narrow ones are few).
    const CUtensorMap& map_b64 = p.BN == 256 ? p.map_b_narrow : p.map_b;   // boxes of 64 W rows, either way
    const long long mt = (M + BM - 1) / BM, t64 = mt * ((p.N + 63) / 64), t128 = mt * ((p.N + 127) / 128);
    if (t64 <= num_sms && !(epilogue == EPI_ROPE && rp.dh == 128)) {
      if (low_tiles(M, p.N, p.K, num_sms) && (p.low_A != p.A || p.low_rows != p.a_rows)) {
        phx_status s = make_map(&p.map_a_low, A, p.a_rows, p.K, 64, err);
        if (s != PHX_OK) return s;
        p.low_A = p.A; p.low_rows = p.a_rows;
      }
      dispatch_note(DK_GEMM_SMALL);
      return launch_small<64>(p, map_b64, C, R, epilogue, rp, nm, M, num_sms, err_flag, stream, err);
    }
    if (t128 <= num_sms) { dispatch_note(DK_GEMM_SMALL); return launch_small<128>(p, map_b64, C, R, epilogue, rp, nm, M, num_sms, err_flag, stream, err); }
  }
  if (p.BN == 256) {
    if (!p.pair) {
      // single CTAs, latency regime: when even the 128-column tiles leave SMs idle, take them - the call's time is one tile's
      // time (a pair's call of that size has gone to one tile per CTA above).  Heads of 128 always: a single CTA's 256-column
      // tiles leave no room for the buffers of a rotated head.
      const long long narrow_tiles = ((M + BM - 1) / BM) * ((p.N + 127) / 128);
      static const bool allow = !(getenv("PHX_GEMM_TILES") && strcmp(getenv("PHX_GEMM_TILES"), "wide") == 0);
      if ((epilogue == EPI_ROPE && rp.dh == 128) || (allow && narrow_tiles <= num_sms)) {
        dispatch_note(DK_GEMM_CTA128);
        GemmPlan q = p;
        q.map_b = p.map_b_narrow; q.BN = 128;
        return launch_e<128, false>(q, epilogue, rp, nm, M, err_flag, num_sms, stream, err);
      }
    }
    dispatch_note(p.pair ? DK_GEMM_PAIR256 : DK_GEMM_CTA256);
    if (out.m_tiles > 0) dispatch_note(DK_FORM_GEMM_KV);
    return p.pair ? launch_e<256, true>(p, epilogue, rp, nm, M, err_flag, num_sms, stream, err, out)
                  : launch_e<256, false>(p, epilogue, rp, nm, M, err_flag, num_sms, stream, err);
  }
  dispatch_note(p.pair ? DK_GEMM_PAIR128 : DK_GEMM_CTA128);
  return p.pair ? launch_e<128, true>(p, epilogue, rp, nm, M, err_flag, num_sms, stream, err)
                : launch_e<128, false>(p, epilogue, rp, nm, M, err_flag, num_sms, stream, err);
}

namespace {
__global__ void wait_selftest_kernel(int* err_flag) {
  __shared__ __align__(8) unsigned long long bar;
  const uint32_t b = smem_u32(&bar);
  mbar_init(b, 1);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  mbar_wait(b, 0, err_flag);   // nothing arrives: returns false once the limit has passed
}
}  // namespace

phx_status wait_selftest_launch(int* err_flag, cudaStream_t stream, std::string& err) {
  wait_selftest_kernel<<<1, 1, 0, stream>>>(err_flag);
  PHX_CUDA_TRY(cudaGetLastError(), err);
  return PHX_OK;
}

phx_status gemm_simt_launch(const bf16* A, const bf16* Wt, bf16* C, const bf16* R, int64_t M, int N, int K,
                            int epilogue, cudaStream_t stream, std::string& err) {
  dispatch_note(DK_GEMM_SIMT);
  dim3 block(32, 32);
  dim3 grid((N + 31) / 32, (unsigned)((M + 31) / 32));
  if (grid.y > 65535) {
    // split rows so gridDim.y stays legal
    const int64_t chunk = 65535LL * 32;
    for (int64_t m0 = 0; m0 < M; m0 += chunk) {
      int64_t mm = (M - m0 < chunk) ? (M - m0) : chunk;
      phx_status s = gemm_simt_launch(A + m0 * K, Wt, C + m0 * N, R ? R + m0 * N : nullptr, mm, N, K, epilogue,
                                      stream, err);
      if (s != PHX_OK) return s;
    }
    return PHX_OK;
  }
  switch (epilogue) {
    case EPI_STORE: gemm_simt_kernel<EPI_STORE><<<grid, block, 0, stream>>>(A, Wt, C, R, M, N, K); break;
    case EPI_RESIDUAL: gemm_simt_kernel<EPI_RESIDUAL><<<grid, block, 0, stream>>>(A, Wt, C, R, M, N, K); break;
    case EPI_GELU: gemm_simt_kernel<EPI_GELU><<<grid, block, 0, stream>>>(A, Wt, C, R, M, N, K); break;
    default: err = "gemm: unknown epilogue"; return PHX_E_ARG;
  }
  PHX_CUDA_TRY(cudaGetLastError(), err);
  return PHX_OK;
}

}  // namespace phx
