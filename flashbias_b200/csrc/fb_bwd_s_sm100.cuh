// Backward FlashBias attention for sm_100a, two-stream key-major form: head_dim up to 64; factor operands, the ALiBi producer or
// neither; no mask tensor.
//
// One CTA (512 threads) per tile of 128 keys of one (batch, head).  The logits are computed transposed,
//     S^T = [Ks|Kb].[Q|Qb]^T        dP^T = V.dO^T          (lane = key, column = query)
// so that P^T and dS^T are the A operands of dV += P^T.dO and dK|dkb += dS^T.[Q|Qb] and stay in TENSOR MEMORY; only dS^T
// also goes to shared memory, as the transposed A operand of dQ|dQb = dS.[K|Kc].  The two compute warpgroups are two streams:
// each has its own half tiles (64 queries), its own S^T and dP^T and its own barriers, so that one stream's exponentials run
// under the other's loads, products and stores.  They meet only where they use the 32 columns of dS^T in turn (and, where
// shared memory holds one dS^T tile, where stream 0 waits for the dQ product of both halves).
//   warps 0-3, 4-7  stream 0 / 1: half tiles 0, 2, 4, ... / 1, 3, 5, ... of 64 queries
//   warps 8-11      drain warpgroup: the dQ|dQb tile of 128 queries goes from tensor memory through a staging tile into the
//                   fp32 accumulators in global memory by bulk reductions
//   warp 12         TMA producer: resident tiles once, then Q|Qb|dO half tiles through a ring; its lanes also write the
//                   stage's table of row statistics (-lse * log2 e with the ALiBi term's share, -delta)
//   warps 13-15     MMA issuers (one thread each): S^T and dP^T; dV; dK|dkb and dQ|dQb
//
// The threads read S^T and dP^T from tensor memory with 16x256b loads: lane t of a warp holds keys t/4 + 8k (k = 0..3) and
// queries 8j + 2(t%4) + {0,1} (j = 0..7) of its 32 keys x 64 queries.  A thread so needs the statistics of 16 queries
// only (from a small shared-memory table), and the row sums of dS over a group of 32 keys -- the warp's keys -- which the
// exact dq_bias needs (see drain_dq_bias) are three additions and three halving exchanges between lanes; with one key per
// lane they are a 32-lane reduction of every column.  The fragments are stored with 16x128b stores (tensor memory) and
// stmatrix (shared memory).
//
// What bounds it: the latency of a half tile's own chain of steps, about 2900 clk a query tile at head_dim 32 (exponentials 1050,
// shared-memory traffic 1900, issue slots 1530).  What brought it there: dP^T and S^T of the next half tile issued as soon as the
// threads have read this one's (dS^T in columns of its own: behind the dK product they came 1400 clk later); satisfied waits
// tested ahead of use (85 to 290 clk each); the next S^T loaded under the row sums.  Sixteen compute warps of 32 x 32 took
// the same time (8000 instead of 6100 instructions a tile).
// Backward kernel, query-major form / this one, us: B2 H8 S32768 D64 R5 16300 / 13900, B1 H16 S1536 D32 R32 112 / 68, B1 H16
// S743 D24 R8 20.5 / 18.5, B1 H50 S8192 D32 R2 causal 1277 / 1180.
#pragma once

#include "fb_bwd_sm100.cuh"

namespace fb {

constexpr int kBwdSThreads = 512;  // 8 compute warps, 4 drain warps, 4 that load and issue

template <int D, int RP, int RC_, int NQ>
struct BwdSCfg {
  static constexpr bool STAGED = true;
  static constexpr int HALF = 64;  // queries of a half tile
  static constexpr int RPX = RP ? RP : 16;
  static constexpr int RC = RC_, RCX = RC ? RC : 16;  // centred k-side factor: (hi, lo) pair
  static constexpr int KT = tile_bytes(D), RT = RP ? tile_bytes(RPX) : 0;
  // [K | Kc] is one MN-major operand: Kc in column blocks as wide as K's
  static constexpr int KC_BLOCKS = RC ? (RC + D - 1) / D : 0;
  // resident: K, (hi, lo) of k*scale when the scale is not a power of two, Kb, V
  static constexpr int OFF_K = 0, OFF_KC = KT, OFF_KS = OFF_KC + KC_BLOCKS * KT, OFF_V = OFF_KS + (NQ == 2 ? 2 * KT : 0),
                       OFF_KB = OFF_V + KT, KV_BYTES = OFF_KB + RT, KV_TMA_BYTES = KV_BYTES - (NQ == 2 ? KT : 0);  // (lo is computed)
  // one stage of the ring: Q, dO, Qb of 64 queries
  static constexpr int OFF_DO = tile_bytes(D, HALF), OFF_QB = 2 * OFF_DO;
  static constexpr int STAGE_BYTES = OFF_QB + (RP ? tile_bytes(RPX, HALF) : 0);
  static constexpr int DS_HALF = tile_bytes(HALF);  // dS^T of a half tile: [128 keys][64 queries]
  // staging tile of dQ and dq_bias
  static constexpr int STG_DQ = 128 * D * 4, STG_BYTES = STG_DQ + 128 * (RC / 2) * 4;
  static constexpr int STAT = 2 * HALF * 4, STAT_BYTES = 6 * STAT;  // per stage (-lse, -delta) x 64 queries
  static constexpr int ROWSUM_BYTES = RP ? 4 * 4 * 128 * 4 : 0;
  static constexpr int KBC_BYTES = RC / 2 * 4 * 4;
  static constexpr int TAIL = 512 + STAT_BYTES + ROWSUM_BYTES + KBC_BYTES + 1024;
  static constexpr int LIM = 227 * 1024;
  static constexpr int fixed_for(int ds_bufs) { return KV_BYTES + ds_bufs * 2 * DS_HALF + STG_BYTES + TAIL; }
  // two dS^T tiles, used in turn, where four stages fit beside them: no thread then waits for the dQ product of the last tile
  static constexpr int DS_BUFS = fixed_for(2) + 4 * STAGE_BYTES <= LIM ? 2 : 1, DS_TILE = 2 * DS_HALF;
  static constexpr int FIXED = fixed_for(DS_BUFS);
  static constexpr int NSTAGE_FIT = (LIM - FIXED) / STAGE_BYTES;
  static constexpr int NSTAGE = NSTAGE_FIT > 6 ? 6 : NSTAGE_FIT;
  static constexpr int OFF_STAGE = KV_BYTES;
  static constexpr int OFF_DS = OFF_STAGE + NSTAGE * STAGE_BYTES;
  static constexpr int OFF_STG = OFF_DS + DS_BUFS * DS_TILE;
  static constexpr int OFF_BAR = OFF_STG + STG_BYTES;
  static constexpr int OFF_STAT = OFF_BAR + 512;
  static constexpr int OFF_ROWSUM = OFF_STAT + STAT_BYTES;  // 4 x 4 x 128 floats: dS row sums per 32-key group
  static constexpr int OFF_KBC = OFF_ROWSUM + ROWSUM_BYTES;
  static constexpr int SMEM = FIXED + NSTAGE * STAGE_BYTES;
  // tensor memory: per stream S^T and dP^T (64 fp32 columns each), the accumulators, 32 columns of dS^T that the streams use in
  // turn, and P^T: 32 columns per stream, or in the place of S^T
  static constexpr int T_S = 0, T_DP = 64, T_STREAM = 128, T_DV = 256, T_DK = T_DV + D, T_DKB = T_DK + D, T_DQ = T_DKB + RP,
                       T_DQB = T_DQ + D, T_DS = T_DQB + RC, T_END = T_DS + 32;
  static constexpr bool SEP_P = T_END + 64 <= 512;
  static constexpr int T_P = SEP_P ? T_END : T_S, P_STRIDE = SEP_P ? 32 : T_STREAM;
  static constexpr bool FITS = NSTAGE >= 3 && T_END <= 512;
};

// Fragments of 16 lanes: regs 4j + 2i + e <-> lane t/4 + 8i, column 8j + 2(t%4) + e
__device__ __forceinline__ void tmem_ld_16x256b_x8(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x8.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
// regs 2j + i <-> lane t/4 + 8i, 32-bit column 4j + t%4
__device__ __forceinline__ void tmem_st_16x128b_x8(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
// four 8x8 matrices of 16-bit values; lane l gives the address of row l%8 of matrix l/8
__device__ __forceinline__ void stmatrix_x4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d)
               : "memory");
}
// A wait on a phase that was tested some time ago: a satisfied wait alone is 85 clocks on an idle SM and 150 to 300 on a busy
// one, and the test's latency is hidden by what stands between.
__device__ __forceinline__ void mbar_wait_tested(bool done, uint32_t bar, uint32_t parity, uint32_t abort_flag) {
  if (!done) mbar_wait(bar, parity, abort_flag);
  __syncwarp();
}
__device__ __forceinline__ uint64_t ld_shared_f2(uint32_t addr) {
  float x, y;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(x), "=f"(y) : "r"(addr) : "memory");
  return f2(x, y);
}
__device__ __forceinline__ void st_shared_v2f(uint32_t addr, float x, float y) {
  asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(x), "f"(y) : "memory");
}

template <typename T, int D, int RP, int RC, int NQ, int MODE>
__global__ void __launch_bounds__(kBwdSThreads, 1)
bwd_s_sm100_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                   const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                   const __grid_constant__ CUtensorMap tmQb, const __grid_constant__ CUtensorMap tmKb,
                   const __grid_constant__ CUtensorMap tmKc, const BwdArgs a) {
  using Cfg = BwdSCfg<D, RP, RC, NQ>;
  constexpr int RPX = Cfg::RPX, HALF = Cfg::HALF, NST = Cfg::NSTAGE;
  constexpr bool kBf16 = std::is_same<T, __nv_bfloat16>::value;
  constexpr float kLog2e = 1.4426950408889634f;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t sbase = smem_u32(smem);
  const uint32_t sK = sbase + Cfg::OFF_K, sKc = sbase + Cfg::OFF_KC, sKs = sbase + Cfg::OFF_KS, sV = sbase + Cfg::OFF_V,
                 sKb = sbase + Cfg::OFF_KB, sStage = sbase + Cfg::OFF_STAGE, sDS = sbase + Cfg::OFF_DS,
                 sStg = sbase + Cfg::OFF_STG, sStat = sbase + Cfg::OFF_STAT;
  const uint32_t bar0 = sbase + Cfg::OFF_BAR;
  // barriers; those of two slots belong to a stream each
  const uint32_t kv_full = bar0, all_done = bar0 + 8, dq_full = bar0 + 16, dq_drained = bar0 + 24, s_full = bar0 + 32,
                 dp_full = bar0 + 48, p_ready = bar0 + 64, ds_ready = bar0 + 80, dv_done = bar0 + 96, dk_done = bar0 + 112,
                 full = bar0 + 128 /*6*/, free_ = bar0 + 176 /*6*/, rs_ready = bar0 + 256 /*4*/, ks_ready = bar0 + 288;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + Cfg::OFF_BAR + 232);
  const uint32_t abort_flag = sbase + Cfg::OFF_BAR + 236;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int BH = a.B * a.H;
  int kt, bh;
  if (a.causal) {  // key tile 0 sees the most query tiles: heaviest first
    kt = (int)(blockIdx.x / BH);
    bh = (int)(blockIdx.x % BH);
  } else {
    kt = (int)(blockIdx.x % a.nk_tiles);
    bh = (int)(blockIdx.x / a.nk_tiles);
  }
  const int b = bh / a.H, h = bh % a.H;
  const int k0 = kt * 128;
  const int i_begin = a.causal ? kt : 0;       // first query tile (128 rows) with a row >= k0
  const int n_it = a.nq_tiles - i_begin;       // may be <= 0 when Sq < Sk under causal masking
  const int n_half = 2 * n_it;

  // producer thread only: one half tile of queries
  auto load_half = [&](int x) {
    const int st = x % NST;
    const uint32_t base = sStage + st * Cfg::STAGE_BYTES, bar = full + 8 * st;
    const int q0 = i_begin * 128 + x * HALF;
    mbar_expect_tx(bar, Cfg::STAGE_BYTES);
    tma_tile_bwd<D, HALF>(base, &tmQ, bar, q0, h, b);
    if (RP) tma_tile_bwd<RPX, HALF>(base + Cfg::OFF_QB, &tmQb, bar, q0, a.hq_bcast ? 0 : h, a.bq_bcast ? 0 : b);
    tma_tile_bwd<D, HALF>(base + Cfg::OFF_DO, &tmDO, bar, q0, h, b);
  };

  if (warp == 12) {
    if (lane == 0) {
      st_shared_flag(abort_flag, 0u);
      mbar_init(kv_full, 1);
      mbar_init(ks_ready, 4);  // the drain warps have split k*scale
      mbar_init(all_done, 2);  // the threads that issue into dV and into dK|dkb
      mbar_init(dq_full, 1);
      mbar_init(dq_drained, 4);  // the drain warps
      for (int i = 0; i < 2; ++i) {
        mbar_init(s_full + 8 * i, 1);
        mbar_init(dp_full + 8 * i, 1);
        mbar_init(p_ready + 8 * i, 4);   // the stream's warps
        mbar_init(ds_ready + 8 * i, 4);  // likewise
        mbar_init(dv_done + 8 * i, 1);
        mbar_init(dk_done + 8 * i, 1);
      }
      // all compute warps: the row sums of a query tile; one barrier per table, as the streams may be past later tiles' before the
      // drain waits for this one's
      for (int i = 0; i < 4; ++i) mbar_init(rs_ready + 8 * i, 8);
      for (int i = 0; i < NST; ++i) {
        mbar_init(full + 8 * i, 2);   // the loads, and the statistics that the producer warp writes
        mbar_init(free_ + 8 * i, 2);  // the dV and the dK|dkb products of the half tile, its last readers
      }
      mbar_fence_init();
      grid_dep_wait();
      if (n_it > 0) {
        const int hk = a.hk_bcast ? 0 : h, bk = a.bk_bcast ? 0 : b;
        mbar_expect_tx(kv_full, Cfg::KV_TMA_BYTES);
        if (NQ == 2) tma_tile_bwd<D>(sKs, &tmK, kv_full, k0, h, b);  // (split in place)
        if (RP) tma_tile_bwd<RPX>(sKb, &tmKb, kv_full, k0, hk, bk);
        tma_tile_bwd<D>(sV, &tmV, kv_full, k0, h, b);
        tma_tile_bwd<D>(sK, &tmK, kv_full, k0, h, b);
        load_half(0);
        for (int i = 0; i < Cfg::KC_BLOCKS; ++i) tma_tile_bwd<D>(sKc + i * Cfg::KT, &tmKc, kv_full, k0, hk, bk, i * D);
        for (int x = 1; x < NST && x < n_half; ++x) load_half(x);
      }
    }
  } else if (warp == 13) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  grid_dep_wait();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;

  if (warp >= 12) {
    setmaxnreg_dec<64>();
    if (warp == 12) {
      // ------------------------------------------------------------------ TMA producer, row statistics
      // Raw loads one half tile ahead.  Queries beyond Sq and queries that saw no key: probabilities exactly zero.
      float lse_raw[2], dlt[2];
      auto load_stats = [&](int x) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int g = i_begin * 128 + x * HALF + lane + 32 * e;
          lse_raw[e] = -INFINITY;
          dlt[e] = 0.f;
          if (g < a.Sq) {
            asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(lse_raw[e]) : "l"(a.lse + (int64_t)bh * a.lse_stride_bh + g));
            asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(dlt[e]) : "l"(a.delta + (int64_t)bh * a.lse_stride_bh + g));
          }
        }
      };
      const float slope2 = MODE == BWD_ALIBI ? __ldg(a.alibi_slopes + h) * kLog2e : 0.f;
      if (n_it > 0) load_stats(0);
#pragma unroll 1
      for (int x = 0; x < n_half; ++x) {
        const int st = x % NST;
        if (x >= NST) {
          // (the whole warp waits here, and leaves together: each lane polls for itself, and may see another end of an expired wait)
          if (!__all_sync(0xffffffffu, mbar_wait(free_ + 8 * st, (x / NST - 1) & 1, abort_flag))) break;
          if (elect_one()) load_half(x);
          __syncwarp();
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          float nl = -INFINITY;
          if (lse_raw[e] != -INFINITY) {
            nl = -lse_raw[e] * kLog2e;
            // The term slope * (key - query) is counted from the half tile's first query on either side (the keys' share: ak).
            // Counted from query 0, two large numbers would cancel near the diagonal, and P lose a bit for every doubling of
            // the position (fp16, slope 0.9, S 65536: gradients 1.9e-3 from 64 bits instead of 3e-4).
            if (MODE == BWD_ALIBI) nl -= slope2 * (float)(lane + 32 * e);
          }
          const uint32_t at = sStat + st * Cfg::STAT + (lane + 32 * e) * 4;
          st_shared_f32(at, nl);
          st_shared_f32(at + HALF * 4, -dlt[e]);
        }
        load_stats(x + 1);
        mbar_arrive_warp(full + 8 * st);
      }
    } else if (n_it > 0 && elect_one()) {
      constexpr uint32_t idS = instr_desc(kBf16, false, false, 128, HALF);       // S^T, dP^T: both operands K-major
      constexpr uint32_t idTD = instr_desc(kBf16, false, true, 128, D);          // dV, dK: A in TMEM, B MN-major
      constexpr uint32_t idTR = instr_desc(kBf16, false, true, 128, RPX);        // dkb
      constexpr uint32_t idQ = instr_desc(kBf16, true, true, 128, D + Cfg::RC);  // dQ|dQb: A = dS (transposed tile)
      if (warp == 13) {
        // ------------------------------------------------------------------ S^T, dP^T
        const DescBase kQ = kmajor_base<D, HALF>(sStage), kQb = kmajor_base<RPX, HALF>(sStage + Cfg::OFF_QB),
                       kK = kmajor_base<D>(NQ == 2 ? sKs : sK), kKb = kmajor_base<RPX>(sKb), kV = kmajor_base<D>(sV),
                       kDO = kmajor_base<D, HALF>(sStage + Cfg::OFF_DO);
        mbar_wait(kv_full, 0, abort_flag);
        if (NQ == 2) mbar_wait(ks_ready, 0, abort_flag);
#pragma unroll 1
        for (int x = 0; x < n_half; ++x) {
          const int w = x & 1, n = x >> 1, st = x % NST;
          const uint32_t so = st * Cfg::STAGE_BYTES, tS = tmem + w * Cfg::T_STREAM + Cfg::T_S;
          mbar_wait(full + 8 * st, (x / NST) & 1, abort_flag);
          // the threads have read the previous S^T and dP^T (or, where P^T lies in the place of S^T, the dV product has read that)
          if (n > 0) mbar_wait((Cfg::SEP_P ? p_ready : dv_done) + 8 * w, (n - 1) & 1, abort_flag);
          tc_fence_after_sync();
          // bias products first, into the empty accumulator (large factor terms cancel among themselves)
          if (RP) {
#pragma unroll
            for (int s = 0; s < RPX / 16; ++s)
              umma_ss(tS, desc_at(kKb, kmajor_step<RPX>(s)), desc_at(kQb, so + kmajor_step<RPX, HALF>(s)), idS, s > 0);
          }
#pragma unroll
          for (int t = 0; t < NQ; ++t) {  // key terms (k, or hi and lo of k*scale) share the Q tile
#pragma unroll
            for (int s = 0; s < D / 16; ++s)
              umma_ss(tS, desc_at(kK, t * Cfg::KT + kmajor_step<D>(s)), desc_at(kQ, so + kmajor_step<D, HALF>(s)), idS,
                      (RP || t > 0 || s > 0) ? 1u : 0u);
          }
          umma_commit(s_full + 8 * w);
          // behind the dV product that read the previous P^T: the threads store the next one once they have seen this dP^T
          if (Cfg::SEP_P && n > 0) {
            mbar_wait(dv_done + 8 * w, (n - 1) & 1, abort_flag);
            tc_fence_after_sync();
          }
#pragma unroll
          for (int s = 0; s < D / 16; ++s)
            umma_ss(tmem + w * Cfg::T_STREAM + Cfg::T_DP, desc_at(kV, kmajor_step<D>(s)),
                    desc_at(kDO, so + kmajor_step<D, HALF>(s)), idS, s > 0);
          umma_commit(dp_full + 8 * w);
        }
      } else if (warp == 14) {
        // ------------------------------------------------------------------ dV += P^T.dO
        const DescBase mDO = mnmajor_base<D, HALF>(sStage + Cfg::OFF_DO);
#pragma unroll 1
        for (int x = 0; x < n_half; ++x) {
          const int w = x & 1, n = x >> 1, st = x % NST;
          const uint32_t so = st * Cfg::STAGE_BYTES;
          mbar_wait(full + 8 * st, (x / NST) & 1, abort_flag);
          mbar_wait(p_ready + 8 * w, n & 1, abort_flag);
          tc_fence_after_sync();
#pragma unroll
          for (int s = 0; s < HALF / 16; ++s)  // contraction over the queries; A: 8 columns per 16 queries
            umma_ts(tmem + Cfg::T_DV, tmem + Cfg::T_P + w * Cfg::P_STRIDE + s * 8, desc_at(mDO, so + mnmajor_step<D>(s)),
                    idTD, (x > 0 || s > 0) ? 1u : 0u);
          umma_commit(dv_done + 8 * w);
          umma_commit(free_ + 8 * st);
        }
        umma_commit(all_done);
      } else {
        // ------------------------------------------------------------------ dK|dkb, dQ|dQb
        const DescBase mQ = mnmajor_base<D, HALF>(sStage), mQb = mnmajor_base<RPX, HALF>(sStage + Cfg::OFF_QB),
                       mDS = mnmajor_base<128>(sDS), mK = mnmajor_base<D>(sK);
        mbar_wait(kv_full, 0, abort_flag);
#pragma unroll 1
        for (int x = 0; x < n_half; ++x) {
          const int w = x & 1, n = x >> 1, st = x % NST;
          const uint32_t so = st * Cfg::STAGE_BYTES;
          mbar_wait(full + 8 * st, (x / NST) & 1, abort_flag);
          mbar_wait(ds_ready + 8 * w, n & 1, abort_flag);
          tc_fence_after_sync();
#pragma unroll
          for (int s = 0; s < HALF / 16; ++s)
            umma_ts(tmem + Cfg::T_DK, tmem + Cfg::T_DS + s * 8, desc_at(mQ, so + mnmajor_step<D>(s)), idTD, (x > 0 || s > 0) ? 1u : 0u);
          if (RP) {
#pragma unroll
            for (int s = 0; s < HALF / 16; ++s)
              umma_ts(tmem + Cfg::T_DKB, tmem + Cfg::T_DS + s * 8, desc_at(mQb, so + mnmajor_step<RPX>(s)), idTR,
                      (x > 0 || s > 0) ? 1u : 0u);
          }
          umma_commit(dk_done + 8 * w);
          umma_commit(free_ + 8 * st);
          if (w == 1) {  // both halves of the query tile are in shared memory
            if (n > 0) {
              mbar_wait(dq_drained, (n - 1) & 1, abort_flag);
              tc_fence_after_sync();
            }
            const uint32_t dso = n % Cfg::DS_BUFS * Cfg::DS_TILE;
#pragma unroll
            for (int s = 0; s < 8; ++s)  // contraction over the 128 keys
              umma_ss(tmem + Cfg::T_DQ, desc_at(mDS, dso + mnmajor_step<128>(s)), desc_at(mK, mnmajor_step<D>(s)), idQ, s > 0);
            umma_commit(dq_full);
          }
        }
        umma_commit(all_done);
      }
    }
  } else if (warp >= 8) {
    setmaxnreg_dec<64>();
    // ------------------------------------------------------------------ drain warpgroup (thread = query row)
    if (n_it > 0) {
      const int row = (warp & 3) * 32 + lane;
      const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
      const int bq = a.bq_bcast ? 0 : b, hq = a.hq_bcast ? 0 : h;
      if (NQ == 2) {
        mbar_wait(kv_full, 0, abort_flag);
        split_scaled_row<T, D>(sKs, row, a.k_scale);
        mbar_arrive_warp(ks_ready);
      }
      if (RP) {
        // k_bias of the four keys the centred copy refers to (one per 32-key group), as fp32: [column pair][key group][2]
        float* s_kbc = reinterpret_cast<float*>(smem + Cfg::OFF_KBC);
        const T* kb_bh = a.k_bias_t<T>() + (a.bk_bcast ? 0 : b) * a.kb_stride[0] + (a.hk_bcast ? 0 : h) * a.kb_stride[1];
        for (int i = (int)threadIdx.x - 256; i < 2 * RC; i += 128) {
          const int c = (i >> 3) * 2 + (i & 1), g = (i >> 1) & 3;
          s_kbc[i] = c < a.R ? to_f32(kb_bh[(int64_t)min(k0 + 32 * g + 16, a.Sk - 1) * a.kb_stride[2] + c]) : 0.f;
        }
        asm volatile("bar.sync 3, 128;" ::: "memory");  // the drain warpgroup only
      }
#pragma unroll 1
      for (int it = 0; it < n_it; ++it) {
        const uint32_t tq = tmem + lane_off;
        mbar_wait(dq_full, it & 1, abort_flag);
        tc_fence_after_sync();
        // Through the staging tile.  The first columns are fetched into registers while the copy engine may still be reading the
        // previous tile; the thread that issued that reduction then waits for its reads.
        uint32_t r0[32];
        tmem_ld32(tq + Cfg::T_DQ, r0);
        if (warp == 8 && lane == 0) bulk_wait_group_read0();
        __syncwarp();
        asm volatile("bar.sync 3, 128;" ::: "memory");
#pragma unroll
        for (int c0 = 0; c0 < D; c0 += 32) {
          if (c0) tmem_ld32(tq + Cfg::T_DQ + c0, r0);
          tmem_wait_ld(r0);
#pragma unroll
          for (int g = 0; g < 8; ++g)
            st_shared_v4(sStg + dq_stage_off(row, c0 / 4 + g), r0[g * 4], r0[g * 4 + 1], r0[g * 4 + 2], r0[g * 4 + 3]);
        }
        if (RP) {
          mbar_wait(rs_ready + 8 * (it & 3), (it >> 2) & 1, abort_flag);
          drain_dq_bias<RC / 2>(tq + Cfg::T_DQB, sbase + Cfg::OFF_ROWSUM + (it & 3) * 2048 + row * 4, sbase + Cfg::OFF_KBC,
                                sStg + Cfg::STG_DQ + row * 4, nullptr, true, a.R);
        }
        tc_fence_before_sync();
        mbar_arrive_warp(dq_drained);  // every tensor-memory and row-sum read of the tile is done
        fence_proxy_async_smem();      // the staged tile becomes visible to the copy engine
        asm volatile("bar.sync 3, 128;" ::: "memory");
        if (warp == 8 && lane == 0) {
          bulk_reduce_add_f32(a.dq_acc + ((int64_t)bh * a.nq_tiles + (i_begin + it)) * (128 * D), sStg, Cfg::STG_DQ);
          if (RP)
            bulk_reduce_add_f32(a.dqb_acc + (bh % a.dqb_slots) * a.dqb_slot_stride +
                                    (((int64_t)bq * a.Hq + hq) * a.nq_tiles + (i_begin + it)) * (128 * a.R),
                                sStg + Cfg::STG_DQ, 128 * a.R * 4);
          bulk_commit_group();
        }
      }
      // the staging tile must outlive the last reduction's reads; its global side completes with the kernel
      if (warp == 8 && lane == 0) bulk_wait_group_read0();
    }
  } else if (n_it > 0) {
    // ------------------------------------------------------------------ compute warps: stream w, 32 keys x 32 queries each
    setmaxnreg_inc<192>();
    const int w = warp >> 2, wl = warp & 3;
    const uint32_t lane_off = (uint32_t)(wl * 32) << 16;
    const uint32_t tS = tmem + w * Cfg::T_STREAM + Cfg::T_S + lane_off, tDP = tmem + w * Cfg::T_STREAM + Cfg::T_DP + lane_off,
                   tP = tmem + Cfg::T_P + w * Cfg::P_STRIDE + lane_off, tDS = tmem + Cfg::T_DS + lane_off;
    const float sl2 = a.scale_log2;
    const int krow = wl * 32 + (lane >> 2), qcol = 2 * (lane & 3);  // first key and query of the thread's fragment
    const float slope2 = MODE == BWD_ALIBI ? __ldg(a.alibi_slopes + h) * kLog2e : 0.f;
    const uint64_t sl2p = f2(sl2, sl2);
    int stg = w;  // ring stage of the half tile
    // stmatrix addresses in the stream's [128 keys][64 queries] half of the dS^T tile (128-byte lines, swizzled): lane l
    // gives row l % 8 of matrix l / 8, whose rows are keys 8 (l / 8 % 2) + ..., and whose columns chunk l / 16 of a pair
    const uint32_t ds_at = sDS + w * Cfg::DS_HALF + (wl * 32 + ((lane >> 3) & 1) * 8 + (lane & 7)) * 128 +
                           (((lane >> 4) ^ (lane & 7)) << 4);
    uint32_t s[2][32];
    auto load_s = [&] {
      tc_fence_after_sync();
      tmem_ld_16x256b_x8(tS, s[0]);
      tmem_ld_16x256b_x8(tS + (16u << 16), s[1]);
    };
    mbar_wait(s_full + 8 * w, 0, abort_flag);
    load_s();
#pragma unroll 1
    for (int n = 0; n < n_it; ++n) {
      const int q0 = i_begin * 128 + (2 * n + w) * HALF;
      const uint32_t st_n = sStat + stg * Cfg::STAT + qcol * 4;  // its statistics, from the thread's first query on
      stg = stg + 2 >= NST ? stg + 2 - NST : stg + 2;
      // s[k2][4j + 2i + e]: key krow + 16 k2 + 8 i, query qcol + 8 j + e
      uint64_t nl[8], ak[4];  // ALiBi: ak, the keys' share of the term
      if (MODE == BWD_ALIBI) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float x = slope2 * (float)(k0 + krow + 8 * k - q0);
          ak[k] = f2(x, x);
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) nl[j] = ld_shared_f2(st_n + j * 32);
      const bool dp_ok = mbar_test_wait(dp_full + 8 * w, n & 1);
      tmem_wait_ld(s[0]);
      tmem_wait_ld(s[1]);
      // dead pairs (keys beyond Sk, above the diagonal) become -inf logits: P and dS are then exactly zero
      if ((a.causal && k0 + 127 > q0) || k0 + 128 > a.Sk) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int key = k0 + krow + 8 * k;
          const int first = key >= a.Sk ? HALF : a.causal ? key - (q0 + qcol) : 0;  // 8j + e of the first live column
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (8 * j < first) s[k >> 1][4 * j + 2 * (k & 1)] = __float_as_uint(-INFINITY);
            if (8 * j + 1 < first) s[k >> 1][4 * j + 2 * (k & 1) + 1] = __float_as_uint(-INFINITY);
          }
        }
      }
      uint32_t pk[2][16];
#pragma unroll
      for (int k2 = 0; k2 < 2; ++k2) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            uint32_t &x0 = s[k2][4 * j + 2 * i], &x1 = s[k2][4 * j + 2 * i + 1];
            float a0, a1;
            f2_unpack(f2_fma(f2(__uint_as_float(x0), __uint_as_float(x1)), sl2p,
                             MODE == BWD_ALIBI ? f2_add(nl[j], ak[2 * k2 + i]) : nl[j]),
                      a0, a1);
            a0 = fast_exp2(a0);
            a1 = fast_exp2(a1);
            pk[k2][2 * j + i] = Pack2<T>::pack(a0, a1);
            x0 = __float_as_uint(a0);
            x1 = __float_as_uint(a1);
          }
        }
      }
      // dP^T is there: so the last dV product has read P^T
      mbar_wait_tested(dp_ok, dp_full + 8 * w, n & 1, abort_flag);
      tc_fence_after_sync();
      uint32_t d[2][32];
      tmem_ld_16x256b_x8(tDP, d[0]);
      tmem_ld_16x256b_x8(tDP + (16u << 16), d[1]);
      tmem_st_16x128b_x8(tP, pk[0]);
      tmem_st_16x128b_x8(tP + (16u << 16), pk[1]);
#pragma unroll
      for (int j = 0; j < 8; ++j) nl[j] = ld_shared_f2(st_n + HALF * 4 + j * 32);
      tmem_wait_st();
      tmem_wait_ld(d[0]);
      tmem_wait_ld(d[1]);
      tc_fence_before_sync();
      mbar_arrive_warp(p_ready + 8 * w);
      // ---- dS^T = P^T o (dP^T - delta)
      const bool dk_ok = mbar_test_wait(dk_done + 8 * (w ^ 1), (w ? n : n - 1) & 1);
      uint64_t sum[8];
#pragma unroll
      for (int k2 = 0; k2 < 2; ++k2) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const uint64_t p = f2(__uint_as_float(s[k2][4 * j + 2 * i]), __uint_as_float(s[k2][4 * j + 2 * i + 1]));
            const uint64_t ds =
                f2_mul(p, f2_add(f2(__uint_as_float(d[k2][4 * j + 2 * i]), __uint_as_float(d[k2][4 * j + 2 * i + 1])), nl[j]));
            if (RP) sum[j] = k2 + i == 0 ? ds : f2_add(sum[j], ds);
            float d0, d1;
            f2_unpack(ds, d0, d1);
            pk[k2][2 * j + i] = Pack2<T>::pack(d0, d1);
          }
        }
      }
      // The dK product of the other stream's last half tile has read dS^T in tensor memory, and the dQ product of the tile before
      // (one dS^T tile: the previous tile's) that in shared memory: one thread issues both kinds, and a commit covers what it
      // issued before.  The drain is then past the row sums of three tiles ago, too (there are four tables).
      if (Cfg::DS_BUFS == 1 && w == 0) {
        if (n > 0) mbar_wait(dq_full, (n - 1) & 1, abort_flag);
      } else if (w == 1 || n > 0) {
        mbar_wait_tested(dk_ok, dk_done + 8 * (w ^ 1), (w ? n : n - 1) & 1, abort_flag);
      }
      tc_fence_after_sync();
      const uint32_t ds_n = ds_at + n % Cfg::DS_BUFS * Cfg::DS_TILE;
      tmem_st_16x128b_x8(tDS, pk[0]);
      tmem_st_16x128b_x8(tDS + (16u << 16), pk[1]);
#pragma unroll
      for (int k2 = 0; k2 < 2; ++k2)
#pragma unroll
        for (int m = 0; m < 4; ++m)
          stmatrix_x4((ds_n + k2 * 2048) ^ (m << 5), pk[k2][4 * m], pk[k2][4 * m + 1], pk[k2][4 * m + 2], pk[k2][4 * m + 3]);
      const bool s_ok = mbar_test_wait(s_full + 8 * w, (n + 1) & 1);
      tmem_wait_st();
      fence_proxy_async_smem();
      tc_fence_before_sync();
      mbar_arrive_warp(ds_ready + 8 * w);
      // the next half tile's S^T is fetched under the row sums (behind the last one: columns that nothing uses any more)
      if (n + 1 < n_it) mbar_wait_tested(s_ok, s_full + 8 * w, (n + 1) & 1, abort_flag);
      load_s();
      if (RP) {
        // row sums over the warp's 32 keys: halve the columns, exchange, add; lane t ends up with queries
        // 8 (t / 4) + 2 (t % 4) + {0, 1}
        float v[8][2];
#pragma unroll
        for (int j = 0; j < 8; ++j) f2_unpack(sum[j], v[j][0], v[j][1]);
#pragma unroll
        for (int o = 4; o; o >>= 1) {
          const bool up = (lane >> 2) & o;
#pragma unroll
          for (int j = 0; j < o; ++j) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const float send = up ? v[j][e] : v[j + o][e], keep = up ? v[j + o][e] : v[j][e];
              v[j][e] = keep + __shfl_xor_sync(0xffffffffu, send, 4 * o);
            }
          }
        }
        st_shared_v2f(sbase + Cfg::OFF_ROWSUM + (n & 3) * 2048 + wl * 512 + (w * HALF + 8 * (lane >> 2) + qcol) * 4, v[0][0], v[0][1]);
        mbar_arrive_warp(rs_ready + 8 * (n & 3));
      }
    }
    tmem_wait_ld(s[0]);
    tmem_wait_ld(s[1]);
    // the dV and dK|dkb accumulators are final once every product has completed
    mbar_wait(all_done, 0, abort_flag);
    tc_fence_after_sync();

    // ---- epilogue: dV, dK (x scale), thread = key row, each warpgroup half of the columns
    constexpr int DH = D / 2;
    const int row = wl * 32 + lane, key = k0 + row;
    T* dvrow = reinterpret_cast<T*>(a.dv) + b * a.dv_stride[0] + h * a.dv_stride[1] + (int64_t)key * a.dv_stride[2];
    T* dkrow = reinterpret_cast<T*>(a.dk) + b * a.dk_stride[0] + h * a.dk_stride[1] + (int64_t)key * a.dk_stride[2];
#pragma unroll 1
    for (int c0 = w * DH; c0 < w * DH + DH; c0 += 16) {
      uint32_t rv[16], rk[16];
      tmem_ld16(tmem + Cfg::T_DV + lane_off + c0, rv);
      tmem_ld16(tmem + Cfg::T_DK + lane_off + c0, rk);
      tmem_wait_ld(rv);
      tmem_wait_ld(rk);
      if (key < a.Sk) {
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          if (c0 + g * 8 >= a.D) break;  // D is a multiple of 8
          auto pv = [&](int i) { return Pack2<T>::pack(__uint_as_float(rv[g * 8 + i]), __uint_as_float(rv[g * 8 + i + 1])); };
          auto pk2 = [&](int i) {
            return Pack2<T>::pack(__uint_as_float(rk[g * 8 + i]) * a.dk_scale, __uint_as_float(rk[g * 8 + i + 1]) * a.dk_scale);
          };
          *reinterpret_cast<uint4*>(dvrow + c0 + g * 8) = make_uint4(pv(0), pv(2), pv(4), pv(6));
          *reinterpret_cast<uint4*>(dkrow + c0 + g * 8) = make_uint4(pk2(0), pk2(2), pk2(4), pk2(6));
        }
      }
    }
    if (RP && w == 0) {
      // dk_bias: staged rank-major, [R][128], in the (now idle) dS^T tile, one bulk reduction into the accumulator (other
      // (batch, head) pairs add to the same rows when the factor is shared)
      static_assert(128 * RP * 4 <= 2 * Cfg::DS_HALF, "dk_bias staging");
      const int bk = a.bk_bcast ? 0 : b, hk = a.hk_bcast ? 0 : h;
      float* stg = reinterpret_cast<float*>(smem + Cfg::OFF_DS) + row;
#pragma unroll 1
      for (int c0 = 0; c0 < RPX && c0 < a.R; c0 += 16) {
        uint32_t r[16];
        tmem_ld16(tmem + Cfg::T_DKB + lane_off + c0, r);
        tmem_wait_ld(r);
#pragma unroll
        for (int i = 0; i < 16; ++i)
          if (c0 + i < a.R) stg[(c0 + i) * 128] = __uint_as_float(r[i]) * a.dkb_scale;
      }
      fence_proxy_async_smem();
      asm volatile("bar.sync 4, 128;" ::: "memory");  // this warpgroup only
      if (threadIdx.x == 0) {
        bulk_reduce_add_f32(a.dkb_acc + (bh % a.dkb_slots) * a.dkb_slot_stride +
                                (((int64_t)bk * a.Hk + hk) * a.nk_tiles + kt) * (128 * a.R),
                            sDS, 128 * a.R * 4);
        bulk_commit_group();
        bulk_wait_group_read0();  // shared memory must stay until it is read; the global side completes with the kernel
      }
    }
  } else {
    // causal with Sq < Sk: these keys are seen by no query; their gradients are zero
    const int w = warp >> 2, key = k0 + (warp & 3) * 32 + lane;
    if (key < a.Sk) {
      T* dvrow = reinterpret_cast<T*>(a.dv) + b * a.dv_stride[0] + h * a.dv_stride[1] + (int64_t)key * a.dv_stride[2];
      T* dkrow = reinterpret_cast<T*>(a.dk) + b * a.dk_stride[0] + h * a.dk_stride[1] + (int64_t)key * a.dk_stride[2];
      const uint4 z = make_uint4(0, 0, 0, 0);
      for (int c0 = w * (D / 2); c0 < min(w * (D / 2) + D / 2, a.D); c0 += 8) {
        *reinterpret_cast<uint4*>(dvrow + c0) = z;
        *reinterpret_cast<uint4*>(dkrow + c0) = z;
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  report_expired_wait(abort_flag, a.status);
  if (warp == 13) {
    settle_expired_wait(abort_flag);
    __syncwarp();
    tmem_dealloc(tmem, 512);
  }
}

// ------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------
template <typename T, int D, int RP, int RC, int NQ, int MODE>
int launch_bwd_s(const fb_params* p, const PackPlan& plan, cudaStream_t st) {
  using Cfg = BwdSCfg<D, RP, RC, NQ>;
  static_assert(Cfg::FITS, "shared or tensor memory");
  int rc;
  const BwdWs w = bwd_layout(p, plan);
  uint8_t* ws = reinterpret_cast<uint8_t*>(p->workspace);
  void *qpack = ws + w.off_qpack, *kpack = ws + w.off_kpack, *kcenter = ws + w.off_kcenter;
  CUtensorMap tQ, tK, tV, tDO, tQb, tKb, tKc;
  if ((rc = make_tmap_4d(&tQ, p->q, p->D, p->Sq, p->H, p->B, p->q_stride[2], p->q_stride[1], p->q_stride[0], D, Cfg::HALF)))
    return rc;
  if ((rc = make_tmap_4d(&tDO, p->dout, p->D, p->Sq, p->H, p->B, p->dout_stride[2], p->dout_stride[1], p->dout_stride[0],
                         D, Cfg::HALF)))
    return rc;
  if ((rc = make_tmap_4d(&tK, p->k, p->D, p->Sk, p->H, p->B, p->k_stride[2], p->k_stride[1], p->k_stride[0], D, 128)))
    return rc;
  if ((rc = make_tmap_4d(&tV, p->v, p->D, p->Sk, p->H, p->B, p->v_stride[2], p->v_stride[1], p->v_stride[0], D, 128)))
    return rc;
  tQb = tKb = tKc = tK;
  if (RP) {
    if ((rc = make_tmap_4d(&tQb, qpack, RP, p->Sq, plan.Hq, plan.Bq, RP, (int64_t)RP * p->Sq, (int64_t)RP * p->Sq * plan.Hq,
                           Cfg::RPX, Cfg::HALF)))
      return rc;
    if ((rc = make_tmap_4d(&tKb, kpack, RP, p->Sk, plan.Hk, plan.Bk, RP, (int64_t)RP * p->Sk, (int64_t)RP * p->Sk * plan.Hk,
                           Cfg::RPX, 128)))
      return rc;
    if ((rc = make_tmap_4d(&tKc, kcenter, RC, p->Sk, plan.Hk, plan.Bk, RC, (int64_t)RC * p->Sk, (int64_t)RC * p->Sk * plan.Hk,
                           D, 128)))
      return rc;
  }
  const BwdArgs a = bwd_args(p, plan, w);
  auto kern = bwd_s_sm100_kernel<T, D, RP, RC, NQ, MODE>;
  // per kernel instantiation and device: raise the dynamic shared-memory limit once
  static std::mutex mu;
  static bool attr_done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  {
    std::lock_guard<std::mutex> lk(mu);
    if (!attr_done[dev & 63]) {
      const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM);
      if (e != cudaSuccess) return (int)e;
      attr_done[dev & 63] = true;
    }
  }
  if ((rc = launch_prepare(p, plan, {qpack, kpack, RP ? kcenter : nullptr, nullptr, fused_delta(p), ws + w.off_dq, w.zero_bytes},
                           st)))
    return rc;
  const unsigned grid = (unsigned)((int64_t)a.nk_tiles * p->B * p->H);
  prof_before(KC_BWD_MAIN, st);
  rc = launch_pdl(kern, grid, kBwdSThreads, Cfg::SMEM, st, tQ, tK, tV, tDO, tQb, tKb, tKc, a);
  prof_after(KC_BWD_MAIN, st);
  if (rc) return rc;
  return launch_store_grads(p, {a.dq_acc, DQ_SWIZZLED, D, a.dqb_acc, a.dkb_acc,
                                {(int64_t)a.nq_tiles * 128, a.dqb_slots, a.dqb_slot_stride},
                                {(int64_t)a.nk_tiles * 128, a.dkb_slots, a.dkb_slot_stride}},
                            st);
}

}  // namespace fb
