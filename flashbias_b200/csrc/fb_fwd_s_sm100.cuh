// Forward FlashBias attention for sm_100a at head_dim 65 to 128, without a mask: two softmax streams per CTA.
//
// Tensor memory holds one CTA per SM at this head_dim, and with one softmax warpgroup (fb_fwd_sm100.cuh) the tensor core waits
// for the exponentials and the exponentials for the tensor core.  Here two softmax warpgroups share a query tile and take its
// key tiles in turn, each with logits and probabilities of its own in tensor memory, so that the maximum of one tile, the
// exponentials of another and the products of a third run at the same time.  There is one output accumulator and one running
// reference maximum per row, which the warpgroups hand to one another through shared memory behind each tile's row maximum; row
// sums stay apart until the end of the item, whose columns the warpgroups then store half each.
//   warps 0-3, 4-7  softmax of the even / odd key tiles, thread = query row; epilogue
//   warp 8          TMA producer          warp 9   S = [Q|Qb].[K|Kb]^T          warp 10   O += P.V
// (Two accumulators with a merge at the end need no hand-over, but leave no room for P beside S: a stream's next S then waits
// for its P.V product, 4800 clk a pair of tiles instead of 4200.)
// What bounds it: the tensor core with a split scale (1640 of the 2100 clk of a key tile), and reading K and V: one query tile
// per CTA draws 68 KB a tile from L2, about 45 bytes per clock and SM, and a stage takes 3000 clk to arrive.
// Forward kernel, one stream / two: B1 H32 S4001 R2 causal fp16 198 / 185 us, B2 H16 S2048 slopes causal bf16 60 / 55 us.
#pragma once

#include "fb_fwd_sm100.cuh"

namespace fb {

template <int RP, int NQ>
struct FwdSCfg {
  static constexpr int D = 128;
  static constexpr int RPX = RP ? RP : 16;
  static constexpr int Q_BYTES = tile_bytes(D), QB_BYTES = RP ? tile_bytes(RPX) : 0;
  // barriers; (maximum, sum) per item parity, stream and row; reference maximum handed over, per stream and row; alignment
  static constexpr int TAIL = 256 + 2 * 2 * 128 * 8 + 2 * 128 * 4 + 1024;
  static constexpr int LIM = 227 * 1024;
  static constexpr int smem_for(int st) { return NQ * Q_BYTES + QB_BYTES + st * (2 * Q_BYTES + QB_BYTES) + TAIL; }
  // Stages of K | Kb and of V.  Two, and not only because three do not fit: the wait for the other stream's last product ahead of a
  // rescale relies on it.
  static constexpr int ST = 2;
  static_assert(smem_for(3) > LIM, "a third stage would fit");
  static constexpr int SMEM = smem_for(ST);
  static constexpr bool FITS = SMEM <= LIM;
  static constexpr int OFF_QB = NQ * Q_BYTES, OFF_K = OFF_QB + QB_BYTES, OFF_KB = OFF_K + ST * Q_BYTES,
                       OFF_V = OFF_KB + ST * QB_BYTES, OFF_BAR = OFF_V + ST * Q_BYTES, OFF_ML = OFF_BAR + 256, OFF_M = OFF_ML + 2 * 2 * 128 * 8;
  static constexpr int T_S = 0, T_P = 256, T_O = 384;  // stream x: S + 128 x, P + 64 x
};

template <typename T, int RP, int NQ, int MODE>
__global__ void __launch_bounds__(384, 1)
fwd_s_sm100_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                   const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmQb,
                   const __grid_constant__ CUtensorMap tmKb, const FwdArgs a) {
  using Cfg = FwdSCfg<RP, NQ>;
  constexpr int D = Cfg::D, RPX = Cfg::RPX, ST = Cfg::ST;
  constexpr bool kBf16 = std::is_same<T, __nv_bfloat16>::value;
  constexpr float kLog2e = 1.4426950408889634f;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t sbase = smem_u32(smem);
  const uint32_t sQ = sbase, sQb = sbase + Cfg::OFF_QB, sK = sbase + Cfg::OFF_K, sKb = sbase + Cfg::OFF_KB,
                 sV = sbase + Cfg::OFF_V;
  const uint32_t bar0 = sbase + Cfg::OFF_BAR;
  // (two slots: one per stream, or per stage)
  const uint32_t q_full = bar0, q_free = bar0 + 8, o_free = bar0 + 16, s_full = bar0 + 24, p_ready = bar0 + 40,
                 pv_done = bar0 + 56, k_full = bar0 + 72, k_free = bar0 + 88, v_full = bar0 + 104, v_free = bar0 + 120,
                 s_read = bar0 + 136, q_ready = bar0 + 152;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + Cfg::OFF_BAR + 160);
  const uint32_t abort_flag = bar0 + 164;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int BH = a.B * a.H;
  struct Item {
    int bh, b, h, q0, n_kv;
    // First key of the j-th key tile visited.  Under causal masking from the diagonal down: a bias that falls with the distance
    // (ALiBi) then shows its maximum first, and the accumulator is hardly ever rescaled (600 clk of a tile's 2500 at steep slopes).
    // B1 H32 S4001 R2: 185 us, in ascending order 250 (one stream, ascending: 200).  With factor operands too, unlike in
    // fwd_sm100_kernel: the errors against 64 bits are no larger (ALiBi, S 2048, bf16, descending / ascending: o 1.90e-3 /
    // 1.93e-3, dq_bias, which is all cancellation there, 1.215 / 1.213).
    __device__ __forceinline__ int key0(int j, int causal) const { return (causal ? n_kv - 1 - j : j) * 128; }
  };
  // the w-th item of this CTA: heaviest first under causal masking, taken in snake order (as in fwd_sm100_kernel)
  auto item_index = [&](int w) {
    const int G = (int)gridDim.x, c = (int)blockIdx.x;
    return w * G + ((w & 1) ? G - 1 - c : c);
  };
  auto item_of = [&](int idx) {
    Item it;
    int qt;
    if (a.causal) {
      qt = a.nq_tiles - 1 - idx / BH;
      it.bh = idx % BH;
    } else {
      qt = idx % a.nq_tiles;
      it.bh = idx / a.nq_tiles;
    }
    it.b = it.bh / a.H;
    it.h = it.bh % a.H;
    it.q0 = qt * 128;
    const int kv_end = a.causal ? min(a.Sk, it.q0 + 128) : a.Sk;
    it.n_kv = (kv_end + 127) / 128;
    return it;
  };

  if (warp == 8) {
    if (lane == 0) {
      st_shared_flag(abort_flag, 0u);
      mbar_init(q_full, 1);
      mbar_init(q_free, 1);
      mbar_init(q_ready, 8);  // the softmax warps have split the item's q*scale
      mbar_init(o_free, 8);  // every softmax warp has read the accumulators of the item
      for (int i = 0; i < 2; ++i) {
        mbar_init(s_full + 8 * i, 1);
        mbar_init(p_ready + 8 * i, 4);  // the stream's warps
        mbar_init(pv_done + 8 * i, 1);
        mbar_init(s_read + 8 * i, 4);  // the logits of the tile are in registers
      }
      for (int i = 0; i < ST; ++i) {
        mbar_init(k_full + 8 * i, 1);
        mbar_init(k_free + 8 * i, 1);
        mbar_init(v_full + 8 * i, 1);
        mbar_init(v_free + 8 * i, 1);
      }
      mbar_fence_init();
    }
  } else if (warp == 9) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  grid_dep_wait();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;

  if (warp >= 8) {
    setmaxnreg_dec<88>();
    if (warp == 8) {
      // ------------------------------------------------------------------ TMA producer
      auto produce = [&] {
        int t = 0, n = 0;  // key tiles and items started
        for (int w = 0, idx; (idx = item_index(w)) < a.total_items; ++w, ++n) {
          const Item it = item_of(idx);
          const int hq = a.hq_bcast ? 0 : it.h, bq = a.bq_bcast ? 0 : it.b;
          const int hk = a.hk_bcast ? 0 : it.h, bk = a.bk_bcast ? 0 : it.b;
          if (n > 0 && !mbar_wait(q_free, (n - 1) & 1, abort_flag)) return;
          mbar_expect_tx(q_full, Cfg::Q_BYTES + Cfg::QB_BYTES);
          tma_tile_4d<D>(sQ, &tmQ, q_full, it.q0, it.h, it.b);
          if (RP) tma_tile_4d<RPX>(sQb, &tmQb, q_full, it.q0, hq, bq);
          for (int j = 0; j < it.n_kv; ++j, ++t) {
            const int st = t % ST;
            if (t >= ST && !mbar_wait(k_free + 8 * st, (t / ST - 1) & 1, abort_flag)) return;
            mbar_expect_tx(k_full + 8 * st, Cfg::Q_BYTES + Cfg::QB_BYTES);
            tma_tile_4d<D>(sK + st * Cfg::Q_BYTES, &tmK, k_full + 8 * st, it.key0(j, a.causal), it.h, it.b);
            if (RP) tma_tile_4d<RPX>(sKb + st * Cfg::QB_BYTES, &tmKb, k_full + 8 * st, it.key0(j, a.causal), hk, bk);
            if (t >= ST && !mbar_wait(v_free + 8 * st, (t / ST - 1) & 1, abort_flag)) return;
            mbar_expect_tx(v_full + 8 * st, Cfg::Q_BYTES);
            tma_tile_4d<D>(sV + st * Cfg::Q_BYTES, &tmV, v_full + 8 * st, it.key0(j, a.causal), it.h, it.b);
          }
        }
      };
      if (elect_one()) produce();
    } else if (warp == 9) {
      // ------------------------------------------------------------------ MMA issuer: S = [Q|Qb].[K|Kb]^T
      if (elect_one()) {
        constexpr uint32_t idS = instr_desc(kBf16, false, false, 128, 128);
        const DescBase dQ = kmajor_base<D>(sQ), dQb = kmajor_base<RPX>(sQb), dK = kmajor_base<D>(sK),
                       dKb = kmajor_base<RPX>(sKb);
        int t = 0, n = 0, c0 = 0, c1 = 0;  // key tiles, items; key tiles of either stream
        for (int w = 0, idx; (idx = item_index(w)) < a.total_items; ++w, ++n) {
          const Item it = item_of(idx);
          mbar_wait(NQ == 2 ? q_ready : q_full, n & 1, abort_flag);
          tc_fence_after_sync();
          for (int j = 0; j < it.n_kv; ++j, ++t) {
            const int x = j & 1, c = x ? c1++ : c0++, st = t % ST;
            if (c > 0) mbar_wait(s_read + 8 * x, (c - 1) & 1, abort_flag);
            mbar_wait(k_full + 8 * st, (t / ST) & 1, abort_flag);
            tc_fence_after_sync();
            const uint32_t tS = tmem + Cfg::T_S + 128 * x, ko = st * Cfg::Q_BYTES, kbo = st * Cfg::QB_BYTES;
            // bias products first, into the empty accumulator (large factor terms cancel among themselves)
            if (RP) {
#pragma unroll
              for (int s = 0; s < RPX / 16; ++s)
                umma_ss(tS, desc_at(dQb, kmajor_step<RPX>(s)), desc_at(dKb, kbo + kmajor_step<RPX>(s)), idS, s > 0);
            }
#pragma unroll
            for (int q = 0; q < NQ; ++q) {  // query terms share the K tile
#pragma unroll
              for (int s = 0; s < D / 16; ++s)
                umma_ss(tS, desc_at(dQ, q * Cfg::Q_BYTES + kmajor_step<D>(s)), desc_at(dK, ko + kmajor_step<D>(s)), idS,
                        (RP || q > 0 || s > 0) ? 1u : 0u);
            }
            umma_commit(s_full + 8 * x);
            umma_commit(k_free + 8 * st);
          }
          umma_commit(q_free);  // Q | Qb of this item are no longer read
        }
      }
    } else if (warp == 10) {
      // ------------------------------------------------------------------ MMA issuer: O += P.V
      if (elect_one()) {
        constexpr uint32_t idO = instr_desc(kBf16, false, true, 128, D);
        const DescBase dV = mnmajor_base<D>(sV);
        int t = 0, n = 0, c0 = 0, c1 = 0;
        for (int w = 0, idx; (idx = item_index(w)) < a.total_items; ++w, ++n) {
          const Item it = item_of(idx);
          for (int j = 0; j < it.n_kv; ++j, ++t) {
            const int x = j & 1, c = x ? c1++ : c0++, st = t % ST;
            mbar_wait(v_full + 8 * st, (t / ST) & 1, abort_flag);
            mbar_wait(p_ready + 8 * x, c & 1, abort_flag);
            if (j == 0 && n > 0) mbar_wait(o_free, (n - 1) & 1, abort_flag);  // the accumulator of the last item has been read
            tc_fence_after_sync();
            const uint32_t tO = tmem + Cfg::T_O, tP = tmem + Cfg::T_P + 64 * x, vo = st * Cfg::Q_BYTES;
#pragma unroll
            for (int s = 0; s < 8; ++s)
              umma_ts(tO, tP + s * 8, desc_at(dV, vo + mnmajor_step<D>(s)), idO, (j > 0 || s > 0) ? 1u : 0u);
            umma_commit(pv_done + 8 * x);
            umma_commit(v_free + 8 * st);
          }
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax + epilogue
    setmaxnreg_inc<208>();
    const int x = warp >> 2, row = (warp & 3) * 32 + lane;
    const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tS = tmem + Cfg::T_S + 128 * x + lane_off, tP = tmem + Cfg::T_P + 64 * x + lane_off,
                   tO = tmem + Cfg::T_O + lane_off;
    const uint32_t m_own = sbase + Cfg::OFF_M + (x * 128 + row) * 4, m_other = sbase + Cfg::OFF_M + ((x ^ 1) * 128 + row) * 4;
    const float sl2 = a.scale_log2;
    const uint64_t sl2p = f2(sl2, sl2);
    int c = 0, co = 0, n = 0;  // key tiles of this stream and of the other, items so far
    uint32_t s[4][32];  // the thread's row of the logit tile
    // The split of q*scale, half a row per thread, in place and into the tile behind; the next item's ahead of this one's
    // epilogue, under the wait for the last products.
    int n_split = 0;
    auto split_q = [&] {
      mbar_wait(q_full, n_split++ & 1, abort_flag);
#pragma unroll
      for (int ch = 0; ch < 8; ++ch) {
        const uint32_t at = sQ + tile_chunk_offset<D>(row, 64 * x + 8 * ch);
        split_scaled_chunk<T>(at, at + Cfg::Q_BYTES, a.q_scale);
      }
      fence_proxy_async_smem();
      mbar_arrive_warp(q_ready);
    };
    if (NQ == 2 && item_index(0) < a.total_items) split_q();
    for (int w = 0, idx; (idx = item_index(w)) < a.total_items; ++w, ++n) {
      const Item it = item_of(idx);
      const int grow = it.q0 + row;
      float m_used = -INFINITY, l = 0.f;  // reference maximum (log2 units: logit * log2 e); row sum of this stream's tiles, relative to it
      const int c0 = c, co0 = co;
      float slope2 = 0.f;                 // ALiBi slope of this head, times log2 e
      if (MODE == FWD_ALIBI) slope2 = __ldg(a.alibi_slopes + it.h) * kLog2e;
      for (int j = x; j < it.n_kv; j += 2, ++c) {
        const int k0 = it.key0(j, a.causal);
        mbar_wait(s_full + 8 * x, c & 1, abort_flag);
        tc_fence_after_sync();
        const bool dead = (a.causal && k0 + 127 > it.q0) || (k0 + 128 > a.Sk);
        // ---- logits from tensor memory (the load of one 32-column chunk overlaps the arithmetic of the previous one),
        // completed (log2 units for ALiBi), and the row maximum, four chains
        float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
        const float abase = slope2 * (float)(k0 - grow);
        auto complete = [&](int ch) {
          if (dead) {
            const int last = (a.causal ? min(grow, a.Sk - 1) : a.Sk - 1) - (k0 + ch * 32);  // last live column of the chunk
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (i > last) s[ch][i] = __float_as_uint(-INFINITY);
          }
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            float v0 = __uint_as_float(s[ch][i]), v1 = __uint_as_float(s[ch][i + 1]);
            if (MODE == FWD_ALIBI) {
              f2_unpack(f2_fma(f2(v0, v1), sl2p,
                               f2(fmaf((float)(ch * 32 + i), slope2, abase), fmaf((float)(ch * 32 + i + 1), slope2, abase))),
                        v0, v1);
              s[ch][i] = __float_as_uint(v0);
              s[ch][i + 1] = __float_as_uint(v1);
            }
            mx4[(i >> 1) & 3] = fmax3(mx4[(i >> 1) & 3], v0, v1);
          }
        };
        tmem_ld32(tS, s[0]);
        tmem_wait_ld(s[0]);
        tmem_ld32(tS + 32, s[1]);
        complete(0);
        tmem_wait_ld(s[1]);
        tmem_ld32(tS + 64, s[2]);
        complete(1);
        tmem_wait_ld(s[2]);
        tmem_ld32(tS + 96, s[3]);
        complete(2);
        tmem_wait_ld(s[3]);
        tc_fence_before_sync();
        mbar_arrive_warp(s_read + 8 * x);  // the tensor core may start on the stream's next tile
        complete(3);
        float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
        if (MODE == FWD_PLAIN) mx *= sl2;  // sl2 > 0
        // ---- the reference maximum, from tile to tile: it moves only when the maximum has grown by more than 2^8 (exact: the row
        // sums carry the same reference)
        const float m_last = m_used;
        if (j > 0) {
          asm volatile("bar.sync %0, 256;" ::"r"(2 + (x ^ 1)) : "memory");
          m_used = __uint_as_float(ld_shared_flag(m_other));
          const float m_new = fmaxf(m_used, mx);
          if (__any_sync(0xffffffffu, m_new - m_used > 8.f)) {
            // O is stable behind the product of tile j - 1.  The wait tests a parity, so the other stream's product before it, tile
            // j - 3, must be known to have completed (or its phase would pass for this one): tile j's logits are here, K(j) was
            // loaded behind V(j - 1), and V(j - 1), in a ring of two, where V(j - 3) had been, behind that product.
            static_assert(ST == 2, "a deeper ring does not order the products of tiles j - 3 and j");
            mbar_wait(pv_done + 8 * (x ^ 1), (co0 + ((j - 1) >> 1)) & 1, abort_flag);
            tc_fence_after_sync();
            const float alpha = m_new == -INFINITY ? 1.f : fast_exp2(m_used - m_new);
            m_used = m_new;
#pragma unroll 1
            for (int ch = 0; ch < D / 32; ++ch) {
              uint32_t r[32];
              tmem_ld32(tO + ch * 32, r);
              tmem_wait_ld(r);
#pragma unroll
              for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
              tmem_st32(tO + ch * 32, r);
            }
            tmem_wait_st();
          }
        } else {
          m_used = mx;
        }
        if (j + 1 < it.n_kv) {
          st_shared_f32(m_own, m_used);
          asm volatile("bar.arrive %0, 256;" ::"r"(2 + x) : "memory");
        }
        if (c > 0) mbar_wait(pv_done + 8 * x, (c - 1) & 1, abort_flag);  // P has been read
        // ---- p = exp2(logit2 - m), row sum, P -> tensor memory (the A operand of O += P.V)
        const float msub = m_used == -INFINITY ? 0.f : m_used;
        l *= fast_exp2(m_last - msub);  // (0 at the stream's first tile, where l is 0)
        uint64_t l2a = f2(0.f, 0.f), l2b = f2(0.f, 0.f);
        const uint64_t nm = f2(-msub, -msub);
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) {
          uint32_t pw[16];  // 32 keys = 16 packed words
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const uint64_t v = f2(__uint_as_float(s[ch][i]), __uint_as_float(s[ch][i + 1]));
            float a0, a1;
            f2_unpack(MODE == FWD_PLAIN ? f2_fma(v, sl2p, nm) : f2_add(v, nm), a0, a1);
            const float p0 = fast_exp2(a0), p1 = fast_exp2(a1);
            if (i & 2) l2b = f2_add(l2b, f2(p0, p1)); else l2a = f2_add(l2a, f2(p0, p1));
            pw[i / 2] = Pack2<T>::pack(p0, p1);
          }
          tmem_st16(tP + ch * 16, pw);
        }
        {
          float x0, x1, x2, x3;
          f2_unpack(l2a, x0, x1);
          f2_unpack(l2b, x2, x3);
          l += (x0 + x1) + (x2 + x3);
        }
        tmem_wait_st();
        tc_fence_before_sync();
        mbar_arrive_warp(p_ready + 8 * x);
      }
      if (NQ == 2 && item_index(w + 1) < a.total_items) split_q();
      // ---- epilogue: O / l -> global, this warpgroup's half of the columns; lse.  The stream of the last tile knows its product
      // to have completed (its commit covers the ones before it, which the same thread issued); the other learns it from the
      // warpgroups' barrier.
      c = c0 + ((it.n_kv + 1 - x) >> 1);
      co = co0 + ((it.n_kv + x) >> 1);
      const int xl = (it.n_kv - 1) & 1;  // stream of the last tile
      if (xl == x) mbar_wait(pv_done + 8 * x, (c - 1) & 1, abort_flag);
      float2* ml = reinterpret_cast<float2*>(smem + Cfg::OFF_ML) + (n & 1) * 256;
      ml[x * 128 + row] = make_float2(m_used, l);
      asm volatile("bar.sync 1, 256;" ::: "memory");  // both warpgroups
      tc_fence_after_sync();
      const float2 other = ml[(x ^ 1) * 128 + row];
      const float m = fmaxf(m_used, other.x), ms = m == -INFINITY ? 0.f : m;  // the last reference is the largest
      const float ls = l * fast_exp2(m_used - ms) + other.y * fast_exp2(other.x - ms), inv = ls > 0.f ? 1.f / ls : 0.f;
      T* orow = reinterpret_cast<T*>(a.o) + it.b * a.o_stride[0] + it.h * a.o_stride[1] + (int64_t)grow * a.o_stride[2] + x * 64;
#pragma unroll 1
      for (int ch = 0; ch < 2; ++ch) {
        uint32_t r[32];
        tmem_ld32(tO + x * 64 + ch * 32, r);
        tmem_wait_ld(r);
        if (grow < a.Sq) {
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            if (x * 64 + ch * 32 + g * 8 >= a.D) break;  // D is a multiple of 8
            auto p2 = [&](int i) {
              return Pack2<T>::pack(__uint_as_float(r[g * 8 + i]) * inv, __uint_as_float(r[g * 8 + i + 1]) * inv);
            };
            *reinterpret_cast<uint4*>(orow + ch * 32 + g * 8) = make_uint4(p2(0), p2(2), p2(4), p2(6));
          }
        }
      }
      // natural-log lse of the logits: (m + log2 l) * ln 2
      if (x == 0 && grow < a.Sq)
        a.lse[(int64_t)it.bh * a.lse_stride_bh + grow] = ls > 0.f ? (m + fast_log2(ls)) * 0.6931471805599453f : -INFINITY;
      tc_fence_before_sync();
      mbar_arrive_warp(o_free);
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  report_expired_wait(abort_flag, a.status);
  if (warp == 9) {
    settle_expired_wait(abort_flag);
    __syncwarp();
    tmem_dealloc(tmem, 512);
  }
}

// ------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------
template <typename T, int RP, int NQ, int MODE>
int launch_fwd_s(const fb_params* p, const PackPlan& plan, cudaStream_t st) {
  using Cfg = FwdSCfg<RP, NQ>;
  static_assert(Cfg::FITS, "shared memory");
  constexpr int D = Cfg::D;
  int rc;
  uint8_t* ws = reinterpret_cast<uint8_t*>(p->workspace);
  void *qpack = ws, *kpack = ws + plan.q_bytes;
  CUtensorMap tQ, tK, tV, tQb, tKb;
  if ((rc = make_tmap_4d(&tQ, p->q, p->D, p->Sq, p->H, p->B, p->q_stride[2], p->q_stride[1], p->q_stride[0], 64, 128))) return rc;
  if ((rc = make_tmap_4d(&tK, p->k, p->D, p->Sk, p->H, p->B, p->k_stride[2], p->k_stride[1], p->k_stride[0], 64, 128))) return rc;
  if ((rc = make_tmap_4d(&tV, p->v, p->D, p->Sk, p->H, p->B, p->v_stride[2], p->v_stride[1], p->v_stride[0], 64, 128))) return rc;
  tQb = tKb = tK;
  if (RP) {
    if ((rc = make_tmap_4d(&tQb, qpack, RP, p->Sq, plan.Hq, plan.Bq, RP, (int64_t)RP * p->Sq, (int64_t)RP * p->Sq * plan.Hq,
                           Cfg::RPX, 128)))
      return rc;
    if ((rc = make_tmap_4d(&tKb, kpack, RP, p->Sk, plan.Hk, plan.Bk, RP, (int64_t)RP * p->Sk, (int64_t)RP * p->Sk * plan.Hk,
                           Cfg::RPX, 128)))
      return rc;
  }
  const FwdArgs a = fwd_args(p, plan);
  if ((rc = launch_prepare(p, plan, {qpack, kpack, nullptr, nullptr, nullptr, nullptr, 0}, st))) return rc;
  auto kern = fwd_s_sm100_kernel<T, RP, NQ, MODE>;
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
  const int sms = device_sm_count(dev);
  if (sms <= 0) return FB_ENOTBUILT;
  const unsigned grid = (unsigned)(a.total_items < sms ? a.total_items : sms);  // persistent: one CTA per SM
  prof_before(KC_FWD_MAIN, st);
  rc = launch_pdl(kern, grid, 384, Cfg::SMEM, st, tQ, tK, tV, tQb, tKb, a);
  prof_after(KC_FWD_MAIN, st);
  return rc;
}

}  // namespace fb
