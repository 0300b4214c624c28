// Plain forward attention for sm_100a: two query tiles per CTA that take turns on the MUFU unit and the tensor pipe.
//
// What bounds it.  One 128 x 128 block at head_dim 72 is 650 cycles of MMA (measured: 5 products of N = 128 from shared
// memory 330, 8 of N = 80 from tensor memory 326) and, with a quarter of the exponentials on the FMA pipe, 768 cycles of
// MUFU.  A softmax warp needs about 1700 cycles from "S is ready" to "P is written" (150 to read S, 330 for the row
// maximum, 1060 for the exponentials, 125 to write P), and from there the product, the next S and the latencies around
// them take 1400: with one query tile per SM both pipes are more than half idle (the CTA-pair kernel that did this pass
// before: 2200 cycles per block).  Here a CTA holds two query tiles of one (batch, head), each with S / P, O and four
// softmax warps of its own: while one tile waits for its products the other computes.  K and V blocks are shared.
//
// Measured (one B200, sustained; the power limit is reached, the SM clock falls to 1.64 GHz): 64 x 16 heads x 1024 tokens,
// head_dim 72: 549 -> 462 us; 256 x 16 x 256 tokens, 72: 191 -> 166 us; 16 x 12 x 2048 tokens, 128: 395 -> 363 us.
// Within 1 % of it or slower: P in columns of its own (one buffer the tiles take in turn) with S issued a block or two
// ahead, with one or two MMA-issuing warps (shorter in cycles, at a lower clock; 15 % slower at two blocks per tile); a
// score row shared by two warps, the maximum exchanged through shared memory (10 % slower).
//
// Warps (320 threads): TMA producer; MMA issuer; four softmax warps per tile (one query row per thread), which also write
// their tile out.  Tensor memory: S_a 128 | S_b 128 | O_a DPAD | O_b DPAD = 416 columns at head_dim 72, 512 at 128; P
// (16-bit) is written over the first 64 columns of its S.  The issue order per key block is
//
//     P_a V_j, S_a,j+1 | P_b V_j, S_b,j+1
//
// and one commit behind each S says "S ready" and "O holds every block before it" (MMAs of one thread execute in order), so
// a rescale of O needs no wait of its own and S may be written over the P that the product before it reads.
//
// Query tiles are double-buffered where shared memory allows (head_dim <= 96); the output tile is staged in the query
// tile's own buffer, which is dead by then, and leaves by TMA store.
//
// Two variants of the per-row arithmetic, by the shape of one (batch, head) alone (duo_cubics).  With an even number of tiles
// and head_dim <= 96 it is that of attn_fwd_pair.cuh (order of the sums, a quarter of the exponentials cubics): o is bit for
// bit the primal output of the dual pass.  Elsewhere it is that of attn_fwd_kernel, which takes these shapes too when they
// are few (fwd_uses_duo in dmf_attn.cu): all exponentials on the MUFU unit, a row's sum as two halves.  So o and lse of an
// element never depend on how many others are in the batch.
#pragma once

#include "attn_fwd.cuh"

namespace dmf {

template <int TAIL>
struct DuoTraits {
  static constexpr int kDPad = 64 + TAIL;
  static constexpr int kMainBytes = 128 * 128;
  static constexpr int kTailBytes = 128 * TAIL * 2;
  static constexpr int kTileBytes = kMainBytes + kTailBytes;
  static constexpr int kVAtoms = (kDPad + 31) / 32;   // V as atoms of 32 columns x 128 rows (see FwdTraits)
  static constexpr int kVAtomBytes = 128 * 64;
  static constexpr int kVTileBytes = kVAtoms * kVAtomBytes;
  static constexpr int kQBufs = TAIL == 64 ? 1 : 2;
  static constexpr int kStagesK = TAIL == 0 ? 4 : 3;
  static constexpr int kStagesV = TAIL == 0 ? 4 : TAIL == 16 ? 3 : 2;
  static constexpr int kTileSmem = 2 * kQBufs * kTileBytes + kStagesK * kTileBytes + kStagesV * kVTileBytes;
  // barriers; Q: [slot * kQBufs + buffer]; S, P, O: per slot
  static constexpr int kBarQFull = 0, kBarQEmpty = 4, kBarSFull = 8, kBarPFull = 10, kBarOFull = 12, kBarKFull = 14, kBarKEmpty = kBarKFull + kStagesK, kBarVFull = kBarKEmpty + kStagesK,
                       kBarVEmpty = kBarVFull + kStagesV, kNumBars = kBarVEmpty + kStagesV;
  static constexpr int kSmemBytes = 1024 + kTileSmem + kNumBars * 8 + 16;
  static_assert(kSmemBytes <= 227 * 1024, "shared memory of one CTA");
  static constexpr uint32_t kColS = 0, kColO = 256;   // slot s: S at kColS + 128 s, O at kColO + kDPad s
  static constexpr uint32_t kTmemCols = 512;
  static constexpr uint32_t kTailSwizzle = TAIL == 64 ? kSwizzle128 : (TAIL == 32 ? kSwizzle64 : kSwizzle32);
  static constexpr uint32_t kTailRowBytes = 2 * TAIL;
};

constexpr int kDuoThreads = 320;

// whether the arithmetic is that of the pair kernel (see above)
constexpr bool duo_cubics(int tail, int num_q_tiles) { return tail <= 32 && num_q_tiles % 2 == 0; }

// p.num_tiles counts units: p.unit_tiles (1 or 2) neighbouring query tiles of one (batch, head); with an odd number of
// tiles the last unit of a head has one.
template <typename T, int TAIL, bool kCubics>
__global__ void __launch_bounds__(kDuoThreads, 1)
attn_fwd_duo_kernel(const __grid_constant__ FwdParams p) {
  using TR = DuoTraits<TAIL>;
  constexpr int DPAD = TR::kDPad;
  constexpr bool kBf16 = Pack2<T>::kIsBf16;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  const uint32_t s_q = smem_u32(smem);                                   // [slot][buffer]
  const uint32_t s_k = s_q + 2 * TR::kQBufs * TR::kTileBytes;
  const uint32_t s_v = s_k + TR::kStagesK * TR::kTileBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + TR::kTileSmem);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + TR::kNumBars);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const uint32_t bar0 = smem_u32(bars);
  auto bar = [&](int i) -> uint32_t { return bar0 + 8u * static_cast<uint32_t>(i); };

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int num_kv_blocks = p.seqlen_kv / kBlockKV;
  const int units_per_bh = (p.num_q_tiles + p.unit_tiles - 1) / p.unit_tiles;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int i = 0; i < TR::kNumBars; ++i)
      mbar_init(bar(i), i == TR::kBarPFull || i == TR::kBarPFull + 1 ? 4 : 1);  // the four softmax warps of a slot
    fence_mbar_init();
  }
  if (warp == 0) {
    __syncwarp();
    tmem_alloc(smem_u32(tmem_slot), TR::kTmemCols);
    tmem_relinquish_alloc_permit();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;

  // query tiles of a unit
  auto unit_slots = [&](int u) -> int {
    return min(p.unit_tiles, p.num_q_tiles - p.unit_tiles * (u % units_per_bh));
  };

  if (warp == 0) {
    // =========================== TMA producer ===============================
    if (lane == 0) {
      prefetch_tensor_map(&p.q_main);
      prefetch_tensor_map(&p.k_main);
      prefetch_tensor_map(&p.v_map);
      uint32_t kcnt = 0, vcnt = 0, qcnt[2] = {0, 0};
      bool ok = true;
      auto wait = [&](int b_, uint32_t parity) -> bool {
        return mbar_wait(bar(b_), parity, abort_flag, p.status_word, kRoleProducer + b_);
      };
      auto load_q = [&](int u) -> bool {
        const int bh_ = u / units_per_bh, b_ = bh_ / p.heads, h_ = bh_ % p.heads;
        const int x_ = -column_shift(p, 0, b_, h_);
        for (int s = 0; s < unit_slots(u); ++s) {
          const int q0 = (p.unit_tiles * (u % units_per_bh) + s) * kBlockQ;
          const uint32_t buf = qcnt[s] % TR::kQBufs, dst = s_q + (s * TR::kQBufs + buf) * TR::kTileBytes;
          const uint32_t fb = bar(TR::kBarQFull + s * TR::kQBufs + buf);
          if (!wait(TR::kBarQEmpty + s * TR::kQBufs + buf, ((qcnt[s] / TR::kQBufs) & 1u) ^ 1u)) return false;
          mbar_arrive_expect_tx(fb, TR::kTileBytes);
          tma_load_4d(dst, &p.q_main, fb, x_, q0, h_, b_);
          if constexpr (TAIL > 0) tma_load_4d(dst + TR::kMainBytes, &p.q_tail, fb, 64 + x_, q0, h_, b_);
          ++qcnt[s];
        }
        return true;
      };
      if (TR::kQBufs == 2 && static_cast<int>(blockIdx.x) < p.num_tiles) ok = load_q(blockIdx.x);
      for (int u = blockIdx.x; ok && u < p.num_tiles; u += gridDim.x) {
        const int bh = u / units_per_bh, b = bh / p.heads, h = bh % p.heads;
        const int xqk = -column_shift(p, 0, b, h), xv = -column_shift(p, 1, b, h);
        for (int j = 0; j < num_kv_blocks; ++j) {
          const int kv0 = j * kBlockKV;
          {
            const uint32_t s = kcnt % TR::kStagesK, ph = (kcnt / TR::kStagesK) & 1u;
            if (!(ok = wait(TR::kBarKEmpty + s, ph ^ 1u))) break;
            const uint32_t dst = s_k + s * TR::kTileBytes, fb = bar(TR::kBarKFull + s);
            mbar_arrive_expect_tx(fb, TR::kTileBytes);
            tma_load_4d(dst, &p.k_main, fb, xqk, kv0, h, b);
            if constexpr (TAIL > 0) tma_load_4d(dst + TR::kMainBytes, &p.k_tail, fb, 64 + xqk, kv0, h, b);
            ++kcnt;
          }
          // one query buffer per slot: the first K block goes ahead of the query tiles, which wait for the tile before
          if (TR::kQBufs == 1 && j == 0 && !(ok = load_q(u))) break;
          {
            const uint32_t s = vcnt % TR::kStagesV, ph = (vcnt / TR::kStagesV) & 1u;
            if (!(ok = wait(TR::kBarVEmpty + s, ph ^ 1u))) break;
            const uint32_t dst = s_v + s * TR::kVTileBytes, fb = bar(TR::kBarVFull + s);
            mbar_arrive_expect_tx(fb, TR::kVTileBytes);
#pragma unroll
            for (int a = 0; a < TR::kVAtoms; ++a)
              tma_load_4d(dst + a * TR::kVAtomBytes, &p.v_map, fb, a * 32 + xv, kv0, h, b);
            ++vcnt;
          }
        }
        if (TR::kQBufs == 2 && ok && u + static_cast<int>(gridDim.x) < p.num_tiles) ok = load_q(u + gridDim.x);
      }
    }
  } else if (warp == 1) {
    // ============================ MMA issuer ================================
    const bool leader = elect_one();
    auto commit = [&](int b_) { tc_commit(bar(b_), leader); };
    constexpr uint32_t idesc_qk = make_idesc(kBf16, false, false, 128, 128);
    constexpr uint32_t idesc_pv = make_idesc(kBf16, false, true, 128, DPAD);
    uint32_t kcnt = 0, vcnt = 0, qcnt[2] = {0, 0}, pcnt[2] = {0, 0};
    bool ok = true;
    auto wait = [&](int b_, uint32_t parity) -> bool {
      return mbar_wait(bar(b_), parity, abort_flag, p.status_word, kRoleMma + b_);
    };
    for (int u = blockIdx.x; ok && u < p.num_tiles; u += gridDim.x) {
      const int slots = unit_slots(u);
      uint32_t q_tile[2];
#pragma unroll
      for (int s = 0; s < 2; ++s) q_tile[s] = s_q + (s * TR::kQBufs + qcnt[s] % TR::kQBufs) * TR::kTileBytes;
      // j = -1: the first S of both slots; then per key block P V and the next S, slot by slot
      for (int j = -1; ok && j < num_kv_blocks; ++j) {
        const uint32_t sk = kcnt % TR::kStagesK, sv = vcnt % TR::kStagesV;
        const bool next_s = j + 1 < num_kv_blocks;
        if (next_s && !(ok = wait(TR::kBarKFull + sk, (kcnt / TR::kStagesK) & 1u))) break;
        if (j >= 0 && !(ok = wait(TR::kBarVFull + sv, (vcnt / TR::kStagesV) & 1u))) break;
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          if (s >= slots) break;
          const uint32_t t_s = tmem + TR::kColS + 128 * s, t_o = tmem + TR::kColO + DPAD * s;
          if (j < 0) {
            if (!(ok = wait(TR::kBarQFull + s * TR::kQBufs + qcnt[s] % TR::kQBufs, (qcnt[s] / TR::kQBufs) & 1u))) break;
            ++qcnt[s];
          } else {
            if (!(ok = wait(TR::kBarPFull + s, pcnt[s] & 1u))) break;
            ++pcnt[s];
          }
          tc_fence_after_sync();
          if (j >= 0) {
            issue_pv_atoms<TR, false>(leader, t_o, t_s, s_v + sv * TR::kVTileBytes, idesc_pv, j > 0);
            if (s == slots - 1) commit(TR::kBarVEmpty + sv);
          }
          if (next_s) {
            issue_qk<TAIL, TR>(leader, t_s, q_tile[s], s_k + sk * TR::kTileBytes, idesc_qk, false);
            commit(TR::kBarSFull + s);  // S of the next block, O up to date
            if (s == slots - 1) commit(TR::kBarKEmpty + sk);
          } else {
            commit(TR::kBarOFull + s);  // (a barrier of its own: S of the next unit does not wait for the epilogue)
          }
        }
        if (j >= 0) ++vcnt;
        if (next_s) ++kcnt;
      }
    }
  } else {
    // ===================== softmax / correction / epilogue ==================
    const int slot = (warp - 2) >> 2;
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;
    const bool issuer = warp == 2 + 4 * slot && lane == 0;  // the thread that stores this slot's output tiles
    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t t_s = tmem + lane_base + TR::kColS + 128 * slot, t_o = tmem + lane_base + TR::kColO + DPAD * slot;
    const float sl2 = p.scale_log2e;
    uint32_t scnt = 0, qcnt = 0;
    bool ok = true;
    auto wait = [&](int b_, uint32_t parity) -> bool {
      return __all_sync(0xffffffffu, mbar_wait(bar(b_), parity, abort_flag, p.status_word, kRoleSoftmax + b_));
    };
    // the buffer of the tile stored last is handed back once the store has read it; with two buffers that can wait
    // until the next tile is under way
    int pending_buf = -1;
    auto release_q = [&]() {
      if (issuer && pending_buf >= 0) {
        tma_store_wait_read();
        mbar_arrive(bar(TR::kBarQEmpty + slot * TR::kQBufs + pending_buf));
      }
      pending_buf = -1;
    };
    for (int u = blockIdx.x; ok && u < p.num_tiles; u += gridDim.x) {
      if (slot >= unit_slots(u)) continue;
      const int bh = u / units_per_bh, b = bh / p.heads, h = bh % p.heads;
      const int q0 = (p.unit_tiles * (u % units_per_bh) + slot) * kBlockQ;
      const uint32_t buf = qcnt % TR::kQBufs;
      float m_used = -CUDART_INF_F, l = 0.f, l_hi = 0.f;  // l_hi (!kCubics): the sum over key columns 64 to 127
      for (int j = 0; j < num_kv_blocks; ++j, ++scnt) {
        ok = wait(TR::kBarSFull + slot, scnt & 1u);
        if (!ok) break;
        tc_fence_after_sync();
        uint32_t r[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld_x32(t_s + c * 32, r[c]);
        tmem_wait_ld();
        float mx0 = -CUDART_INF_F, mx1 = -CUDART_INF_F, mx2 = -CUDART_INF_F, mx3 = -CUDART_INF_F;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            mx0 = max3(mx0, __uint_as_float(r[c][i]), __uint_as_float(r[c][i + 1]));
            mx1 = max3(mx1, __uint_as_float(r[c][i + 2]), __uint_as_float(r[c][i + 3]));
            mx2 = max3(mx2, __uint_as_float(r[c][i + 4]), __uint_as_float(r[c][i + 5]));
            mx3 = max3(mx3, __uint_as_float(r[c][i + 6]), __uint_as_float(r[c][i + 7]));
          }
        }
        const float m_blk = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3)) * sl2;
        if (j == 0) {
          m_used = m_blk;
        } else {
          const bool need = m_blk > m_used + kRescaleThreshold;
          if (__any_sync(0xffffffffu, need)) {  // O holds every earlier block: S of this one was issued behind them
            float alpha = 1.f;
            if (need) {
              alpha = fast_exp2(m_used - m_blk);
              m_used = m_blk;
            }
            l *= alpha;
            l_hi *= alpha;
#pragma unroll 1
            for (int c = 0; c < DPAD / 16; ++c) {
              uint32_t a[16];
              tmem_ld_x16(t_o + c * 16, a);
              tmem_wait_ld();
#pragma unroll
              for (int i = 0; i < 16; ++i) a[i] = __float_as_uint(__uint_as_float(a[i]) * alpha);
              tmem_st_x16(t_o + c * 16, a);
            }
          }
        }
        const uint64_t sl2_2 = pack_f2(sl2, sl2), neg_m2 = pack_f2(-m_used, -m_used);
        uint64_t la = pack_f2(0.f, 0.f), lb = la;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            float x0, x1, p2, p3;
            unpack_f2(fma2(pack_u2(r[c][i], r[c][i + 1]), sl2_2, neg_m2), x0, x1);
            const uint64_t xb = fma2(pack_u2(r[c][i + 2], r[c][i + 3]), sl2_2, neg_m2);
            if (kCubics && kPolyEvery > 0 && ((i / 4) % (kPolyEvery > 0 ? kPolyEvery : 1)) == (kPolyEvery - 1)) {
              poly_exp2_x2(xb, p2, p3);
            } else {
              float x2, x3;
              unpack_f2(xb, x2, x3);
              p2 = fast_exp2(x2);
              p3 = fast_exp2(x3);
            }
            const float p0 = fast_exp2(x0), p1 = fast_exp2(x1);
            la = add2(la, pack_f2(p0, p1));
            lb = add2(lb, pack_f2(p2, p3));
            pk[i / 2] = Pack2<T>::pack(p0, p1);
            pk[i / 2 + 1] = Pack2<T>::pack(p2, p3);
          }
          tmem_st_x16(t_s + c * 16, pk);  // over S columns this warp holds in registers
          if (c == 3 || (!kCubics && c == 1)) {
            float s0, s1;
            unpack_f2(add2(la, lb), s0, s1);
            (!kCubics && c == 3 ? l_hi : l) += s0 + s1;
            la = lb = pack_f2(0.f, 0.f);
          }
        }
        tmem_wait_st();
        tc_fence_before_sync();
        mbar_arrive_warp(bar(TR::kBarPFull + slot));
        if (j == 0) release_q();
      }
      // ---- end of the tile: o = O / l through the query tile's buffer, lse -----------------
      if (ok) ok = wait(TR::kBarOFull + slot, qcnt & 1u);
      ++qcnt;
      ok = named_bar_and(1 + slot, 128, ok);  // every warp of the slot arrives here, whatever happened to its waits
      if (!ok) break;
      tc_fence_after_sync();
      if constexpr (!kCubics) l += l_hi;
      const float inv_l = 1.f / l;
      p.lse[(static_cast<int64_t>(b) * p.heads + h) * p.seqlen_q + q0 + row] =
          (m_used + __log2f(l)) * 0.6931471805599453f;
      uint8_t* stage = smem + (slot * TR::kQBufs + buf) * TR::kTileBytes;
      auto chunk_off = [&](int cc) -> uint32_t {  // cc: head-dim column, a multiple of 8
        if (cc < 64) return static_cast<uint32_t>(row * 128 + (((cc >> 3) ^ (row & 7)) << 4));
        const int ct = (cc - 64) >> 3;
        if constexpr (TAIL == 64) return static_cast<uint32_t>(TR::kMainBytes + row * 128 + ((ct ^ (row & 7)) << 4));
        else if constexpr (TAIL == 32) return static_cast<uint32_t>(TR::kMainBytes + row * 64 + ((ct ^ ((row >> 1) & 3)) << 4));
        else return static_cast<uint32_t>(TR::kMainBytes + row * 32 + ((ct ^ ((row >> 2) & 1)) << 4));
      };
      const int shift = column_shift(p, 1, b, h);  // accumulator column c is head-dim column c - shift
#pragma unroll
      for (int c = 0; c < DPAD / 16; ++c) {
        uint32_t a[16];
        tmem_ld_x16(t_o + c * 16, a);
        tmem_wait_ld();
        uint32_t po[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
          po[i] = Pack2<T>::pack(__uint_as_float(a[2 * i]) * inv_l, __uint_as_float(a[2 * i + 1]) * inv_l);
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          const int col = c * 16 + hh * 8 - shift;
          if (col >= 0)
            *reinterpret_cast<uint4*>(stage + chunk_off(col)) = make_uint4(po[4 * hh], po[4 * hh + 1], po[4 * hh + 2], po[4 * hh + 3]);
        }
      }
      tc_fence_before_sync();
      fence_proxy_async_smem();
      named_bar_sync(1 + slot, 128);
      if (issuer) {
        tma_store_4d(&p.o_main, smem_u32(stage), 0, q0, h, b);
        if constexpr (TAIL > 0) tma_store_4d(&p.o_tail, smem_u32(stage) + TR::kMainBytes, 64, q0, h, b);
        tma_store_commit();
      }
      pending_buf = buf;
      if (TR::kQBufs == 1) release_q();
    }
    if (issuer) tma_store_wait_all();
  }

  // ============================== teardown ==================================
  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (warp == 0) tmem_dealloc(tmem, TR::kTmemCols);
}

}  // namespace dmf
