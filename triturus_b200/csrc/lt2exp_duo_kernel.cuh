// lt2exp in plain TF32 on tiles of 128 rows s x 256 columns k, the generated operand in tensor memory, two k-blocks per stage.
//
// The arithmetic and the roles of lt2exp_tmem_kernel.cuh (D^T[k, s] = P^T * W^T; replaces triturus/lt2exp.py:227-357 and
// :365-506): the tile is two 128-column blocks that share every tile of w, two M = 128 MMAs per k-step.  There a k-block
// is 512 cycles of MMAs and took 730: the MMA issuer needs some 200 cycles from one stage to the next (the barrier, the fence, the
// election, the descriptors), and the tensor core, which queues no more than an MMA or two, stands still meanwhile.  Here a
// stage holds the k-blocks of two consecutive rows i, the issuer asks for the next stage in the middle of one, and the
// tiles of w have a ring of their own, four stages deep, beside the two operand stages that tensor memory has room for:
// 1 075 to 1 160 cycles per stage of 1 024.  us in a loop: R16 128x64x64x2048 74.8 -> 61.6, R8 100x100x100x3000 167 -> 142, R30
// 128x64x64x2048 132 -> 108; with other inputs in every pass the first 71.9 -> 63.8.  What is left of the first (102 000 cycles): 13 300 before the first MMA, which are HBM's (a, b and the first
// tiles of w of all SMs at once), 2 900 where the j-chunk changes, 7 900 in the epilogue.
//
// TMEM: [0, 256) accumulators of the two blocks, then two operand stages of [block][row of the pair][32 j] = 128 columns.
// Barriers of stages are rings of four (index = stage counter `it` % 4, phase it / 4).  The producer of w waits for the commit of
// the MMAs of stage it - 4, the transform for that of it - 2; that is enough for the barriers as well (lm2exp_pair3x_kernel.cuh).
//
//   warp 0      TMA producer: w boxes {32 j, 1 i, 128 s, 1 r}, 128-byte swizzle.
//   warp 1      TMEM allocation; the warp walks the stages and one elected lane issues tcgen05.mma.kind::tf32 with A in TMEM.
//   warps 4-7   epilogue: out[s, k] = m[k] + log(acc), or fp32 reductions into the zero-filled result when the contraction is split.
//   warps 8-15  transform: warp w writes TMEM lane quarter w % 4 of block (w - 8) / 4.  Column maxima first.
#pragma once

#include "lt2exp_tmem_kernel.cuh"

namespace tb200 {

struct Lt2expDuoCfg {
  static constexpr int BM = 128, BK = 32, NB = 2, BN = 128 * NB, MT = 1, PREC = 0, NTW = 8, RING = 4;
  static constexpr bool PROMOTE = false;
  static constexpr int CHUNK = 1 << 30;
  static constexpr int W_TILE = BM * BK * 4, STAGE = 2 * W_TILE;
  static constexpr int BLK_COLS = BM;
  static constexpr int P_COL0 = NB * BLK_COLS, P_STAGE = NB * 2 * BK, NSP = 2;  // operand columns of a stage, stages
  static constexpr int TMEM_COLS = 512;
  static constexpr int NTHREADS = (8 + NTW) * 32, NTT = NTW * 32;
  static constexpr int CQ = BN / 4, RG = NTT / CQ, MPART = 2 * RG * BN;
  static constexpr int NBAR = 2 * RING + 5;
  static constexpr int EPI_STAGE = 4 * 2 * 32 * 128;  // per epilogue warp two 32 x 32 boxes
  static constexpr int SMEM_BYTES = 1024 + RING * STAGE + EPI_STAGE + 2 * BN * 4 + 2 * MPART * 4 + NBAR * 8 + 64;
  static_assert(P_COL0 + NSP * P_STAGE <= TMEM_COLS, "TMEM capacity");
  static_assert(NTT == BN, "a transform thread per column");
  static_assert(SMEM_BYTES <= 232448, "shared memory capacity");
};

__global__ void __launch_bounds__(Lt2expDuoCfg::NTHREADS, 1) lt2exp_duo_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ Lt2expParams p) {
  using Cfg = Lt2expDuoCfg;
  constexpr int BM = Cfg::BM, BN = Cfg::BN, BK = Cfg::BK, RING = Cfg::RING;
  constexpr int PF = 8;  // prefetch distance (rows i) for the a values

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* stage_base = smem;
  uint8_t* epi_stage = smem + RING * Cfg::STAGE;
  float* msum = reinterpret_cast<float*>(epi_stage + Cfg::EPI_STAGE);  // [2][BN]: ma + mb of the tile's columns
  float* mpart = msum + 2 * BN;                                      // [2][2][RG][BN] partial column maxima
  uint64_t* bars = reinterpret_cast<uint64_t*>(mpart + 2 * Cfg::MPART);
  uint64_t* full = bars;         // [4] tiles of w landed and operand stage written to TMEM
  uint64_t* done = bars + RING;  // [4] MMAs of the stage retired
  uint64_t* acc_full = bars + 2 * RING;
  uint64_t* acc_empty = acc_full + 1;
  uint64_t* msum_empty = acc_empty + 1;  // [2]
  uint64_t* mx_bar = msum_empty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mx_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = warp_uniform(threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const AbortCtl ctl{abort_flag, p.status};

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < RING; ++s) {
      mbar_init(&full[s], 1 + Cfg::NTW);
      mbar_init(&done[s], 1);
    }
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, 4);
    for (int s = 0; s < 2; ++s) mbar_init(&msum_empty[s], 4);
    mbar_init(mx_bar, Cfg::NTW);
    fence_mbar_init();
    tma_prefetch_desc(&tmap_w);
    if (p.out_tma) tma_prefetch_desc(&p.tmap_out);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = warp_uniform(*tmem_slot);

  const int JC = (p.J + BK - 1) / BK;
  const int KBT = JC * p.I;  // k-blocks per output tile
  const bool split_mode = p.nsplit > 1 || p.stream != 0;
  if (split_mode) pdl_launch_dependents();  // the log pass takes its column maxima meanwhile

  // Output tile -> (r, n0 = first column k, s0 = first row s); the items of a CTA come from LtWork.
  auto decode = [&](int tile, int& r, int& n0, int& s0) {
    const int tm = tile % p.tiles_m;
    const int rest = tile / p.tiles_m;
    const int tn = rest % p.tiles_n;
    r = rest / p.tiles_n;
    n0 = tn * BN;
    s0 = tm * BM;
  };
  // The commit of stage `it - back`.
  auto wait_done = [&](uint32_t it, uint32_t back, int code, bool warp_wide) -> bool {
    if (it < back) return true;
    const uint32_t x = it - back;
    return warp_wide ? mbar_wait_warp(&done[x % RING], (x / RING) & 1, ctl, code) : mbar_wait(&done[x % RING], (x / RING) & 1, ctl, code);
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      LtWork work(p, KBT);
      for (LtItem w; ok && work.next(w);) {
        int r, n0, s0;
        decode(w.tile, r, n0, s0);
        for (int jc = w.kb_lo / p.I; ok && jc * p.I < w.kb_hi; ++jc) {
          const int i_hi = lt_row_hi(w, jc, p.I);
          for (int i = lt_row_lo(w, jc, p.I); i < i_hi; i += 2, ++it) {
            if (!(ok = wait_done(it, RING, STATUS_TIMEOUT_PRODUCER, false))) break;
            const bool two = i + 1 < i_hi;
            uint64_t* landed = &full[it % RING];
            uint8_t* dst = stage_base + (it % RING) * Cfg::STAGE;
            mbar_arrive_expect_tx(landed, two ? Cfg::STAGE : Cfg::W_TILE);
            tma_load_4d(dst, &tmap_w, landed, jc * BK, i, s0, r);
            if (two) tma_load_4d(dst + Cfg::W_TILE, &tmap_w, landed, jc * BK, i + 1, s0, r);
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (see lt2exp_tmem_kernel.cuh)
    constexpr uint32_t idesc = umma_idesc_tf32(128, BM);  // M = 128 columns k, N = rows s
    const uint64_t dw0 = umma_desc_k_sw128(smem_u32(stage_base));
    uint32_t it = 0, tcount = 0;
    bool ok = true, ready = false;
    LtWork work(p, KBT);
    for (LtItem w; ok && work.next(w); ++tcount) {
      if (!(ok = mbar_wait_warp(acc_empty, (tcount & 1) ^ 1, ctl, STATUS_TIMEOUT_MMA))) break;
      tc_fence_after_sync();
      bool first = true;
      for (int jc = w.kb_lo / p.I; ok && jc * p.I < w.kb_hi; ++jc) {
        const int i_hi = lt_row_hi(w, jc, p.I);
        for (int i = lt_row_lo(w, jc, p.I); i < i_hi; i += 2, ++it) {
          const uint32_t st = it % RING, nx = (it + 1) % RING;
          if (!ready) {
            if (!(ok = mbar_wait_warp(&full[st], (it / RING) & 1, ctl, STATUS_TIMEOUT_MMA))) break;
          }
          tc_fence_after_sync();
          const uint64_t dw = dw0 + st * (Cfg::STAGE >> 4);
          const uint32_t pa = tmem_base + Cfg::P_COL0 + (it % Cfg::NSP) * Cfg::P_STAGE;
          if (elect_one_sync()) {
#pragma unroll
            for (int blk = 0; blk < Cfg::NB; ++blk) {  // the column blocks share the w tile
#pragma unroll
              for (int ks = 0; ks < BK / 8; ++ks)
                umma_tf32_ts(tmem_base + blk * Cfg::BLK_COLS, pa + blk * 2 * BK + ks * 8, dw + 2 * ks, idesc, (!first || ks > 0) ? 1u : 0u);
            }
          }
          // The tensor core takes the next MMA only when it is about done with the one before, so what this warp does between
          // two stages is lost to it: the next stage's barrier is asked here, in the middle of this one.
          const bool peek = mbar_try_wait(&full[nx], ((it + 1) / RING) & 1);
          if (elect_one_sync()) {
            if (i + 1 < i_hi) {
#pragma unroll
              for (int blk = 0; blk < Cfg::NB; ++blk) {
#pragma unroll
                for (int ks = 0; ks < BK / 8; ++ks)
                  umma_tf32_ts(tmem_base + blk * Cfg::BLK_COLS, pa + blk * 2 * BK + BK + ks * 8, dw + (Cfg::W_TILE >> 4) + 2 * ks, idesc, 1u);
              }
            }
            umma_commit(&done[st]);
          }
          ready = __all_sync(0xffffffffu, peek);
          first = false;
        }
      }
      if (ok && elect_one_sync()) umma_commit(acc_full);
      __syncwarp();
    }
  } else if (warp >= 4 && warp < 8) {
    // ------------------------------------------------------------------ epilogue
    const int q = warp & 3;
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
    if (split_mode) pdl_wait();  // the zero-filled result
    const bool use_tma = p.out_tma != 0 && !split_mode;
    uint32_t nbox = 0;
    uint32_t tcount = 0;
    bool ok = true;
    LtWork work(p, KBT);
    for (LtItem w; ok && work.next(w); ++tcount) {
      int r, n0, s0;
      decode(w.tile, r, n0, s0);
      const int slot = tcount & 1;
      if (!(ok = mbar_wait_warp(acc_full, tcount & 1, ctl, STATUS_TIMEOUT_EPILOGUE))) break;
      tc_fence_after_sync();
#pragma unroll 1
      for (int blk = 0; blk < Cfg::NB; ++blk) {  // column blocks of the tile: this lane's column in each
        const int k0 = n0 + blk * 128 + q * 32, kcol = k0 + lane;
        const bool col_ok = kcol < p.K;
        float* out_col = p.out + static_cast<int64_t>(r) * p.out_s0 + kcol;
        const float m = msum[slot * BN + blk * 128 + q * 32 + lane];
        float cmx = -INFINITY;  // running maximum of this lane's column over the rows of the tile
        // One chunk = 32 rows s for this lane's column: through a staging box (the 32 lanes of a store fill one row in the
        // 128-byte swizzle) and from there as one TMA store, clipped at the edges of the result.  Row by row from the registers
        // a chunk took 2 600 cycles (all of the tile's stores at once, and 20 KB of unrolled code), now 960.
        const uint32_t acc0 = lane_base + blk * Cfg::BLK_COLS;
#pragma unroll 1
        for (int c = 0; c < Cfg::BLK_COLS / 32; ++c) {
          const int sb = s0 + c * 32;
          if (sb >= p.S) break;
          uint32_t v[32];
          tmem_ld_32x32(acc0 + c * 32, v);
          uint8_t* stg = epi_stage + q * 8192 + (nbox & 1) * 4096;
          if (use_tma && lane == 0) tma_store_wait_read<1>();  // the store before the previous one has read this box out
          tmem_ld_wait();
          if (split_mode) {
#pragma unroll
            for (int e = 0; e < 32; ++e) {
              if (col_ok && sb + e < p.S) atomicAdd(out_col + static_cast<int64_t>(sb + e) * p.out_s1, __uint_as_float(v[e]));
            }
            continue;
          }
          __syncwarp();
          const int nrows = p.S - sb;
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            const float o = m + lg2_approx(__uint_as_float(v[e])) * LN2_F;
            if (e < nrows) cmx = fmaxf(cmx, o);
            v[e] = __float_as_uint(o);
          }
          if (use_tma) {
            ++nbox;
#pragma unroll
            for (int e = 0; e < 32; ++e) *reinterpret_cast<uint32_t*>(stg + sw128_offset(e, lane)) = v[e];
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0 && k0 < p.K) {
              tma_store_3d(&p.tmap_out, stg, k0, sb, r);
              tma_store_commit();
            }
          } else {
#pragma unroll
            for (int e = 0; e < 32; ++e) {
              if (col_ok && e < nrows) out_col[static_cast<int64_t>(sb + e) * p.out_s1] = __uint_as_float(v[e]);
            }
          }
        }
        if (p.out_max != nullptr && !split_mode && col_ok) {
          // the next layer's stabiliser: this lane owns the column, so the maximum is a register
          float* dst = p.out_max + static_cast<int64_t>(r) * p.K + kcol;
          if (p.tiles_m == 1) *dst = cmx;
          else red_max_f32(dst, cmx);
        }
      }
      tmem_ld_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(acc_empty);
        mbar_arrive(&msum_empty[slot]);
      }
    }
    if (use_tma && lane == 0) tma_store_wait_all();  // shared memory must outlive the last box
  } else if (warp >= 8) {
    // ------------------------------------------------------------------ transform: operand generator
    const int tt = threadIdx.x - 8 * 32;
    const int n = tt;  // column of the tile owned by this thread
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + Cfg::P_COL0 + static_cast<uint32_t>((tt / 128) * 2 * BK);
    uint32_t it = 0, tcount = 0;
    bool ok = true;
    if (p.ma_wait) pdl_wait();
    LtWork work(p, KBT);
    for (LtItem w; ok && work.next(w); ++tcount) {
      int r, n0, s0;
      decode(w.tile, r, n0, s0);
      const int kcol = n0 + n;
      const bool col_ok = kcol < p.K;
      const float* a_col = p.a + static_cast<int64_t>(r) * p.a_s0 + static_cast<int64_t>(kcol) * p.a_s2;
      const float* b_col = p.b + static_cast<int64_t>(r) * p.b_s0 + static_cast<int64_t>(kcol) * p.b_s2;

      // Column maxima over the full I and J (see lt2exp_kernel.cuh).
      float* part = mpart + (tcount & 1) * Cfg::MPART;
      int nparts = 0;
      if (p.ma_in != nullptr) {
        // maxima supplied by the caller: no scan
      } else if (p.vec_ab) {
        const int q4 = tt % Cfg::CQ, rg = tt / Cfg::CQ;
        float4 pa = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY), pb = pa;
        if (n0 + 4 * q4 < p.K) {
          pa = quad_column_max(p.a + static_cast<int64_t>(r) * p.a_s0 + n0 + 4 * q4, p.a_s1, p.I, rg, Cfg::RG);
          pb = quad_column_max(p.b + static_cast<int64_t>(r) * p.b_s0 + n0 + 4 * q4, p.b_s1, p.J, rg, Cfg::RG);
        }
        *reinterpret_cast<float4*>(part + rg * BN + 4 * q4) = pa;
        *reinterpret_cast<float4*>(part + (Cfg::RG + rg) * BN + 4 * q4) = pb;
        nparts = Cfg::RG;
      } else {
        part[n] = col_ok ? strided_column_max(a_col, p.a_s1, p.I, 0, 1) : -INFINITY;
        part[Cfg::RG * BN + n] = col_ok ? strided_column_max(b_col, p.b_s1, p.J, 0, 1) : -INFINITY;
        nparts = 1;
      }
      // The b values of the first j-chunk are on their way while the blocks' maxima meet.
      float eb[32];
      auto load_b = [&](int jc) {
#pragma unroll
        for (int x = 0; x < 32; ++x) {
          const int j = jc * BK + x;
          eb[x] = -INFINITY;  // padding (past J or K) enters the exp as -inf: exact zero
          if (col_ok && j < p.J) eb[x] = __ldg(b_col + static_cast<int64_t>(j) * p.b_s1);
        }
      };
      const int jc0 = w.kb_lo / p.I;
      load_b(jc0);
      float ma = -INFINITY, mb = -INFINITY;
      if (p.ma_in != nullptr) {
        if (col_ok) {
          ma = __ldg(p.ma_in + static_cast<int64_t>(r) * p.K + kcol);
          mb = __ldg(p.mb_in + static_cast<int64_t>(r) * p.K + kcol);
        }
      } else {
        __syncwarp();
        if (lane == 0) mbar_arrive(mx_bar);
        if (!(ok = mbar_wait_warp(mx_bar, tcount & 1, ctl, STATUS_TIMEOUT_TRANSFORM))) break;
        for (int g = 0; g < nparts; ++g) {
          ma = fmaxf(ma, part[g * BN + n]);
          mb = fmaxf(mb, part[(Cfg::RG + g) * BN + n]);
        }
      }
      ma = clamp_stab(ma);
      mb = clamp_stab(mb);
      const int slot = tcount & 1;
      // (the operand stages order this write before the epilogue's read)
      if (!(ok = mbar_wait_warp(&msum_empty[slot], ((tcount >> 1) & 1) ^ 1, ctl, STATUS_TIMEOUT_TRANSFORM))) break;
      msum[slot * BN + n] = ma + mb;

      for (int jc = jc0; ok && jc * p.I < w.kb_hi; ++jc) {
        const int i_lo = lt_row_lo(w, jc, p.I);
        const int In = lt_row_hi(w, jc, p.I) - i_lo;  // rows of this j-chunk in the item
        const float* a_sl = a_col + static_cast<int64_t>(i_lo) * p.a_s1;
        if (jc > jc0) load_b(jc);
        float apf[PF];
#pragma unroll
        for (int x = 0; x < PF; ++x) apf[x] = (col_ok && x < In) ? __ldg(a_sl + static_cast<int64_t>(x) * p.a_s1) : -INFINITY;
#pragma unroll
        for (int x = 0; x < 32; ++x) eb[x] = exp_shifted(eb[x], mb);
        for (int ib = 0; ok && ib < In; ib += PF) {
          float ea[PF];
#pragma unroll
          for (int x = 0; x < PF; ++x) {
            ea[x] = exp_shifted(apf[x], ma);
            const int i = ib + PF + x;
            apf[x] = (col_ok && i < In) ? __ldg(a_sl + static_cast<int64_t>(i) * p.a_s1) : -INFINITY;
          }
#pragma unroll
          for (int x = 0; x < PF; x += 2) {
            const int i = ib + x;
            if (i >= In) break;
            const uint32_t stage = lane_base + (it % Cfg::NSP) * Cfg::P_STAGE;
            uint32_t pv[32];
#pragma unroll
            for (int e = 0; e < 32; ++e) pv[e] = tf32_round_bits(ea[x] * eb[e]);
            if (!(ok = wait_done(it, Cfg::NSP, STATUS_TIMEOUT_TRANSFORM, true))) break;
            tc_fence_after_sync();
            tmem_st_32x32(stage, pv);
            if (i + 1 < In) {
#pragma unroll
              for (int e = 0; e < 32; ++e) pv[e] = tf32_round_bits(ea[x + 1] * eb[e]);
              tmem_st_32x32(stage + BK, pv);
            }
            tmem_st_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[it % RING]);
            ++it;
          }
        }
      }
    }
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000LL) {
    }
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

}  // namespace tb200
