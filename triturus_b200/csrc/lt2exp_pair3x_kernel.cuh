// lt2exp in 3xTF32 on CTA pairs: tiles of 256 columns k x up to 192 rows s, the generated operand in tensor memory.
//
// The arithmetic of lt2exp_tmem_kernel.cuh (D^T[k, s] = P^T * W^T, chunks of 24 k-blocks re-summed in a master copy; replaces
// triturus/lt2exp.py:227-357 and :365-506) on the structure of lm2exp_pair3x_kernel.cuh: M = 256 columns k over the pair (128 per CTA =
// the CTA's TMEM lanes), N = the tile's rows s, half of them in each CTA's shared memory, two accumulators of 192 columns and two
// operand stages of 64.  There a CTA of its own works on 128 x 128 and its tensor core stands still for a quarter of every
// k-block of 768 cycles, while the issuer goes from one stage to the next; a k-block of 192 rows is 1 152 cycles, and every tile of w
// is fetched, split and read by half as many SMs.  Measured per k-block, all pairs busy (R74, K = 256): 0.72 us with 192
// rows, 0.52 with 128, 0.43 with 32, where the transform warps bound it.  us, 128 x 128 tiles -> pairs: R32 256^4 1 194 -> 1 169 in a
// sustained loop (1 105 -> 1 044 before the power limit sets in), R8 256x128x128x4096 969 -> 914, R40 64x90x200x500 407 -> 341, R1 256^4
// 65.9 -> 59.3; which of the two a call takes is lt2exp_pair3x_wins in api.cu.
//
// The rows of S are cut into even tiles of whole units of 32 (p.tiles_m of them); the items of a pair come from LtWork, pairs in
// the place of CTAs.  Rings as in lm2exp_pair3x_kernel.cuh: barriers of k-blocks in rings of eight, TMEM stage it % 2,
// shared-memory stage of w it % 4, and who overwrites a stage waits for the commit of the k-block that used it last.
//
//   warp 0      TMA producer: w boxes {32 j, 1 i, half of the tile's rows s, 1 r}, 128-byte swizzle.
//   warp 1      TMEM allocation; in the leader CTA the warp walks the k-blocks and one elected lane issues the pair MMAs.
//   warps 4-7   epilogue: re-summation of finished chunks; out[s, k] = m[k] + log(acc), or parked sums, or reductions into the zero-filled
//               result when the contraction is split (lt2exp_tmem_kernel.cuh).
//   warps 8-15  transform: two groups of four warps (one per lane quarter) take alternate k-blocks.  Column maxima first.
//   warps 16-19 the low parts of the w tiles.
#pragma once

#include "lm2exp_tspair_kernel.cuh"
#include "lt2exp_tmem_kernel.cuh"
#include "row_tiles.cuh"

namespace tb200 {

struct Lt2expPair3xCfg {
  static constexpr int CTAS = 2;
  static constexpr int BM = 192, MT = 1;           // rows s per tile at most
  static constexpr int UNITS = BM / 32;
  static constexpr int BN = 256, CTA_COLS = 128;   // columns k per tile and per CTA
  static constexpr int BK = 32, PREC = 1, NTW = 8, NPW = 4, NGROUPS = 2, RING = 8;
  static constexpr bool PROMOTE = true;
  static constexpr int CHUNK = 24;                 // k-blocks
  static constexpr int NSP = 2, NSW = 4;           // stages: operand (tensor memory), w
  static constexpr int W_TILE = BM / 2 * BK * 4, STAGE = 2 * W_TILE;  // this CTA's rows of a tile of w, and their low parts
  static constexpr int P_STAGE = 2 * BK, P_COL0 = 2 * BM, TMEM_COLS = 512;
  static constexpr int NTHREADS = (8 + NTW + NPW) * 32, NTT = NTW * 32;
  static constexpr int CQ = CTA_COLS / 4, RG = NTT / CQ, MPART = 2 * RG * CTA_COLS;
  static constexpr int MASTER = BM * CTA_COLS * 4;
  static constexpr int NBAR = 3 * RING + 9;
  static constexpr int SMEM_BYTES = 1024 + NSW * STAGE + MASTER + 2 * CTA_COLS * 4 + 2 * MPART * 4 + NBAR * 8 + 64;
  static_assert(P_COL0 + NSP * P_STAGE <= TMEM_COLS, "TMEM capacity");
  static_assert(NSP == NGROUPS, "an operand stage belongs to one transform group");
  static_assert(SMEM_BYTES <= 232448, "shared memory capacity");
};

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(Lt2expPair3xCfg::NTHREADS, 1)
lt2exp_pair3x_kernel(const __grid_constant__ CUtensorMap tmap_w, const Lt2expParams p) {
  using Cfg = Lt2expPair3xCfg;
  constexpr int BM = Cfg::BM, BN = Cfg::CTA_COLS, BK = Cfg::BK, NG = Cfg::NGROUPS;
  constexpr int PF = 4;  // prefetch distance (own k-blocks) for the a values
  constexpr uint32_t RING = Cfg::RING;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* stage_base = smem;
  // [BM / 4 row quads][128 columns][4] master copy of the accumulator, each thread its own column
  float4* master = reinterpret_cast<float4*>(smem + Cfg::NSW * Cfg::STAGE);
  float* msum = reinterpret_cast<float*>(smem + Cfg::NSW * Cfg::STAGE + Cfg::MASTER);  // [2][BN]: ma + mb of the tile's columns
  float* mpart = msum + 2 * BN;                                                          // [2][2][RG][BN] partial column maxima
  uint64_t* bars = reinterpret_cast<uint64_t*>(mpart + 2 * Cfg::MPART);
  uint64_t* w_full = bars;               // [8] this CTA's rows of the w tile landed
  uint64_t* xf_done = bars + RING;       // [8] (leader's copy is used) operand stage and low parts written, both CTAs
  uint64_t* kb_done = bars + 2 * RING;   // [8] MMAs of the k-block retired (committed by the leader)
  uint64_t* acc_full = bars + 3 * RING;  // [2] (committed by the leader)
  uint64_t* acc_empty = acc_full + 2;    // [2] (leader's copy is used)
  uint64_t* msum_full = acc_empty + 2;   // [2]
  uint64_t* msum_empty = msum_full + 2;  // [2]
  uint64_t* mx_bar = msum_empty + 2;     // [1]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mx_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = warp_uniform(threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const uint32_t rank = warp_uniform(cluster_ctarank());
  const bool leader = rank == 0;
  const AbortCtl ctl{abort_flag, p.status};

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (uint32_t s = 0; s < RING; ++s) {
      mbar_init(&w_full[s], 1);
      mbar_init(&xf_done[s], 2 * (4 + Cfg::NPW));
      mbar_init(&kb_done[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&acc_full[s], 1);
      mbar_init(&acc_empty[s], 8);
      mbar_init(&msum_full[s], 4);
      mbar_init(&msum_empty[s], 4);
    }
    mbar_init(mx_bar, Cfg::NTW);
    fence_mbar_init();
    tma_prefetch_desc(&tmap_w);
  }
  // (both CTAs run before the pair allocation, and hold their tensor memory before the roles start)
  cluster_sync_all();
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, Cfg::TMEM_COLS);
    tmem_relinquish_pair();
  }
  tc_fence_before_sync();
  cluster_sync_all();
  tc_fence_after_sync();
  const uint32_t tmem_base = warp_uniform(*tmem_slot);

  const int JC = (p.J + BK - 1) / BK;
  const int KBT = JC * p.I;  // k-blocks per output tile
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
  const int units = (p.S + 31) / 32;
  const bool parking = p.stream != 0 && p.park != nullptr;  // shared tiles are completed through scratch memory
  const bool split_mode = (p.nsplit > 1 || p.stream != 0) && !parking;
  if (split_mode) pdl_launch_dependents();  // the log pass takes its column maxima meanwhile

  // Output tile -> r, this CTA's first column, first row s, rows (a multiple of 32).
  auto decode = [&](int tile, int& r, int& n0, int& s0, int& rows) {
    const int tm = tile % p.tiles_m;
    const int rest = tile / p.tiles_m;
    const int tn = rest % p.tiles_n;
    r = rest / p.tiles_n;
    n0 = tn * 2 * BN + static_cast<int>(rank) * BN;
    const RowTile t = row_tile(units, p.tiles_m, tm);
    s0 = t.first * 32;
    rows = t.units * 32;
  };
  // The commit of k-block `it - back`.
  auto wait_kb = [&](uint32_t it, uint32_t back, int code, bool warp_wide) -> bool {
    if (it < back) return true;
    const uint32_t x = it - back;
    return warp_wide ? mbar_wait_warp(&kb_done[x % RING], (x / RING) & 1, ctl, code) : mbar_wait(&kb_done[x % RING], (x / RING) & 1, ctl, code);
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      LtWork work(p, KBT, pair, npairs);
      for (LtItem w; ok && work.next(w);) {
        int r, n0, s0, rows;
        decode(w.tile, r, n0, s0, rows);
        const int my_s0 = s0 + static_cast<int>(rank) * (rows / 2);  // (the box may have more rows than this tile)
        for (int jc = w.kb_lo / p.I; ok && jc * p.I < w.kb_hi; ++jc) {
          const int i_hi = lt_row_hi(w, jc, p.I);
          for (int i = lt_row_lo(w, jc, p.I); i < i_hi; ++i, ++it) {
            if (!(ok = wait_kb(it, Cfg::NSW, STATUS_TIMEOUT_PRODUCER, false))) break;
            uint64_t* landed = &w_full[it % RING];
            mbar_arrive_expect_tx(landed, static_cast<uint32_t>(p.box_rows) * 128u);
            tma_load_4d(stage_base + (it % Cfg::NSW) * Cfg::STAGE, &tmap_w, landed, jc * BK, i, my_s0, r);
          }
        }
      }
      // The leader's commits arrive on both CTAs' barriers: this CTA stays until the last ones are in.
      for (uint32_t d = ok ? min(it, RING) : 0u; ok && d > 0; --d) ok = wait_kb(it, d, STATUS_TIMEOUT_PRODUCER, false);
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ pair MMA issuer (leader CTA only)
    if (leader) {
      const uint64_t dw0 = umma_desc_k_sw128(smem_u32(stage_base));
      constexpr uint32_t STAGE_ENC = Cfg::STAGE >> 4, LO_ENC = Cfg::W_TILE >> 4;
      uint32_t it = 0, ccount = 0;  // k-blocks and accumulation chunks issued so far
      bool ok = true;
      LtWork work(p, KBT, pair, npairs);
      for (LtItem w; ok && work.next(w);) {
        int r, n0, s0, rows;
        decode(w.tile, r, n0, s0, rows);
        const uint32_t idesc = umma_idesc_tf32(2 * BN, rows);  // M = 256 columns k, N = rows s
        const int KB = w.kb_hi - w.kb_lo;
        for (int kb = 0; ok && kb < KB; ++ccount) {
          const int kb0 = kb, kb_end = min(KB, kb0 + Cfg::CHUNK);
          const uint32_t buf = ccount & 1;
          if (!(ok = mbar_wait_warp(&acc_empty[buf], ((ccount >> 1) & 1) ^ 1, ctl, STATUS_TIMEOUT_MMA))) break;
          tc_fence_after_sync();
          const uint32_t d = tmem_base + buf * BM;
          for (; kb < kb_end; ++kb, ++it) {
            if (!(ok = mbar_wait_warp(&xf_done[it % RING], (it / RING) & 1, ctl, STATUS_TIMEOUT_MMA))) break;
            tc_fence_after_sync();
            if (elect_one_sync()) {
              const uint64_t dw = dw0 + (it % Cfg::NSW) * STAGE_ENC;
              const uint32_t pa = tmem_base + Cfg::P_COL0 + (it % Cfg::NSP) * Cfg::P_STAGE;
              // the corrections first, while the accumulator of a chunk is empty and does not truncate them to its bits
#pragma unroll
              for (int ks = 0; ks < BK / 8; ++ks)
                umma_tf32_ts_pair(d, pa + BK + ks * 8, dw + 2 * ks, idesc, (kb > kb0 || ks > 0) ? 1u : 0u);
#pragma unroll
              for (int ks = 0; ks < BK / 8; ++ks) umma_tf32_ts_pair(d, pa + ks * 8, dw + LO_ENC + 2 * ks, idesc, 1u);
#pragma unroll
              for (int ks = 0; ks < BK / 8; ++ks) umma_tf32_ts_pair(d, pa + ks * 8, dw + 2 * ks, idesc, 1u);
              umma_commit_pair_mcast(smem_u32(&kb_done[it % RING]), 3);
            }
            __syncwarp();
          }
          if (ok && elect_one_sync()) umma_commit_pair_mcast(smem_u32(&acc_full[buf]), 3);
          __syncwarp();
        }
      }
    }
    __syncwarp();
  } else if (warp >= 4 && warp < 8) {
    // ------------------------------------------------------------------ epilogue (this CTA's 128 columns k)
    const int q = warp & 3;
    const int kl = q * 32 + lane;  // this lane's column
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
    const uint32_t acc_empty_leader0 = map_to_cta(smem_u32(acc_empty), 0);
    if (split_mode) pdl_wait();  // the zero-filled result
    uint32_t tcount = 0, ccount = 0;
    bool ok = true;
    // (see lt2exp_tmem_kernel.cuh: whichever warp parks the last part of its columns adds the parts up)
    const int shared_parts = p.lw_parts > 0 ? p.lw_parts : p.lw_main < KBT ? 2 : 1;
    LtWork work(p, KBT, pair, npairs);
    for (LtItem w; ok && work.next(w); ++tcount) {
      int r, n0, s0, rows;
      decode(w.tile, r, n0, s0, rows);
      const int kcol = n0 + kl;
      const bool col_ok = kcol < p.K;
      float* out_col = p.out + static_cast<int64_t>(r) * p.out_s0 + kcol;
      const int slot = tcount & 1;
      const int nch = (w.kb_hi - w.kb_lo + Cfg::CHUNK - 1) / Cfg::CHUNK;
      const bool park_it = parking && w.tile >= p.lw_first && shared_parts > 1;
      const int shared_tile = w.tile - p.lw_first;
      constexpr int PARK_TILE = BM * BN;  // floats per parked part and CTA, in the order of `master`
      float4* const parked =
          reinterpret_cast<float4*>(p.park + (static_cast<int64_t>(shared_tile) * 2 + static_cast<int>(rank)) * shared_parts * PARK_TILE) + kl;
      float cmx = -INFINITY;  // running maximum of this lane's column over the rows of the tile
      for (int ch = 0; ok && ch < nch; ++ch, ++ccount) {
        const uint32_t buf = ccount & 1;
        const bool first = ch == 0, last = ch == nch - 1;
        if (!(ok = mbar_wait_warp(&acc_full[buf], (ccount >> 1) & 1, ctl, STATUS_TIMEOUT_EPILOGUE))) break;
        if (first && !(ok = mbar_wait_warp(&msum_full[slot], (tcount >> 1) & 1, ctl, STATUS_TIMEOUT_EPILOGUE))) break;
        tc_fence_after_sync();
        const float m = msum[slot * BN + kl];
#pragma unroll 1
        for (int c = 0; c < rows / 32; ++c) {
          const int sb = s0 + c * 32;
          uint32_t v[32];
          tmem_ld_32x32(lane_base + buf * BM + c * 32, v);
          float4* mst = master + c * 8 * 128 + kl;
          tmem_ld_wait();
          if (!first) {
#pragma unroll
            for (int g = 0; g < 8; ++g) add_quad(v, g, mst[g * 128]);
          }
          if (!last || park_it) {
            float4* dst = last ? parked + w.part * (PARK_TILE / 4) + c * 8 * 128 : mst;
#pragma unroll
            for (int g = 0; g < 8; ++g)
              dst[g * 128] = make_float4(__uint_as_float(v[g * 4]), __uint_as_float(v[g * 4 + 1]), __uint_as_float(v[g * 4 + 2]),
                                         __uint_as_float(v[g * 4 + 3]));
            continue;
          }
          if (split_mode) {
#pragma unroll
            for (int e = 0; e < 32; ++e) {
              if (col_ok && sb + e < p.S) atomicAdd(out_col + static_cast<int64_t>(sb + e) * p.out_s1, __uint_as_float(v[e]));
            }
            continue;
          }
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            const float o = m + logf(__uint_as_float(v[e]));
            if (col_ok && sb + e < p.S) {
              out_col[static_cast<int64_t>(sb + e) * p.out_s1] = o;
              cmx = fmaxf(cmx, o);
            }
          }
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive_cluster(acc_empty_leader0 + buf * 8u);
          if (last) mbar_arrive(&msum_empty[slot]);
        }
        if (park_it && last) {
          __threadfence();  // this lane's sums are visible ...
          __syncwarp();
          int before = 0;
          if (lane == 0) before = atomicAdd(p.park_flags + (shared_tile * 2 + static_cast<int>(rank)) * 4 + q, 1);  // ... before they are counted
          if (__shfl_sync(0xffffffffu, before, 0) == shared_parts - 1) {
            __threadfence();
#pragma unroll 1
            for (int c = 0; c < rows / 32; ++c) {
              const int sb = s0 + c * 32;
              uint32_t v[32] = {};
#pragma unroll 1
              for (int part = 0; part < shared_parts; ++part) {
                const float4* src = parked + part * (PARK_TILE / 4) + c * 8 * 128;
#pragma unroll
                for (int g = 0; g < 8; ++g) add_quad(v, g, __ldcg(src + g * 128));  // written during this launch: not through the read-only path
              }
#pragma unroll
              for (int e = 0; e < 32; ++e) {
                const float o = m + logf(__uint_as_float(v[e]));
                if (col_ok && sb + e < p.S) {
                  out_col[static_cast<int64_t>(sb + e) * p.out_s1] = o;
                  cmx = fmaxf(cmx, o);
                }
              }
            }
          }
        }
      }
      if (ok && p.out_max != nullptr && !split_mode && col_ok) {
        float* dst = p.out_max + static_cast<int64_t>(r) * p.K + kcol;
        if (!park_it && p.tiles_m == 1) *dst = cmx;
        else red_max_f32(dst, cmx);  // (a part that did not complete its tile: -inf)
      }
    }
  } else if (warp >= 8 + Cfg::NTW) {
    // ------------------------------------------------------------------ splitting: the low parts of the w tile
    const int t = threadIdx.x - (8 + Cfg::NTW) * 32;
    const int nq = p.box_rows / 16;  // 16-byte pieces per thread: box_rows rows of eight over 128 threads
    const uint32_t xf_done_leader0 = map_to_cta(smem_u32(&xf_done[0]), 0);
    uint32_t it = 0;
    bool ok = true;
    LtWork work(p, KBT, pair, npairs);
    for (LtItem w; ok && work.next(w);) {
      for (int kb = w.kb_lo; kb < w.kb_hi; ++kb, ++it) {
        if (!(ok = mbar_wait_warp(&w_full[it % RING], (it / RING) & 1, ctl, STATUS_TIMEOUT_TRANSFORM))) break;
        const float4* src = reinterpret_cast<const float4*>(stage_base + (it % Cfg::NSW) * Cfg::STAGE) + t;
        float4* dst = reinterpret_cast<float4*>(stage_base + (it % Cfg::NSW) * Cfg::STAGE + Cfg::W_TILE) + t;
        float4 v[BM / 32];
#pragma unroll
        for (int c = 0; c < BM / 32; ++c)
          if (c < nq) v[c] = src[c * 128];
#pragma unroll
        for (int c = 0; c < BM / 32; ++c)
          if (c < nq)
            dst[c * 128] = make_float4(tf32_lo_trunc(v[c].x), tf32_lo_trunc(v[c].y), tf32_lo_trunc(v[c].z), tf32_lo_trunc(v[c].w));
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(xf_done_leader0 + (it % RING) * 8u);
      }
    }
  } else if (warp >= 8) {
    // ------------------------------------------------------------------ transform: operand generator
    const int tt = threadIdx.x - 8 * 32;
    const int n = tt % BN;    // this CTA's column = TMEM lane owned by this thread
    const int grp = tt / BN;  // this thread's group takes every second k-block
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + Cfg::P_COL0;
    const uint32_t xf_done_leader0 = map_to_cta(smem_u32(&xf_done[0]), 0);
    uint32_t it = 0, tcount = 0;
    bool ok = true;
    if (p.ma_wait) pdl_wait();
    LtWork work(p, KBT, pair, npairs);
    for (LtItem w; ok && work.next(w); ++tcount) {
      int r, n0, s0, rows;
      decode(w.tile, r, n0, s0, rows);
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
        part[grp * BN + n] = col_ok ? strided_column_max(a_col, p.a_s1, p.I, grp, NG) : -INFINITY;
        part[(Cfg::RG + grp) * BN + n] = col_ok ? strided_column_max(b_col, p.b_s1, p.J, grp, NG) : -INFINITY;
        nparts = NG;
      }
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
      if (grp == 0) {
        if (!(ok = mbar_wait_warp(&msum_empty[slot], ((tcount >> 1) & 1) ^ 1, ctl, STATUS_TIMEOUT_TRANSFORM))) break;
        msum[slot * BN + n] = ma + mb;
        if (NG > 1) {
          __syncwarp();
          if (lane == 0) mbar_arrive(&msum_full[slot]);
        }
      }

      for (int jc = w.kb_lo / p.I; ok && jc * p.I < w.kb_hi; ++jc) {
        const int i_lo = lt_row_lo(w, jc, p.I);
        const int In = lt_row_hi(w, jc, p.I) - i_lo;  // rows of this j-chunk in the item
        const float* a_sl = a_col + static_cast<int64_t>(i_lo) * p.a_s1;
        // exp(b - mb) of the 32 j of the chunk; padding (past J or K) enters the exp as -inf: exact zero.
        float eb[32];
#pragma unroll
        for (int x = 0; x < 32; ++x) {
          const int j = jc * BK + x;
          eb[x] = -INFINITY;
          if (col_ok && j < p.J) eb[x] = __ldg(b_col + static_cast<int64_t>(j) * p.b_s1);
        }
#pragma unroll
        for (int x = 0; x < 32; ++x) eb[x] = exp_shifted(eb[x], mb);
        float apf[PF];
        // Groups alternate over the stage counter, not over i: a group's consecutive stages are then NG apart whatever
        // the row counts of the chunks, so that a stage it waits for by parity is never two uses behind (with NS = 2
        // or 3 stages and odd row counts it could be, counted over i).
        const int g0 = (grp + NG - static_cast<int>(it % NG)) % NG;
#pragma unroll
        for (int x = 0; x < PF; ++x) {
          const int i = g0 + x * NG;
          apf[x] = (col_ok && i < In) ? __ldg(a_sl + static_cast<int64_t>(i) * p.a_s1) : -INFINITY;
        }
        for (int ib = 0; ok && ib < In; ib += PF * NG) {
          float acur[PF];
#pragma unroll
          for (int x = 0; x < PF; ++x) {
            acur[x] = apf[x];
            const int i = ib + PF * NG + g0 + x * NG;
            apf[x] = (col_ok && i < In) ? __ldg(a_sl + static_cast<int64_t>(i) * p.a_s1) : -INFINITY;
          }
#pragma unroll
          for (int x = 0; x < PF; ++x) {
            const int i = ib + g0 + x * NG;
            if (i >= In) break;
            const uint32_t my_it = it + static_cast<uint32_t>(i);
            const float ea = exp_shifted(acur[x], ma);
            if (!(ok = wait_kb(my_it, Cfg::NSP, STATUS_TIMEOUT_TRANSFORM, true))) break;
            tc_fence_after_sync();
            const uint32_t stage = lane_base + (my_it % Cfg::NSP) * Cfg::P_STAGE;
#pragma unroll
            for (int h = 0; h < 2; ++h) {  // 16 of the 32 terms at a time: both words of all 32 do not fit in registers
              float hi[16], lo[16];
#pragma unroll
              for (int e = 0; e < 16; ++e) tf32_split_rn(ea * eb[h * 16 + e], hi[e], lo[e]);
              tmem_st_32x16(stage + h * 16, hi);
              tmem_st_32x16(stage + BK + h * 16, lo);
            }
            tmem_st_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(xf_done_leader0 + (my_it % RING) * 8u);
          }
        }
        it += static_cast<uint32_t>(In);
      }
    }
  }

  // ------------------------------------------------------------------ teardown
  // Neither CTA may leave while the other can still signal into its shared memory or use its TMEM half.
  tc_fence_before_sync();
  cluster_sync_all();
  if (*abort_flag) {
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000LL) {
    }
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, Cfg::TMEM_COLS);
  }
  cluster_sync_all();  // (the pair deallocation involves both CTAs: neither leaves before the other has done it)
}

}  // namespace tb200
