// lm2exp in 3xTF32 on CTA pairs: the generated operand in tensor memory, TWO accumulators.
//
// The arithmetic and the roles of lm2exp_tspair_kernel.cuh: D^T[k, i] = sum_j E^T[k, j] * a[i, j] with E = exp(b - m)
// (replaces triturus/lm2exp.py:63-164), E^T in tensor memory, `a` as the K-major (a transposed view: MN-major) B operand,
// e_lo * a_hi + e_hi * a_lo + e_hi * a_hi, all as tf32 MMAs.  (The two corrections as bf16 MMAs of twice the rate, both
// factors of a term packed into one word, were a fifth faster.  But bf16 has 8 significant bits: a single term was off by up to
// 7.1e-6 of itself instead of 1.1e-6, and that does not average out where one term dominates a sum.)
//
// A tile is 256 columns k (M, 128 per CTA = the CTA's TMEM lanes) x up to 192 rows i (N, half of them in each CTA's shared
// memory): two accumulators of 192 columns and two operand stages of 64 (both parts of E^T) fill the 512 TMEM columns, and the
// epilogue of a tile runs under the MMAs of the next.  (256 rows with one accumulator and four stages left 15 100 of the
// 62 900 cycles of a tile of J = 1024 to the epilogue.)  A k-block of 192 rows is 1 152 cycles of MMAs, long enough for two stages:
// measured 1 150 per k-block.  Below about 160 rows the transform warps bound it, 950 cycles per k-block, whatever the rows.
//
// Work.  Rows are counted in units of 32.  The pairs form groups, one pair per 256-column slab; every group takes an equal
// contiguous share of the R * ceil(I / 32) row units, its pairs the same rows for their own columns, so that they read the
// same tiles of a at the same time.  A share is cut at the borders of batch entries and then into even tiles of at most six units
// (PairWalk), so that pairs differ by one unit and not by one tile: R40 1000x700x700 is three slabs, 72 of 74 pairs with 53 or 54
// units each; as 720 equal tiles round robin some pairs would have ten of them, 60 units.  Where the groups would leave more
// pairs idle than equal tiles do, tiles go round robin.
//
// Measured against 256-row tiles with one accumulator, us per call in a loop: R40 1000x700x700 206 -> 180, R48 260x1000x300 128 -> 82,
// R64 512x512x256 62.7 -> 55.8 (with other inputs in every pass 63.2 -> 59.3); which of the two a call takes is pair3x_wins in api.cu.
//
// Rings.  The barriers of k-blocks are rings of eight (index = k-block counter `it` % 8, phase it / 8), whatever the number
// of stages that the memory allows: TMEM stage it % 2, shared-memory stage of a it % 4.  Who wants to overwrite a stage waits
// for the commit of the MMAs of k-block it - 2 (it - 4).  That is enough for the barriers as well: those MMAs were issued after
// every arrival for their k-block, so k-block it - 8 and all before it are through every barrier.
//
//   warp 0      TMA producer: this CTA's half of the tile's rows of a (128B swizzle).
//   warp 1      TMEM allocation; in the leader CTA the warp walks the k-blocks and one elected lane issues the pair MMAs.
//   warp 2      TMA producer: this CTA's 128 columns of b (no swizzle).
//   warps 4-7   epilogue (TMEM lane quarter = warp % 4).
//   warps 8-15  transform: two groups of four warps (one per lane quarter) take alternate k-blocks.
//   warps 16-19 wait for the tiles of a, write their low parts to a second tile and say so on xf_done.
#pragma once

#include "lm2exp_tspair_kernel.cuh"
#include "row_tiles.cuh"

namespace tb200 {

struct Lm2expPair3xCfg {
  static constexpr int BM = 128;  // columns k per CTA (256 per pair): TMEM lanes
  static constexpr int BN = 192;  // rows i per pair tile at most
  static constexpr int UNITS = BN / 32;
  static constexpr int BK = 32, NG = 2, NTW = 4 * NG, NPW = 4, RING = 8;
  static constexpr int NSE = 2, NSA = 4, NSB = 6;  // stages: E^T (tensor memory), a, b
  static constexpr int B_TILE = BK * BM * 4;       // 16 KB
  static constexpr int A_TILE = BN / 2 * BK * 4;   // 12 KB
  static constexpr int A_STAGE = 2 * A_TILE;       // the tile and its low parts
  static constexpr int E_COLS = 2 * BK;            // TMEM columns of an operand stage
  static constexpr int E_COL0 = 2 * BN;
  static constexpr int TMEM_COLS = 512;
  static constexpr int NTHREADS = (8 + NTW + NPW) * 32;
  static constexpr int EPI_STAGE = 4 * 2 * 32 * 128;  // per epilogue warp two 32 x 32 fp32 boxes
  static constexpr int NBAR = 3 * RING + 2 * NSB + 4;
  static constexpr int SMEM_BYTES = 1024 + NSA * A_STAGE + NSB * B_TILE + EPI_STAGE + NBAR * 8 + 64;
  static_assert(E_COL0 + NSE * E_COLS <= TMEM_COLS, "TMEM capacity");
  static_assert(NSE <= RING && NSA <= RING && NSE == NG && NSB % NG == 0, "rings (a stage and a slot of b belong to one transform group)");
  static_assert(SMEM_BYTES <= 232448, "shared memory capacity");
};

// The tiles of one pair, in the order every role walks them.  p.tiles_m: row units of 32 per batch entry; p.tiles_n: 256-column
// slabs; p.pair_groups > 0: that many groups of tiles_n pairs (see above); 0: p.num_tiles tiles round robin, row tiles fastest.
struct PairWalk {
  int64_t u, hi;  // groups: next unit and end of the share; round robin: next tile (hi unused)
  __device__ PairWalk(const Lm2expParams& p, int pair) {
    if (p.pair_groups > 0) {
      const int64_t total = static_cast<int64_t>(p.R) * p.tiles_m;
      const int g = pair / p.tiles_n;
      u = total * g / p.pair_groups;
      hi = total * (g + 1) / p.pair_groups;
    } else {
      u = pair;
      hi = 0;
    }
  }
  __device__ bool next(const Lm2expParams& p, int pair, int npairs, int& r, int& n0, int& i0, int& rows) {
    constexpr int UNITS = Lm2expPair3xCfg::UNITS;
    int lo, take;
    if (p.pair_groups > 0) {
      if (u >= hi) return false;
      r = static_cast<int>(u / p.tiles_m);
      lo = static_cast<int>(u - static_cast<int64_t>(r) * p.tiles_m);
      const int left = static_cast<int>(min(hi - u, static_cast<int64_t>(p.tiles_m - lo)));  // of the share in this entry
      const int nt = (left + UNITS - 1) / UNITS;
      take = (left + nt - 1) / nt;
      n0 = (pair % p.tiles_n) * (2 * Lm2expPair3xCfg::BM);
      u += take;
    } else {
      if (u >= p.num_tiles) return false;
      const int nt = (p.tiles_m + UNITS - 1) / UNITS;
      const int tile = static_cast<int>(u);
      const int tm = tile % nt, rest = tile / nt;
      r = rest / p.tiles_n;
      n0 = (rest % p.tiles_n) * (2 * Lm2expPair3xCfg::BM);
      const RowTile t = row_tile(p.tiles_m, nt, tm);
      lo = t.first;
      take = t.units;
      u += npairs;
    }
    i0 = lo * 32;
    rows = take * 32;
    return true;
  }
};

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(Lm2expPair3xCfg::NTHREADS, 1)
lm2exp_pair3x_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                     const __grid_constant__ CUtensorMap tmap_out, const Lm2expParams p) {
  using Cfg = Lm2expPair3xCfg;
  constexpr int BM = Cfg::BM, BN = Cfg::BN, BK = Cfg::BK, NSB = Cfg::NSB, NSA = Cfg::NSA, NSE = Cfg::NSE;
  constexpr uint32_t RMASK = Cfg::RING - 1;

  // A conditional launch: runs only if the launch before it raised the flag.
  if (p.only_if != nullptr) {
    pdl_wait();
    if (*p.only_if == 0) return;
    // (a flag republished in a second word by a conditional pre-pass: all readers of the first one are done)
    if (blockIdx.x == 0 && threadIdx.x == 0 && p.reset_flag != nullptr) *p.reset_flag = 0;
  }

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* a_base = smem;
  uint8_t* b_base = smem + NSA * Cfg::A_STAGE;
  uint8_t* epi_stage = b_base + NSB * Cfg::B_TILE;
  uint64_t* bars = reinterpret_cast<uint64_t*>(epi_stage + Cfg::EPI_STAGE);
  uint64_t* a_full = bars;                  // [8] this CTA's tile of a landed
  uint64_t* xf_done = bars + Cfg::RING;     // [8] (leader's copy is used) E^T stage and low parts of a written, both CTAs
  uint64_t* kb_done = xf_done + Cfg::RING;  // [8] MMAs of the k-block retired (committed by the leader)
  uint64_t* b_full = kb_done + Cfg::RING;   // [NSB]
  uint64_t* b_empty = b_full + NSB;         // [NSB] the four transform warps of the k-block hold it in registers
  uint64_t* acc_full = b_empty + NSB;       // [2] accumulator complete (committed by the leader)
  uint64_t* acc_empty = acc_full + 2;       // [2] (leader's copy is used) epilogues of both CTAs drained it
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + Cfg::NBAR);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = warp_uniform(threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const uint32_t rank = warp_uniform(cluster_ctarank());
  const bool leader = rank == 0;
  const AbortCtl ctl{abort_flag, p.status};

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < Cfg::RING; ++s) {
      mbar_init(&a_full[s], 1);
      mbar_init(&xf_done[s], 2 * (4 + Cfg::NPW));  // four transform and four splitting warps in each CTA
      mbar_init(&kb_done[s], 1);
    }
    for (int s = 0; s < NSB; ++s) {
      mbar_init(&b_full[s], 1);
      mbar_init(&b_empty[s], 4);
    }
    for (int h = 0; h < 2; ++h) {
      mbar_init(&acc_full[h], 1);
      mbar_init(&acc_empty[h], 8);
    }
    fence_mbar_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    if (p.out_tma) tma_prefetch_desc(&tmap_out);
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

  const int KB = (p.J + BK - 1) / BK;
  const int npairs = gridDim.x >> 1;
  const int pair = blockIdx.x >> 1;
  int r, n0, i0, rows;  // the tile: batch entry, first column, first row, rows (a multiple of 32)

  // The commit of k-block `it - back` (the caller's own k-blocks before it are long committed).
  auto wait_kb = [&](uint32_t it, uint32_t back, int code, bool warp_wide) -> bool {
    if (it < back) return true;
    const uint32_t x = it - back;
    return warp_wide ? mbar_wait_warp(&kb_done[x & RMASK], (x / Cfg::RING) & 1, ctl, code)
                     : mbar_wait(&kb_done[x & RMASK], (x / Cfg::RING) & 1, ctl, code);
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer: this CTA's rows of a
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      for (PairWalk walk(p, pair); ok && walk.next(p, pair, npairs, r, n0, i0, rows);) {
        // (the box has BN / 2 rows whatever the rows of the tile: rows behind them are loaded and not used)
        const int my_i0 = i0 + static_cast<int>(rank) * (rows / 2);
        for (int kb = 0; kb < KB; ++kb, ++it) {
          if (!(ok = wait_kb(it, NSA, STATUS_TIMEOUT_PRODUCER, false))) break;
          TB200_TL(9, it);
          uint8_t* dst = a_base + (it % NSA) * Cfg::A_STAGE;
          uint64_t* bar = &a_full[it & RMASK];
          mbar_arrive_expect_tx(bar, Cfg::A_TILE);
          if (p.a_mn) {
#pragma unroll
            for (int g = 0; g < BN / 64; ++g) tma_load_3d(dst + g * 4096, &tmap_a, bar, my_i0 + g * 32, kb * BK, r);
          } else {
            tma_load_3d(dst, &tmap_a, bar, kb * BK, my_i0, r);
          }
        }
      }
      // The leader's commits arrive on both CTAs' barriers: this CTA stays until the last ones are in.
      for (uint32_t d = ok ? min(it, static_cast<uint32_t>(Cfg::RING)) : 0u; ok && d > 0; --d)
        ok = wait_kb(it, d, STATUS_TIMEOUT_PRODUCER, false);
    }
    __syncwarp();
  } else if (warp == 2) {
    // ------------------------------------------------------------------ TMA producer: this CTA's columns of b
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      for (PairWalk walk(p, pair); ok && walk.next(p, pair, npairs, r, n0, i0, rows);) {
        const int my_n0 = n0 + static_cast<int>(rank) * BM;
        for (int kb = 0; kb < KB; ++kb, ++it) {
          const int s = it % NSB;
          if (!(ok = mbar_wait(&b_empty[s], ((it / NSB) & 1) ^ 1, ctl, STATUS_TIMEOUT_PRODUCER))) break;
          TB200_TL(10, it);
          mbar_arrive_expect_tx(&b_full[s], Cfg::B_TILE);
          tma_load_3d(b_base + s * Cfg::B_TILE, &tmap_b, &b_full[s], my_n0, kb * BK, r);
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ pair MMA issuer (leader CTA only)
    if (leader) {
      const bool a_mn = p.a_mn != 0;
      const uint32_t a_step = a_mn ? 64u : 2u;  // encoded address step per 8 contraction values
      constexpr uint32_t STAGE_ENC = Cfg::A_STAGE >> 4, LO_ENC = Cfg::A_TILE >> 4;
      const uint64_t db0 = a_mn ? umma_desc_mn_sw128_base32(smem_u32(a_base), 4096) : umma_desc_k_sw128(smem_u32(a_base));
      uint32_t it = 0, tcount = 0;
      bool ok = true;
      for (PairWalk walk(p, pair); ok && walk.next(p, pair, npairs, r, n0, i0, rows); ++tcount) {
        const uint32_t buf = tcount & 1;
        // M = 256 columns k over the pair (A from TMEM), N = rows i of the tile, half of them in each CTA's shared memory
        const uint32_t idesc = umma_idesc_tf32(2 * BM, rows) | (a_mn ? 1u << 16 : 0u);
        const uint32_t d = tmem_base + buf * BN;
        TB200_TL(11, tcount);
        if (!(ok = mbar_wait_warp(&acc_empty[buf], ((tcount >> 1) & 1) ^ 1, ctl, STATUS_TIMEOUT_MMA))) break;
        TB200_TL(12, tcount);
        tc_fence_after_sync();
        for (int kb = 0; kb < KB; ++kb, ++it) {
          if (!(ok = mbar_wait_warp(&xf_done[it & RMASK], (it / Cfg::RING) & 1, ctl, STATUS_TIMEOUT_MMA))) break;
          TB200_TL(0, it);
          tc_fence_after_sync();
          if (elect_one_sync()) {
            const uint64_t db = db0 + (it % NSA) * STAGE_ENC;
            const uint32_t ea = tmem_base + Cfg::E_COL0 + (it % NSE) * Cfg::E_COLS;
            // The corrections first, while the accumulator of a tile is empty: the sum of the first k-block's is not
            // truncated to the bits of the whole sum then.
#pragma unroll
            for (int ks = 0; ks < BK / 8; ++ks)
              umma_tf32_ts_pair(d, ea + BK + ks * 8, db + a_step * ks, idesc, (kb > 0 || ks > 0) ? 1u : 0u);
#pragma unroll
            for (int ks = 0; ks < BK / 8; ++ks) umma_tf32_ts_pair(d, ea + ks * 8, db + LO_ENC + a_step * ks, idesc, 1u);
#pragma unroll
            for (int ks = 0; ks < BK / 8; ++ks) umma_tf32_ts_pair(d, ea + ks * 8, db + a_step * ks, idesc, 1u);
            umma_commit_pair_mcast(smem_u32(&kb_done[it & RMASK]), 3);
          }
          __syncwarp();
          TB200_TL(1, it);
        }
        if (ok && elect_one_sync()) umma_commit_pair_mcast(smem_u32(&acc_full[buf]), 3);
        __syncwarp();
      }
    }
    __syncwarp();
  } else if (warp >= 4 && warp < 8) {
    // ------------------------------------------------------------------ epilogue (this CTA's 128 columns k x the tile's rows i)
    const int q = warp & 3;
    uint8_t* stg2 = epi_stage + q * 8192;  // two boxes: one is filled while the TMA unit still reads the other
    uint32_t nbox = 0;
    const bool use_tma = p.out_tma != 0;
    const uint32_t acc_empty_leader0 = map_to_cta(smem_u32(acc_empty), 0);
    pdl_wait();  // m comes from the pre-pass, which may still be running when this kernel starts
    uint32_t tcount = 0;
    bool ok = true;
    uint32_t acc_max = 0;  // largest accumulator bit pattern of this lane (sums of non-negative products, so +inf and NaN
                           // are exactly the patterns >= 0x7f800000 read as unsigned)
    for (PairWalk walk(p, pair); ok && walk.next(p, pair, npairs, r, n0, i0, rows); ++tcount) {
      const uint32_t buf = tcount & 1;
      const uint32_t tbase = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + buf * BN;
      const int k0 = n0 + static_cast<int>(rank) * BM + q * 32;  // first column of this warp's 32
      const int kcol = k0 + lane;
      const bool col_ok = kcol < p.K;
      float m = 0.f;
      if (col_ok) m = clamp_stab(__ldg(p.m_ws + static_cast<int64_t>(r) * p.K + kcol));
      float* ocol = p.out + static_cast<int64_t>(r) * p.out_s0 + kcol;
      float cmx = -INFINITY;  // largest result of this lane's column in the tile, for the next layer of a chain
      if (!(ok = mbar_wait_warp(&acc_full[buf], (tcount >> 1) & 1, ctl, STATUS_TIMEOUT_EPILOGUE))) break;
      if (warp == 4 && lane == 0) TB200_TL(7, tcount);
      tc_fence_after_sync();
      const uint32_t acc_empty_leader = acc_empty_leader0 + buf * 8u;
      const int nchunks = k0 >= p.K ? 0 : rows / 32;
      if (nchunks == 0) {
        // nothing to store (this warp's columns are padding): release the accumulator right away
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(acc_empty_leader);
        continue;
      }
#pragma unroll 1
      for (int c = 0; c < nchunks; ++c) {
        uint32_t v[32];  // (one buffer: the logarithms want the registers of a second)
        tmem_ld_32x32(tbase + c * 32, v);
        tmem_ld_wait();
        if (c + 1 == nchunks) {
          // all of it is in registers: hand it back to the MMA issuer
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(acc_empty_leader);
        }
        const int ib = i0 + c * 32;
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          acc_max = max(acc_max, v[e]);
          // (lg2.approx of the mantissa is off by 2^-22 whatever the result, several ulp for sums near 1)
          const float o = m + logf(__uint_as_float(v[e]));
          cmx = fmaxf(cmx, o);  // (rows past I hold log 0 = -inf)
          v[e] = __float_as_uint(o);
        }
        // Register e of this lane is row ib + e, column kcol of the result.  The 32 x 32 block goes through a staging box
        // (row e at byte e * 128 in the 128-byte swizzle, the 32 lanes of a store fill one row) and from there as one TMA
        // store.
        if (use_tma) {
          uint8_t* stg = stg2 + (nbox & 1) * 4096;
          ++nbox;
          if (lane == 0) tma_store_wait_read<1>();  // the store before the previous one has read this box out
          __syncwarp();
#pragma unroll
          for (int e = 0; e < 32; ++e) *reinterpret_cast<uint32_t*>(stg + sw128_offset(e, lane)) = v[e];
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_3d(&tmap_out, stg, k0, ib, r);  // clipped at the edges of the tensor
            tma_store_commit();
          }
        } else {
          // A result that a TMA store cannot write (K not a multiple of 4, unaligned base): row by row.
          float* orow = ocol + static_cast<int64_t>(ib) * p.out_s1;
          const int nrows = min(32, p.I - ib);
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            if (col_ok && e < nrows) orow[static_cast<int64_t>(e) * p.out_s1] = __uint_as_float(v[e]);
          }
        }
      }
      if (warp == 4 && lane == 0) TB200_TL(8, tcount);
      if (p.out_max != nullptr && col_ok) red_max_f32(p.out_max + static_cast<int64_t>(r) * p.K + kcol, cmx);
    }
    if (use_tma && lane == 0) tma_store_wait_all();  // shared memory must outlive the last box
    if (p.opt_flag != nullptr) {  // stabiliser from the first 32 rows only: say whether a result overflowed
      if (__any_sync(0xffffffffu, acc_max >= 0x7f800000u) && lane == 0) *p.opt_flag = 1;
    }
  } else if (warp >= 8 + Cfg::NTW) {
    // ------------------------------------------------------------------ splitting: the low parts of the tile of a
    // The tile itself stays as it is (the tensor core drops the low 13 bits).
    const int t = threadIdx.x - (8 + Cfg::NTW) * 32;
    const uint32_t xf_done_leader0 = map_to_cta(smem_u32(&xf_done[0]), 0);
    uint32_t it = 0;
    bool ok = true;
    for (PairWalk walk(p, pair); ok && walk.next(p, pair, npairs, r, n0, i0, rows);) {
      for (int kb = 0; kb < KB; ++kb, ++it) {
        if (!(ok = mbar_wait_warp(&a_full[it & RMASK], (it / Cfg::RING) & 1, ctl, STATUS_TIMEOUT_TRANSFORM))) break;
        const float4* src = reinterpret_cast<const float4*>(a_base + (it % NSA) * Cfg::A_STAGE) + t;
        float4* dst = reinterpret_cast<float4*>(a_base + (it % NSA) * Cfg::A_STAGE + Cfg::A_TILE) + t;
        float4 v[BN / 32];
#pragma unroll
        for (int c = 0; c < BN / 32; ++c) v[c] = src[c * 128];
#pragma unroll
        for (int c = 0; c < BN / 32; ++c)
          dst[c * 128] = make_float4(tf32_lo_trunc(v[c].x), tf32_lo_trunc(v[c].y), tf32_lo_trunc(v[c].z), tf32_lo_trunc(v[c].w));
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(xf_done_leader0 + (it & RMASK) * 8u);
      }
    }
  } else if (warp >= 8) {
    // ------------------------------------------------------------------ transform: b tile -> E^T in tensor memory
    const int q = warp & 3;  // TMEM lane quarter this warp may write
    const int grp = (warp - 8) >> 2;
    const int kl = q * 32 + lane;
    const uint32_t ebase = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + Cfg::E_COL0;
    const uint32_t xf_done_leader0 = map_to_cta(smem_u32(&xf_done[0]), 0);
    pdl_wait();  // m comes from the pre-pass (the producer warp is already loading operand tiles meanwhile)
    // Groups alternate over the k-block counter of the launch and not of the tile (see lm2exp_tspair_kernel.cuh).
    uint32_t it0 = 0;  // k-blocks before this tile
    bool ok = true;
    for (PairWalk walk(p, pair); ok && walk.next(p, pair, npairs, r, n0, i0, rows); it0 += static_cast<uint32_t>(KB)) {
      const int kcol = n0 + static_cast<int>(rank) * BM + kl;
      // A column past K reads zero-filled values; the stabiliser +inf turns them into exact zeros.
      const float m = kcol < p.K ? clamp_stab(__ldg(p.m_ws + static_cast<int64_t>(r) * p.K + kcol)) : INFINITY;
      for (int kb = static_cast<int>((grp + it0) & 1); kb < KB; kb += Cfg::NG) {
        const uint32_t it = it0 + static_cast<uint32_t>(kb);
        const uint32_t sb = it % NSB;
        if (!(ok = mbar_wait_warp(&b_full[sb], (it / NSB) & 1, ctl, STATUS_TIMEOUT_TRANSFORM))) break;
        if (warp == 8 && lane == 0) TB200_TL(2, it);
        const float* col = reinterpret_cast<const float*>(b_base + sb * Cfg::B_TILE) + kl;
        float e[32];
#pragma unroll
        for (int x = 0; x < 32; ++x) e[x] = col[x * BM];
        const int jrem = p.J - kb * BK;
        if (jrem < BK) {
          // rows past J are zero-filled by TMA (in log space): they enter the exp as -inf, exact zero out
#pragma unroll
          for (int x = 0; x < 32; ++x) e[x] = x < jrem ? e[x] : -INFINITY;
        }
        // (the exps stay in fp32 until the stage is free and are split there, 16 at a time: both words of all 32 do not
        // fit in the 96 registers of a thread)
#pragma unroll
        for (int x = 0; x < 32; x += 2) exp_shifted_x2(e[x], e[x + 1], m, e[x], e[x + 1]);
        // Every lane has consumed its values of the b tile: hand the tile back to its producer.
        __syncwarp();
        if (lane == 0) mbar_arrive(&b_empty[sb]);
        // The E^T stage is free once the MMAs that read it last time have retired.
        if (!(ok = wait_kb(it, NSE, STATUS_TIMEOUT_TRANSFORM, true))) break;
        if (warp == 8 && lane == 0) TB200_TL(4, it);
        tc_fence_after_sync();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float hi[16], lo[16];
#pragma unroll
          for (int x = 0; x < 16; ++x) tf32_split_rn(e[h * 16 + x], hi[x], lo[x]);
          tmem_st_32x16(ebase + (it % NSE) * Cfg::E_COLS + h * 16, hi);
          tmem_st_32x16(ebase + (it % NSE) * Cfg::E_COLS + BK + h * 16, lo);
        }
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(xf_done_leader0 + (it & RMASK) * 8u);
        if (warp == 8 && lane == 0) TB200_TL(6, it);
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
