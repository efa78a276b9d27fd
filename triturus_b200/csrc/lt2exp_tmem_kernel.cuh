// lt2exp with the generated operand in TENSOR MEMORY (some plain TF32 tiles, and all of 3xTF32 as the PREC instance).
//
// Same contraction as lt2exp_kernel.cuh (which replaces triturus/lt2exp.py:227-357 and :365-506), computed
// transposed:
//
//     D^T[k, s] = sum_{(i,j)} P^T[k, (i,j)] * W^T[(i,j), s],   P^T[k, (i,j)] = exp(a[i,k]-ma[k]) * exp(b[j,k]-mb[k])
//
// so that the Khatri-Rao operand P^T is the tensor core's A operand, which tcgen05.mma can read from TMEM.  A
// transform thread owns one column k of the tile = one TMEM lane; per k-block (one i, 32 consecutive j) it
// forms its 32 products in registers and writes them to its lane with a single tcgen05.st.  The generated
// operand therefore never touches shared memory.  Per k-block the shared-memory pipe, which bounds
// lt2exp_kernel (w in, operand stores, operand reads), carries only the w tile: TMA in + one read by the
// tensor core (B operand, N = s, K-major as it lies in memory), which balances the tensor pipe exactly
// (128 x 256 x 32 MACs = 512 cycles; 64 KB at 128 B/clk = 512 cycles).
//
// Tile: 128 columns k (MMA M) x 128*MT rows s (MMA N, one instruction even for N = 256: the MT w boxes of a
// stage are contiguous and form one K-major tile).  The accumulator holds D^T: TMEM lane = k, column = s, so in
// the epilogue the 32 lanes of a warp hold 32 consecutive k of one output row, m = ma + mb is a per-lane
// constant and every store instruction writes one full 128-byte row segment.
//
// TMEM: NBUF accumulators of 128*MT columns (two when MT = 1) followed by NS operand stages of 32 columns.
// Stage s of shared memory (w) and operand stage s of TMEM are released together by one tcgen05.commit.
//
//   warp 0      TMA producer: w boxes {32 j, 1 i, 128 s, 1 r}, 128-byte swizzle.
//   warp 1      TMEM allocation; the warp walks the k-blocks and one elected lane issues tcgen05.mma.kind::tf32 with A in TMEM
//               (M = 128, N = 128*MT, K = 8).
//   warps 4-7   epilogue: tcgen05.ld, out[s, k] = m[k] + log(acc), coalesced 128-byte stores (or fp32 reductions
//               into the zero-filled result when the contraction is split, see lt2exp_kernel.cuh); 3xTF32: re-summation of
//               finished chunks meanwhile.
//   warps 8-15  transform: warp w writes TMEM lane quarter w % 4; the two warps of a quarter take alternate
//               k-blocks.  Column maxima first (cooperative, as in lt2exp_kernel.cuh).
//   warps 16-19 3xTF32: the low parts of the w tiles.
#pragma once

#include "lt2exp_kernel.cuh"

namespace tb200 {

// PREC (3xTF32): p_lo * w_hi + p_hi * w_lo + p_hi * w_hi, all as tf32 MMAs.  The w tile serves them as it lies in shared
// memory (the tensor core truncates); four splitting warps (16-19) write its low parts to a second tile, the transform
// warps both parts of P^T to 64 TMEM columns.  (The corrections as bf16 MMAs of twice the rate: R32 256^4 1 154 instead of
// 1 298 us, but terms off by up to 7e-6, see lm2exp_tspair_kernel.cuh.)
// Per k-block of a 128 x 128 tile: 16 KB TMA in, 16 KB read and 16 KB written by the splitting, 48 KB read by the tensor
// core = 768 cycles of the shared-memory pipe next to 768 of the tensor pipe (both operands in shared memory: 1 400).
// Measured 1 000 cycles per k-block (R32 256^4, 1 030 before the issuer asked for the next stage in the middle of one): what it does
// between two stages bounds it, and what the queue of the tensor core does not cover.  Calls that fill pairs of CTAs run
// lt2exp_pair3x_kernel.cuh instead.
// At 96 registers a thread (20 warps) 92 bytes are spilled, outside the loops over k-blocks: 68 loads and 52 stores per
// CTA of one tile.
// Every CHUNK k-blocks the MMA warp changes to the other accumulator and the epilogue warps add the finished one to a
// master copy in shared memory (see "Accumulator promotion" in lt2exp_kernel.cuh; TMEM has no room for a third).
// Chunks of 24 (768 terms): rms error of a long flat sum 1.2e-5.  16: 0.8e-5, but 1 to 9 % slower, the drain being no longer
// hidden (R16 128x64x64x2048 150 -> 162 us, 1 x 256^4 71 -> 79); 32: 1.6e-5, at most 2 % faster (R64 256x128x128x4096 8 560 ->
// 8 370 us, R32 256^4 1 163 -> 1 156).
template <int MT_, int NS_, int PREC_ = 0>
struct Lt2expTmemCfg {
  static constexpr int BM = 128, BK = 32;  // BM: rows s per w box
  static constexpr int BN = 128;           // columns k per tile
  static constexpr int MT = MT_, NS = NS_, PREC = PREC_, NTW = 8;
  static constexpr bool PROMOTE = PREC != 0;  // chunked re-summation of the accumulator
  static constexpr int CHUNK = PROMOTE ? 24 : 1 << 30;  // k-blocks
  static constexpr int W_TILE = BM * BK * 4;
  static constexpr int W_BYTES = MT * W_TILE;             // what TMA brings per stage
  static constexpr int STAGE = (PREC ? 2 : 1) * W_BYTES;  // ... and the low parts of it
  static constexpr int ACC_COLS = MT * BM;
  static constexpr int P_STAGE = (PREC ? 2 : 1) * BK;  // operand columns per stage
  static constexpr int NBUF = (2 * ACC_COLS + NS * P_STAGE <= 512) ? 2 : 1;
  static constexpr int P_COL0 = NBUF * ACC_COLS;  // first operand column
  static constexpr int TMEM_USED = P_COL0 + NS * P_STAGE;
  static constexpr int TMEM_COLS = 512;
  static constexpr int NPW = PREC ? 4 : 0;  // splitting warps
  static constexpr int NTHREADS = (8 + NTW + NPW) * 32;
  static constexpr int NTT = NTW * 32;
  static constexpr int NGROUPS = NTT / BN;
  static constexpr int CQ = BN / 4;
  static constexpr int RG = NTT / CQ;
  static constexpr int MPART = 2 * RG * BN;
  static constexpr int NBAR = 3 * NS + 9;
  static constexpr int MASTER = PROMOTE ? MT * BM * BN * 4 : 0;
  static_assert(!PREC || (MT == 1 && NBUF == 2), "3xTF32: 128 x 128 tiles, two accumulators");
  static constexpr int SMEM_BYTES = 1024 + NS * STAGE + MASTER + 2 * BN * 4 + 2 * MPART * 4 + NBAR * 8 + 64;
  static_assert(TMEM_USED <= 512, "TMEM capacity");
  static_assert(NGROUPS == 2, "eight transform warps: two groups");
  static_assert(SMEM_BYTES <= 232448, "shared memory capacity");
};

__device__ __forceinline__ void add_quad(uint32_t (&v)[32], int g, float4 x) {
  v[g * 4 + 0] = __float_as_uint(__uint_as_float(v[g * 4 + 0]) + x.x);
  v[g * 4 + 1] = __float_as_uint(__uint_as_float(v[g * 4 + 1]) + x.y);
  v[g * 4 + 2] = __float_as_uint(__uint_as_float(v[g * 4 + 2]) + x.z);
  v[g * 4 + 3] = __float_as_uint(__uint_as_float(v[g * 4 + 3]) + x.w);
}

template <class Cfg>
__global__ void __launch_bounds__(Cfg::NTHREADS, 1)
lt2exp_tmem_kernel(const __grid_constant__ CUtensorMap tmap_w, const Lt2expParams p) {
  constexpr int BM = Cfg::BM, BN = Cfg::BN, BK = Cfg::BK, MT = Cfg::MT, NS = Cfg::NS;
  constexpr int PF = Cfg::PREC ? 4 : 8;  // prefetch distance (own k-blocks) for the a values

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* stage_base = smem;
  // PROMOTE: [BM / 4 row quads][128 columns][4] master copy of the accumulator, each thread its own column
  float4* master = reinterpret_cast<float4*>(smem + NS * Cfg::STAGE);
  float* msum = reinterpret_cast<float*>(smem + NS * Cfg::STAGE + Cfg::MASTER);  // [2][BN]: ma + mb of the tile's columns
  float* mpart = msum + 2 * BN;                                    // [2][2][RG][BN] partial column maxima
  uint64_t* bars = reinterpret_cast<uint64_t*>(mpart + 2 * Cfg::MPART);
  uint64_t* full = bars;                 // [NS] w tile landed (TMA bytes) and operand stage written to TMEM
  uint64_t* w_full = bars + NS;          // PREC [NS] w tile landed (the splitting warps wait for it)
  uint64_t* opnd_empty = bars + 2 * NS;  // [NS] MMAs reading the stage (shared memory and TMEM) retired
  uint64_t* acc_full = bars + 3 * NS;    // [2]
  uint64_t* acc_empty = acc_full + 2;    // [2]
  uint64_t* msum_full = acc_empty + 2;   // [2] (NGROUPS > 1, see lt2exp_kernel.cuh)
  uint64_t* msum_empty = msum_full + 2;  // [2]
  uint64_t* mx_bar = msum_empty + 2;     // [1]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mx_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = warp_uniform(threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const AbortCtl ctl{abort_flag, p.status};

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < NS; ++s) {
      if (Cfg::PREC) mbar_init(&w_full[s], 1);
      // the producer (PREC: the splitting warps instead) and the warps that write the operand stage
      mbar_init(&full[s], (Cfg::PREC ? Cfg::NPW : 1) + Cfg::NTW / Cfg::NGROUPS);
      mbar_init(&opnd_empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&acc_full[s], 1);
      mbar_init(&acc_empty[s], 4);
      mbar_init(&msum_full[s], BN / 32);
      mbar_init(&msum_empty[s], 4);
    }
    mbar_init(mx_bar, Cfg::NTW);
    fence_mbar_init();
    tma_prefetch_desc(&tmap_w);
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
  const bool parking = Cfg::PROMOTE && p.stream != 0 && p.park != nullptr;  // shared tiles are completed through scratch memory
  const bool split_mode = (p.nsplit > 1 || p.stream != 0) && !parking;
  if (split_mode) pdl_launch_dependents();  // the log pass takes its column maxima meanwhile

  // Output tile -> (r, n0 = first column k, s0 = first row s); the items of a CTA come from LtWork.
  auto decode = [&](int tile, int& r, int& n0, int& s0) {
    const int tm = tile % p.tiles_m;
    const int rest = tile / p.tiles_m;
    const int tn = rest % p.tiles_n;
    r = rest / p.tiles_n;
    n0 = tn * BN;
    s0 = tm * (BM * MT);
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
          for (int i = lt_row_lo(w, jc, p.I); i < i_hi; ++i, ++it) {
            const int s = it % NS;
            const uint32_t ph = (it / NS) & 1;
            if (!(ok = mbar_wait(&opnd_empty[s], ph ^ 1, ctl, STATUS_TIMEOUT_PRODUCER))) break;
            uint64_t* landed = Cfg::PREC ? &w_full[s] : &full[s];
            mbar_arrive_expect_tx(landed, Cfg::W_BYTES);
#pragma unroll
            for (int t = 0; t < MT; ++t)
              tma_load_4d(stage_base + s * Cfg::STAGE + t * Cfg::W_TILE, &tmap_w, landed, jc * BK, i, s0 + t * BM, r);
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    // The whole warp runs the loop with uniform control flow and one elected lane issues, so stage indices,
    // descriptors and TMEM addresses stay in uniform registers.  One barrier per stage, and the barrier of
    // the next stage is polled before this stage's MMAs are issued so that the answer arrives meanwhile: a
    // single thread issuing four MMAs per k-block after two fresh barrier round trips took ~790 cycles per
    // k-block against 512 cycles of tensor work.
    {
      constexpr uint32_t idesc = umma_idesc_tf32(128, BM * MT);  // M = 128 columns k, N = rows s
      const uint32_t stage0 = smem_u32(stage_base);
      uint32_t ccount = 0;  // accumulation chunks issued so far (one per work item unless PROMOTE)
      int s = 0;
      uint32_t ph = 0;
      bool ok = true, ready = false;
      LtWork work(p, KBT);
      for (LtItem w; ok && work.next(w);) {
       const int KB = w.kb_hi - w.kb_lo;
       for (int kb = 0; ok && kb < KB; ++ccount) {
        const int kb0 = kb, kb_end = Cfg::PROMOTE ? min(KB, kb0 + Cfg::CHUNK) : KB;
        const int buf = ccount % Cfg::NBUF;
        const uint32_t aph = (ccount / Cfg::NBUF) & 1;
        if (!(ok = mbar_wait_warp(&acc_empty[buf], aph ^ 1, ctl, STATUS_TIMEOUT_MMA))) break;
        tc_fence_after_sync();
        const uint32_t d = tmem_base + buf * Cfg::ACC_COLS;
        for (; kb < kb_end; ++kb) {
          if (!ready) {
            if (!(ok = mbar_wait_warp(&full[s], ph, ctl, STATUS_TIMEOUT_MMA))) break;
          }
          const int sn = (s + 1 == NS) ? 0 : s + 1;
          const uint32_t phn = (s + 1 == NS) ? ph ^ 1 : ph;
          tc_fence_after_sync();
          const uint64_t dw = umma_desc_k_sw128(stage0 + s * Cfg::STAGE);
          const uint32_t pa = tmem_base + Cfg::P_COL0 + s * Cfg::P_STAGE;
          if (Cfg::PREC) {
            if (elect_one_sync()) {
              // the corrections first, while the accumulator of a chunk is empty and does not truncate them to its bits
#pragma unroll
              for (int ks = 0; ks < BK / 8; ++ks)
                umma_tf32_ts(d, pa + BK + ks * 8, dw + 2 * ks, idesc, (kb > kb0 || ks > 0) ? 1u : 0u);
#pragma unroll
              for (int ks = 0; ks < BK / 8; ++ks) umma_tf32_ts(d, pa + ks * 8, dw + (Cfg::W_BYTES >> 4) + 2 * ks, idesc, 1u);
            }
          }
          // The tensor core takes the next MMA only when it is about done with the one before, so what this warp does between
          // two stages is lost to it: 3xTF32 asks for the next stage in the middle of this one.
          const bool peek = mbar_try_wait(&full[sn], phn);
          if (elect_one_sync()) {
#pragma unroll
            for (int ks = 0; ks < BK / 8; ++ks)
              umma_tf32_ts(d, pa + ks * 8, dw + 2 * ks, idesc, (Cfg::PREC || kb > kb0 || ks > 0) ? 1u : 0u);
            umma_commit(&opnd_empty[s]);
          }
          ready = __all_sync(0xffffffffu, peek);
          s = sn;
          ph = phn;
        }
        if (ok && elect_one_sync()) umma_commit(&acc_full[buf]);
        __syncwarp();
       }
      }
    }
  } else if (warp >= 4 && warp < 8) {
    // ------------------------------------------------------------------ epilogue
    const int q = warp & 3;
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
    if (split_mode) pdl_wait();  // the zero-filled result
    uint32_t tcount = 0;
    bool ok = true;
    LtWork work(p, KBT);
    if constexpr (Cfg::PROMOTE) {
      uint32_t ccount = 0;
      const int kl = q * 32 + lane;  // this lane's column of the tile
      for (LtItem w; ok && work.next(w); ++tcount) {
        int r, n0, s0;
        decode(w.tile, r, n0, s0);
        const int kcol = n0 + kl;
        const bool col_ok = kcol < p.K;
        float* out_col = p.out + static_cast<int64_t>(r) * p.out_s0 + kcol;
        const int slot = tcount & 1;
        const int nch = (w.kb_hi - w.kb_lo + Cfg::CHUNK - 1) / Cfg::CHUNK;
        // A tile of the shared last wave: every part parks its sums, and the warp that parks the last part of its columns
        // adds them up, in the order of the parts whoever it is.  No CTA waits for another, which need not have started
        // where a second kernel shares the GPU.
        const int shared_parts = p.lw_parts > 0 ? p.lw_parts : p.lw_main < KBT ? 2 : 1;
        const bool park_it = parking && w.tile >= p.lw_first && shared_parts > 1;
        const int shared_tile = w.tile - p.lw_first;
        constexpr int PARK_TILE = BM * BN;  // floats per parked tile, in the order of `master`
        float4* const parked = reinterpret_cast<float4*>(p.park + static_cast<int64_t>(shared_tile) * shared_parts * PARK_TILE) + kl;
        float cmx = -INFINITY;  // running maximum of this lane's column over the rows of the tile
        for (int ch = 0; ok && ch < nch; ++ch, ++ccount) {
          const int buf = ccount % Cfg::NBUF;
          const bool first = ch == 0, last = ch == nch - 1;
          if (!(ok = mbar_wait_warp(&acc_full[buf], (ccount / Cfg::NBUF) & 1, ctl, STATUS_TIMEOUT_EPILOGUE))) break;
          if (Cfg::NGROUPS > 1 && first && !(ok = mbar_wait_warp(&msum_full[slot], (tcount >> 1) & 1, ctl, STATUS_TIMEOUT_EPILOGUE))) break;
          tc_fence_after_sync();
          const float m = msum[slot * BN + kl];
#pragma unroll 1
          for (int c = 0; c < BM / 32; ++c) {
            const int sb = s0 + c * 32;
            if (sb >= p.S) break;
            uint32_t v[32];
            tmem_ld_32x32(lane_base + buf * Cfg::ACC_COLS + c * 32, v);
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
                dst[g * 128] = make_float4(__uint_as_float(v[g * 4]), __uint_as_float(v[g * 4 + 1]),
                                           __uint_as_float(v[g * 4 + 2]), __uint_as_float(v[g * 4 + 3]));
              continue;
            }
#pragma unroll
            for (int e = 0; e < 32; ++e) {
              float* dst = out_col + static_cast<int64_t>(sb + e) * p.out_s1;
              const bool valid = col_ok && sb + e < p.S;
              const float acc = __uint_as_float(v[e]);
              if (split_mode) {
                if (valid) atomicAdd(dst, acc);
              } else {
                const float o = m + logf(acc);
                if (valid) {
                  *dst = o;
                  cmx = fmaxf(cmx, o);
                }
              }
            }
          }
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) {
            mbar_arrive(&acc_empty[buf]);
            if (last) mbar_arrive(&msum_empty[slot]);
          }
          if (park_it && last) {
            __threadfence();  // this lane's sums are visible ...
            __syncwarp();
            int before = 0;
            if (lane == 0) before = atomicAdd(p.park_flags + shared_tile * 4 + q, 1);  // ... before they are counted
            if (__shfl_sync(0xffffffffu, before, 0) == shared_parts - 1) {
              __threadfence();
#pragma unroll 1
              for (int c = 0; c < BM / 32; ++c) {
                const int sb = s0 + c * 32;
                if (sb >= p.S) break;
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
    } else
    for (LtItem w; ok && work.next(w); ++tcount) {
      int r, n0, s0;
      decode(w.tile, r, n0, s0);
      const int buf = tcount % Cfg::NBUF;
      const uint32_t aph = (tcount / Cfg::NBUF) & 1;
      const int slot = tcount & 1;
      if (!(ok = mbar_wait_warp(&acc_full[buf], aph, ctl, STATUS_TIMEOUT_EPILOGUE))) break;
      if (Cfg::NGROUPS > 1 && !(ok = mbar_wait_warp(&msum_full[slot], (tcount >> 1) & 1, ctl, STATUS_TIMEOUT_EPILOGUE))) break;
      tc_fence_after_sync();
      {
        const int kcol = n0 + q * 32 + lane;
        const bool col_ok = kcol < p.K;
        float* out_col = p.out + static_cast<int64_t>(r) * p.out_s0 + kcol;
        const float m = msum[slot * BN + q * 32 + lane];
        float cmx = -INFINITY;  // running maximum of this lane's column over the rows of the tile
        // One chunk = 32 rows s for this lane's column.  The loop stays rolled (two chunks per trip, the
        // next one loading while the current one is finished): unrolled, every chunk was straight-line code
        // run once per tile and the epilogue ran at instruction-fetch speed (2 000-10 000 cycles per chunk).
        auto finish = [&](const uint32_t(&cur)[32], int sb) {
          if (split_mode) {
#pragma unroll
            for (int e = 0; e < 32; ++e) {
              if (col_ok && sb + e < p.S)
                atomicAdd(out_col + static_cast<int64_t>(sb + e) * p.out_s1, __uint_as_float(cur[e]));
            }
          } else {
#pragma unroll
            for (int e = 0; e < 32; ++e) {
              const float o = m + lg2_approx(__uint_as_float(cur[e])) * LN2_F;
              if (col_ok && sb + e < p.S) {
                out_col[static_cast<int64_t>(sb + e) * p.out_s1] = o;
                cmx = fmaxf(cmx, o);
              }
            }
          }
        };
        const uint32_t acc0 = lane_base + buf * Cfg::ACC_COLS;
        uint32_t v0[32], v1[32];
        tmem_ld_32x32(acc0, v0);
#pragma unroll 1
        for (int c = 0; c < Cfg::ACC_COLS / 32; c += 2) {
          const int sb = s0 + c * 32;
          if (sb >= p.S) break;
          tmem_ld_wait();
          tmem_ld_32x32(acc0 + (c + 1) * 32, v1);
          finish(v0, sb);
          tmem_ld_wait();
          if (c + 2 < Cfg::ACC_COLS / 32) tmem_ld_32x32(acc0 + (c + 2) * 32, v0);
          if (sb + 32 < p.S) finish(v1, sb + 32);
        }
        tmem_ld_wait();
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
        mbar_arrive(&acc_empty[buf]);
        mbar_arrive(&msum_empty[slot]);
      }
    }
  } else if (Cfg::PREC && warp >= 8 + Cfg::NTW) {
    // ------------------------------------------------------------------ splitting: the low parts of the w tile
    const int t = threadIdx.x - (8 + Cfg::NTW) * 32;
    int s = 0;
    uint32_t ph = 0;
    bool ok = true;
    LtWork work(p, KBT);
    for (LtItem w; ok && work.next(w);) {
      for (int kb = w.kb_lo; kb < w.kb_hi; ++kb) {
        if (!(ok = mbar_wait_warp(&w_full[s], ph, ctl, STATUS_TIMEOUT_TRANSFORM))) break;
        write_tile_lo(stage_base + s * Cfg::STAGE, stage_base + s * Cfg::STAGE + Cfg::W_BYTES, t);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&full[s]);
        if (++s == NS) {
          s = 0;
          ph ^= 1;
        }
      }
    }
  } else if (warp >= 8) {
    // ------------------------------------------------------------------ transform: operand generator
    const int tt = threadIdx.x - 8 * 32;
    const int n = tt % BN;   // column of the tile = TMEM lane owned by this thread
    const int grp = tt / BN; // this thread's group takes every NGROUPS-th k-block
    constexpr int NG = Cfg::NGROUPS;
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + Cfg::P_COL0;
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
            const int s = my_it % NS;
            const uint32_t ph = (my_it / NS) & 1;
            const float ea = exp_shifted(acur[x], ma);
            if constexpr (Cfg::PREC != 0) {
              if (!(ok = mbar_wait_warp(&opnd_empty[s], ph ^ 1, ctl, STATUS_TIMEOUT_TRANSFORM))) break;
              tc_fence_after_sync();
#pragma unroll
              for (int h = 0; h < 2; ++h) {  // 16 of the 32 terms at a time: both words of all 32 do not fit in registers
                float hi[16], lo[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) tf32_split_rn(ea * eb[h * 16 + e], hi[e], lo[e]);
                tmem_st_32x16(lane_base + s * Cfg::P_STAGE + h * 16, hi);
                tmem_st_32x16(lane_base + s * Cfg::P_STAGE + BK + h * 16, lo);
              }
              tmem_st_wait();
              tc_fence_before_sync();
              __syncwarp();
              if (lane == 0) mbar_arrive(&full[s]);
              continue;
            }
            uint32_t pv[32];
#pragma unroll
            for (int e = 0; e < 32; ++e) pv[e] = tf32_round_bits(ea * eb[e]);
            if (!(ok = mbar_wait_warp(&opnd_empty[s], ph ^ 1, ctl, STATUS_TIMEOUT_TRANSFORM))) break;
            tc_fence_after_sync();
            tmem_st_32x32(lane_base + s * Cfg::P_STAGE, pv);
            tmem_st_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s]);
          }
        }
        it += static_cast<uint32_t>(In);
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
