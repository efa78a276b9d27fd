// lm2exp on CTA pairs with the generated operand in tensor memory (plain TF32, and 3xTF32 as the PREC instance).
//
// Same arithmetic as lm2exp_pair_kernel.cuh (replaces triturus/lm2exp.py:63-164), but the contraction is
// written transposed, D^T[k, i] = sum_j E^T[k, j] * a[i, j] with E = exp(b - m): the generated operand E^T is the
// tensor core's A operand, which tcgen05.mma can read from tensor memory, and `a` in its natural layout
// (j contiguous) is the K-major B operand.  A transform thread owns one column k of b = one TMEM lane: it
// reads its 32 values of a k-block from the b tile in shared memory (row j at 512-byte pitch, the 32 lanes of
// a warp read 128 consecutive bytes), takes the exps and writes them with one tcgen05.st.  The generated
// operand therefore never goes back to shared memory and is never read from it by the tensor core.
//
// Shared-memory bytes per k-block and CTA: 32 KB TMA in (128 rows of a, 128 columns of b), 16 KB transform
// reads, 16 KB tensor-core reads of a, 8 KB of result staging = 72 KB, against 124 KB for the kernel that keeps
// E in shared memory (which is bound by exactly that pipe: 970 cycles per k-block for 512 cycles of MMAs).
//
// One pair tile is 256 columns k (M, 128 per CTA = the CTA's TMEM lanes) x 256 rows i (N, 128 per CTA's
// shared memory).  Tensor memory per CTA: columns [0, 256) accumulator D^T, [256, 256 + 32 * NS) the E^T stages.
// The accumulator is single-buffered (a second one would leave no room for the operand), so the epilogue of a
// tile is not hidden behind the next tile's MMAs; the transform warps run ahead by NS k-blocks meanwhile.  (Short
// contractions fill and drain it in two halves, see HALVES below.  3xTF32, R32 1024^3: 1 533 cycles per k-block in the main
// loop, which is the tensor core's 1 536, and 14 400 of the 62 900 cycles of a tile in the epilogue.)
// In the transposed result a lane owns a column k, so the stabiliser m[k] is a lane constant; a 32 x 32 block of
// results is staged in shared memory (the 32 lanes of a store fill one row) and written by one TMA store; two boxes per warp alternate.
//
//   warp 0      TMA producer of ring 1: this CTA's 128 rows of a (128B swizzle).
//   warp 1      TMEM allocation; in the leader CTA the warp walks the k-blocks and one elected lane issues the pair MMAs.
//   warp 2      TMA producer of ring 2: this CTA's 128 columns of b (no swizzle).
//   warp 3      watches the a tiles land and says so on the leader's xf_done barriers (3xTF32: idle).
//   warps 4-7   epilogue (TMEM lane quarter = warp % 4).
//   warps 8-15  transform: NG = two groups of four warps (one per lane quarter) take alternate tiles of b (three
//               groups, 20 warps at 96 registers, ran 5 % slower; ring depths 6+6, 5+7, 7+5 instead of 8+4 the same).
//   warps 16-19 3xTF32: wait for the tiles of a, write their low parts to a second tile and say so on xf_done.
// 3xTF32 has four stages of 2 x 16 KB (a and its low parts) and 64 TMEM columns (both parts of E^T), takes a transposed a as
// well (MN-major tiles) and folds column maxima of the result.
#pragma once

#include "lm2exp_kernel.cuh"

namespace tb200 {

// Development aid (compiled only with -DTB200_TIMELINE, never in the shipped library): CTA 0 records clock64()
// at the hand-over points of its roles, 256 entries per slot.
#ifdef TB200_TIMELINE
__device__ long long g_timeline[16 * 256];
#define TB200_TL(slot, idx)                                                                  \
  do {                                                                                       \
    if (blockIdx.x == 0 && (idx) < 256u) g_timeline[(slot) * 256 + (idx)] = clock64();        \
  } while (0)
#else
#define TB200_TL(slot, idx) \
  do {                      \
  } while (0)
#endif

// Two rings.  Ring 1 (NS stages): a tile of `a` in shared memory together with the E^T stage in tensor memory
// that the same MMAs read; both are handed back by the MMA commit.  Ring 2 (NSB stages): the b tiles, which the
// transform threads hand back as soon as they hold the values in registers.  The chain "stage free -> TMA
// (1-2 us from L2 / HBM) -> transform -> MMA -> commit" is several thousand cycles long, so the number of
// k-blocks in flight, not any pipe, bounds a single ring of six stages (measured 1 100 cycles per k-block for
// 512 cycles of MMAs); two rings put 8 + 5 tiles in flight in the same shared memory.
template <int NS_, int NSB_, int NG_ = 2, bool OPT_ = false, bool FUSED_ = false, int PREC_ = 0, bool HALVES_ = false>
struct Lm2expTsPairCfg {
  static constexpr int BM = 128;   // columns k per CTA (256 per pair): TMEM lanes
  static constexpr int BN = 256;   // rows i per pair tile (N of the MMA), 128 per CTA's shared memory
  static constexpr int BK = 32, NG = NG_, NTW = 4 * NG_, NS = NS_, NSB = NSB_;
  static constexpr int A_TILE = 128 * BK * 4;  // this CTA's rows of a: 16 KB
  static constexpr int B_TILE = BK * BM * 4;   // this CTA's columns of b: 32 rows j x 128 k = 16 KB
  // PREC (3xTF32): e_lo * a_hi + e_hi * a_lo + e_hi * a_hi, all as tf32 MMAs.  A ring-1 stage also holds the low parts, of
  // a in a second 16 KB tile and of E^T in 32 more TMEM columns.  (The two corrections as bf16 MMAs of twice the rate,
  // both factors of a term packed into one word, ran R32 1024^3 in 234 us instead of 298 and R64
  // 512x512x256 in 51 instead of 58.  But bf16 has 8 significant bits: a single term was off by up to 7.1e-6 of itself
  // instead of 1.1e-6, and that does not average out where one term dominates a sum.)
  static constexpr int PREC = PREC_;
  static constexpr int A_STAGE = (PREC ? 2 : 1) * A_TILE;
  static constexpr int E_COLS = (PREC ? 2 : 1) * BK;  // TMEM columns of an operand stage
  static constexpr int ACC_COLS = BN;
  static constexpr int E_COL0 = ACC_COLS;  // first TMEM column of the operand stages
  static constexpr int TMEM_COLS = 512;
  static constexpr int NPW = PREC_ ? 4 : 0;  // PREC: warps that write the low parts of a (behind the transform warps)
  static constexpr int NTHREADS = (8 + NTW + NPW) * 32;
  static constexpr int EPI_STAGE = 4 * 2 * 32 * 128;  // per epilogue warp two 32 x 32 fp32 boxes
  // OPT: no stabiliser pre-pass.  The stabiliser of a column is the maximum over its first k-block (32 rows j),
  // found by the transform warp that handles that k-block and handed to the other roles through shared memory
  // (two slots of 128 floats, per-quarter barriers).  Later values may exceed it: exp(b - m) then exceeds 1,
  // which fp32 absorbs up to e^88; a result that overflowed all the same (+inf or NaN) raises *opt_flag and the
  // caller's conditional launches redo the call with the exact column maxima.
  static constexpr bool OPT = OPT_;
  // FUSED: the exact stabiliser inside the kernel (the conditional launch behind an optimistic one).  Every tile
  // starts with a max pass: its b tiles stream through ring 2 once more, each transform group keeps the running
  // maximum of its k-blocks per lane, the groups other than the first hand theirs over through shared memory,
  // and the first group publishes the column maxima like the optimistic instance publishes its estimate.
  static constexpr bool FUSED = FUSED_;
  static constexpr bool SLOTS = OPT || FUSED;  // stabilisers handed from the transform warps to the other roles
  static_assert(!(OPT && FUSED), "one or the other");
  // HALVES, for short contractions (KB <= NS, all k-blocks of a tile in the operand stages at once): the accumulator is
  // filled in two halves of 128 rows which the MMA issuer and the epilogue hand over separately, so that the epilogue of one
  // half runs under the MMAs of the other (R128 I256 J256 K8192: 482 -> 447 us).  Not beyond: N = 128 MMAs read the operand
  // in TMEM twice, and the main loop then loses more than the borders of the tiles gain (R32 1024^3: 160 -> 174 us).
  static constexpr bool HALVES = HALVES_;
  static constexpr int NH = HALVES ? 2 : 1;
  static_assert(!PREC || !HALVES, "not instantiated");
  static_assert(!PREC || !SLOTS, "3xTF32 takes its stabilisers from a pre-pass");
  static constexpr int NBAR = 3 * NS + 2 * NSB + 4 + (SLOTS ? 16 : 0) + (FUSED ? 4 * (NG - 1) : 0);
  static constexpr int M_TILE_BYTES = (SLOTS ? 2 * BM * 4 : 0) + (FUSED ? (NG - 1) * BM * 4 : 0);
  static constexpr int SMEM_BYTES = 1024 + NS * A_STAGE + NSB * B_TILE + EPI_STAGE + M_TILE_BYTES + NBAR * 8 + 64;
  static_assert(E_COL0 + NS * E_COLS <= TMEM_COLS, "TMEM capacity");
  static_assert(SMEM_BYTES <= 232448, "shared memory capacity");
};

// D[tmem] (+)= A[tmem] * B[smem] on a CTA pair: each CTA supplies its 128 rows of A from its own tensor memory
// (same address in both) and its half of the N rows of B from its own shared memory (same offset in both).
__device__ __forceinline__ void umma_tf32_ts_pair(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                                  uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::tf32 [%0], [%1], %2, %3, p;\n\t"
      "}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

template <class Cfg>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(Cfg::NTHREADS, 1)
lm2exp_tspair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                     const __grid_constant__ CUtensorMap tmap_out, const Lm2expParams p) {
  constexpr int BM = Cfg::BM, BN = Cfg::BN, BK = Cfg::BK, NS = Cfg::NS, NSB = Cfg::NSB;

  // A conditional launch: runs only if the launch before it raised the flag (same value for every thread of
  // both CTAs, read before any barrier or allocation exists).
  if (p.only_if != nullptr) {
    pdl_wait();  // (launched as a programmatic dependent of the kernel that may have raised the flag)
    if (*p.only_if == 0) return;
    // (a flag republished in a second word by a conditional pre-pass: all readers of the first one are done)
    if (!Cfg::FUSED && blockIdx.x == 0 && threadIdx.x == 0 && p.reset_flag != nullptr) *p.reset_flag = 0;
  }
  // Optimistic instances let the conditional launch behind them take its place as this grid's CTAs leave, and
  // clear the counter with which that launch, should it run, finds its last CTA (nothing else uses the word
  // while this kernel runs).
  if (Cfg::OPT) {
    pdl_launch_dependents();
    if (blockIdx.x == 0 && threadIdx.x == 0) p.opt_flag[1] = 0;
  }

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* a_base = smem;                     // ring 1: NS tiles of a
  uint8_t* b_base = smem + NS * Cfg::A_STAGE;  // ring 2: NSB tiles of b
  uint8_t* epi_stage = b_base + NSB * Cfg::B_TILE;  // 4 warps x 4 KB staging boxes, 1024-byte aligned
  float* m_tile = reinterpret_cast<float*>(epi_stage + Cfg::EPI_STAGE);  // OPT: [2][BM] stabilisers of two tiles
  uint64_t* bars = reinterpret_cast<uint64_t*>(epi_stage + Cfg::EPI_STAGE + Cfg::M_TILE_BYTES);
  uint64_t* a_full = bars;                // [NS] this CTA's tile of a landed
  uint64_t* xf_done = bars + NS;          // [NS] (leader's copy is used) E^T stage written and a landed, both CTAs
  uint64_t* stage_empty = bars + 2 * NS;  // [NS] pair MMAs reading ring-1 stage retired (committed by the leader)
  uint64_t* b_full = bars + 3 * NS;       // [NSB] this CTA's tile of b landed
  uint64_t* b_empty = b_full + NSB;       // [NSB] the four transform warps of the k-block hold it in registers
  uint64_t* acc_full = b_empty + NSB;     // [NH] accumulator (half) complete (committed by the leader)
  uint64_t* acc_empty = acc_full + 2;     // [NH] (leader's copy is used) epilogues of both CTAs drained it
  uint64_t* m_ready = acc_empty + 2;      // SLOTS [2][4] slot, lane quarter: stabilisers written
  uint64_t* m_free = m_ready + 8;         // SLOTS [2][4] every reader of the quarter (epilogue warp, other groups) is done
  uint64_t* part_ready = m_free + 8;      // FUSED [NG - 1][4] group g > 0, lane quarter: its partial maxima written
  float* m_part = m_tile + 2 * BM;        // FUSED [NG - 1][BM] partial column maxima of the groups other than the first
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2 + (Cfg::SLOTS ? 16 : 0) +
                                                    (Cfg::FUSED ? 4 * (Cfg::NG - 1) : 0));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = warp_uniform(threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const uint32_t rank = warp_uniform(cluster_ctarank());  // 0 = leader
  const bool leader = rank == 0;
  const AbortCtl ctl{abort_flag, p.status};

  auto a_tile = [&](int s) -> uint8_t* { return a_base + s * Cfg::A_STAGE; };
  auto b_tile = [&](int s) -> uint8_t* { return b_base + s * Cfg::B_TILE; };

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < NS; ++s) {
      mbar_init(&a_full[s], 1);
      mbar_init(&xf_done[s], 2 * 4 + 2 * (Cfg::PREC ? Cfg::NPW : 1));  // four transform warps (one per lane quarter) and the a-tile watcher (PREC: the splitting warps), in each CTA
      mbar_init(&stage_empty[s], 1);
    }
    for (int s = 0; s < NSB; ++s) {
      mbar_init(&b_full[s], 1);
      mbar_init(&b_empty[s], 4);
    }
    for (int h = 0; h < Cfg::NH; ++h) {
      mbar_init(&acc_full[h], 1);
      mbar_init(&acc_empty[h], 8);
    }
    if (Cfg::SLOTS) {
      for (int i = 0; i < 8; ++i) {
        mbar_init(&m_ready[i], 1);
        mbar_init(&m_free[i], Cfg::NG);  // the epilogue warp and one warp of every other transform group
      }
    }
    if (Cfg::FUSED) {
      for (int i = 0; i < 4 * (Cfg::NG - 1); ++i) mbar_init(&part_ready[i], 1);
    }
    fence_mbar_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    if (p.out_tma) tma_prefetch_desc(&tmap_out);
  }
  // Both CTAs run and have initialised their barriers before anything crosses between them.  The pair allocation
  // below is such a crossing (it takes both CTAs' tensor memory): the CTAs of a cluster do not start at the same
  // instant, and an allocation by the first one before the second exists is an access to an absent block.
  cluster_sync_all();
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, Cfg::TMEM_COLS);
    tmem_relinquish_pair();
  }
  // The leader's MMAs write both CTAs' tensor memory: both allocations are done before the roles start.
  tc_fence_before_sync();
  cluster_sync_all();
  tc_fence_after_sync();
  const uint32_t tmem_base = warp_uniform(*tmem_slot);

  const int KB = (p.J + BK - 1) / BK;
  const int npairs = gridDim.x >> 1;
  const int pair = blockIdx.x >> 1;

  // Pair tile id -> (batch r, first column k, first row i of the 256 x 256 tile); row tiles vary fastest.
  auto decode = [&](int tile, int& r, int& n0, int& i0) {
    const int tm = tile % p.tiles_m;
    const int rest = tile / p.tiles_m;
    const int tn = rest % p.tiles_n;
    r = rest / p.tiles_n;
    n0 = tn * (2 * BM);
    i0 = tm * BN;
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer, ring 1: this CTA's rows of a
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      for (int tile = pair; ok && tile < p.num_tiles; tile += npairs) {
        int r, n0, i0;
        decode(tile, r, n0, i0);
        const int my_i0 = i0 + static_cast<int>(rank) * 128;
        for (int kb = 0; kb < KB; ++kb, ++it) {
          const int s = it % NS;
          const uint32_t ph = (it / NS) & 1;
          if (!(ok = mbar_wait(&stage_empty[s], ph ^ 1, ctl, STATUS_TIMEOUT_PRODUCER))) break;
          TB200_TL(9, it);
          mbar_arrive_expect_tx(&a_full[s], Cfg::A_TILE);
          if (Cfg::PREC && p.a_mn) {
#pragma unroll
            for (int g = 0; g < 4; ++g) tma_load_3d(a_tile(s) + g * 4096, &tmap_a, &a_full[s], my_i0 + g * 32, kb * BK, r);
          } else {
            tma_load_3d(a_tile(s), &tmap_a, &a_full[s], kb * BK, my_i0, r);
          }
        }
      }
      // The leader's commits arrive on both CTAs' stage_empty barriers: this CTA stays until the last ones are in.
      for (uint32_t d = ok ? min(it, static_cast<uint32_t>(NS)) : 0u; ok && d > 0; --d)
        ok = mbar_wait(&stage_empty[(it - d) % NS], ((it - d) / NS) & 1, ctl, STATUS_TIMEOUT_PRODUCER);
    }
    __syncwarp();
  } else if (warp == 2) {
    // ------------------------------------------------------------------ TMA producer, ring 2: this CTA's columns of b
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      for (int tile = pair; ok && tile < p.num_tiles; tile += npairs) {
        int r, n0, i0;
        decode(tile, r, n0, i0);
        const int my_n0 = n0 + static_cast<int>(rank) * BM;
        for (int pass = Cfg::FUSED ? 0 : 1; ok && pass < 2; ++pass) {  // 0 = max pass, 1 = contraction
          for (int kb = 0; kb < KB; ++kb, ++it) {
            const int s = it % NSB;
            const uint32_t ph = (it / NSB) & 1;
            if (!(ok = mbar_wait(&b_empty[s], ph ^ 1, ctl, STATUS_TIMEOUT_PRODUCER))) break;
            TB200_TL(10, it);
            mbar_arrive_expect_tx(&b_full[s], Cfg::B_TILE);
            tma_load_3d(b_tile(s), &tmap_b, &b_full[s], my_n0, kb * BK, r);
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ pair MMA issuer (leader CTA only)
    // The whole warp runs the loop and one elected lane issues: control flow and descriptors are uniform and stay in uniform
    // registers.  (One lane in a branch of its own took 80 - 100 cycles per MMA for moving them there, more than the 64 to
    // 128 of the MMA itself: 750 cycles per k-block in plain TF32.)
    if (leader) {
      // M = 256 columns k over the pair (A from TMEM), N = 256 rows i (B = a, K-major, 128 rows per CTA)
      // PREC takes a transposed a too: MN-major (bit 16), its low parts in the same layout.
      const bool a_mn = Cfg::PREC && p.a_mn != 0;
      const uint32_t idesc = umma_idesc_tf32(2 * BM, BN / Cfg::NH) | (a_mn ? 1u << 16 : 0u);
      const uint32_t a_step = a_mn ? 64u : 2u;  // encoded address step per 8 contraction values
      constexpr uint32_t HALF_ENC = (64 * BK * 4) >> 4;  // 64 rows of a further
      constexpr uint32_t STAGE_ENC = Cfg::A_STAGE >> 4;
      const uint64_t db0 = a_mn ? umma_desc_mn_sw128_base32(smem_u32(a_tile(0)), 4096) : umma_desc_k_sw128(smem_u32(a_tile(0)));
      uint32_t s = 0, ph = 0, tcount = 0;
      bool ok = true;
      auto advance = [&]() {
        if (++s == NS) {
          s = 0;
          ph ^= 1;
        }
      };
      // One k-block: all 256 rows, or (HALVES) rows h * 64 .. + 63 of both CTAs into accumulator half h.
      auto issue = [&](uint32_t st, uint32_t h, bool accumulate) {
        const uint32_t d = tmem_base + h * (BN / 2);
        const uint64_t db = db0 + st * STAGE_ENC + h * HALF_ENC;
        const uint32_t ea = tmem_base + Cfg::E_COL0 + st * Cfg::E_COLS;
        if (Cfg::PREC) {
          // The corrections first, while the accumulator of a tile is empty: the sum of the first k-block's is not
          // truncated to the bits of the whole sum then.
#pragma unroll
          for (int ks = 0; ks < BK / 8; ++ks)
            umma_tf32_ts_pair(d, ea + BK + ks * 8, db + a_step * ks, idesc, (accumulate || ks > 0) ? 1u : 0u);
#pragma unroll
          for (int ks = 0; ks < BK / 8; ++ks)
            umma_tf32_ts_pair(d, ea + ks * 8, db + (Cfg::A_TILE >> 4) + a_step * ks, idesc, 1u);
        }
#pragma unroll
        for (int ks = 0; ks < BK / 8; ++ks)
          umma_tf32_ts_pair(d, ea + ks * 8, db + a_step * ks, idesc, (Cfg::PREC || accumulate || ks > 0) ? 1u : 0u);
      };
      for (int tile = pair; ok && tile < p.num_tiles; tile += npairs, ++tcount) {
        TB200_TL(11, tcount);
        if (!(ok = mbar_wait_warp(&acc_empty[0], (tcount & 1) ^ 1, ctl, STATUS_TIMEOUT_MMA))) break;
        TB200_TL(12, tcount);
        tc_fence_after_sync();
        if (Cfg::HALVES) {
          // The first half of the accumulator takes all k-blocks of the tile (they fit the operand stages) as soon as the
          // epilogue of the previous tile has drained it, the second half when it is drained too.
          const uint32_t s_first = s;
          for (int kb = 0; kb < KB; ++kb) {
            if (!(ok = mbar_wait_warp(&xf_done[s], ph, ctl, STATUS_TIMEOUT_MMA))) break;
            TB200_TL(0, tcount * KB + kb);
            tc_fence_after_sync();
            if (elect_one_sync()) issue(s, 0, kb > 0);
            __syncwarp();
            advance();
          }
          if (!ok) break;
          if (elect_one_sync()) umma_commit_pair_mcast(smem_u32(&acc_full[0]), 3);
          if (!(ok = mbar_wait_warp(&acc_empty[1], (tcount & 1) ^ 1, ctl, STATUS_TIMEOUT_MMA))) break;
          tc_fence_after_sync();
          for (int kb = 0; kb < KB; ++kb) {
            const uint32_t st = s_first + kb < NS ? s_first + kb : s_first + kb - NS;
            if (elect_one_sync()) {
              issue(st, 1, kb > 0);
              // free the stage (shared memory and TMEM) in both CTAs once these MMAs retire
              umma_commit_pair_mcast(smem_u32(&stage_empty[st]), 3);
            }
            __syncwarp();
            TB200_TL(1, tcount * KB + kb);
          }
          if (elect_one_sync()) umma_commit_pair_mcast(smem_u32(&acc_full[1]), 3);
        } else {
          for (int kb = 0; kb < KB; ++kb) {
            if (!(ok = mbar_wait_warp(&xf_done[s], ph, ctl, STATUS_TIMEOUT_MMA))) break;
            TB200_TL(0, tcount * KB + kb);
            tc_fence_after_sync();
            if (elect_one_sync()) {
              issue(s, 0, kb > 0);
              umma_commit_pair_mcast(smem_u32(&stage_empty[s]), 3);
            }
            __syncwarp();
            TB200_TL(1, tcount * KB + kb);
            advance();
          }
          if (ok && elect_one_sync()) umma_commit_pair_mcast(smem_u32(&acc_full[0]), 3);
        }
      }
    }
    __syncwarp();
  } else if (warp == 3 && !Cfg::PREC) {
    // ------------------------------------------------------------------ a-tile watcher
    // (3xTF32: the splitting warps wait for the tile of a)
    // The leader's MMA thread reads both CTAs' tiles of a and waits only on xf_done: this lane adds "this CTA's
    // tile of a has landed" to that barrier, so that the transform warps need not wait for it in their chain.
    if (lane == 0) {
      const uint32_t xf_done_leader0 = map_to_cta(smem_u32(&xf_done[0]), 0);
      uint32_t it = 0;
      bool ok = true;
      for (int tile = pair; ok && tile < p.num_tiles; tile += npairs) {
        for (int kb = 0; kb < KB; ++kb, ++it) {
          const int s = it % NS;
          if (!(ok = mbar_wait(&a_full[s], (it / NS) & 1, ctl, STATUS_TIMEOUT_TRANSFORM))) break;
          mbar_arrive_cluster(xf_done_leader0 + static_cast<uint32_t>(s) * 8u);
        }
      }
    }
    __syncwarp();
  } else if (warp >= 4 && warp < 8) {
    // ------------------------------------------------------------------ epilogue (this CTA's 128 columns k x 256 rows i)
    const int q = warp & 3;
    uint8_t* stg2 = epi_stage + q * 8192;  // two boxes: one is filled while the TMA unit still reads the other
    uint32_t nbox = 0;
    const bool use_tma = p.out_tma != 0;
    const uint32_t acc_empty_leader0 = map_to_cta(smem_u32(acc_empty), 0);
    const uint32_t tbase = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
    pdl_wait();  // m comes from the pre-pass, which may still be running when this kernel starts
    uint32_t tcount = 0;
    bool ok = true;
    const bool opt = Cfg::OPT || (Cfg::PREC && p.opt_flag != nullptr);  // PREC: pre-pass over the first 32 rows only
    uint32_t acc_max = 0;  // opt: largest accumulator bit pattern of this lane (sums of non-negative products, so
                           // +inf and NaN are exactly the patterns >= 0x7f800000 read as unsigned)
    for (int tile = pair; ok && tile < p.num_tiles; tile += npairs, ++tcount) {
      int r, n0, i0;
      decode(tile, r, n0, i0);
      const int k0 = n0 + static_cast<int>(rank) * BM + q * 32;  // first column of this warp's 32
      const int kcol = k0 + lane;
      const bool col_ok = kcol < p.K;
      float m = 0.f;
      if (!Cfg::SLOTS && col_ok) m = clamp_stab(__ldg(p.m_ws + static_cast<int64_t>(r) * p.K + kcol));
      float* ocol = p.out + static_cast<int64_t>(r) * p.out_s0 + kcol;
      float cmx = -INFINITY;  // PREC: largest result of this lane's column in the tile, for the next layer of a chain
      // Accumulator column c holds row i0 + c; in halves, columns 128 hf + (0 .. 63) the leader's rows of a, i0 + 64 hf on,
      // and the 64 behind them the other CTA's, i0 + 128 + 64 hf on.
#pragma unroll 1
      for (int hf = 0; ok && hf < Cfg::NH; ++hf) {
      const uint32_t acc_empty_leader = acc_empty_leader0 + static_cast<uint32_t>(hf) * 8u;
      if (!(ok = mbar_wait_warp(&acc_full[hf], tcount & 1, ctl, STATUS_TIMEOUT_EPILOGUE))) break;
      if (warp == 4 && lane == 0) TB200_TL(7, tcount);
      tc_fence_after_sync();
      if (Cfg::SLOTS && hf == 0) {
        // the stabilisers this tile was computed with (written long before the accumulator completed)
        const uint32_t slot = (tcount & 1) * 4 + q;
        if (!(ok = mbar_wait_warp(&m_ready[slot], (tcount >> 1) & 1, ctl, STATUS_TIMEOUT_EPILOGUE))) break;
        const float mt = m_tile[(tcount & 1) * BM + q * 32 + lane];
        m = col_ok ? mt : 0.f;
        __syncwarp();
        if (lane == 0) mbar_arrive(&m_free[slot]);
      }
      const int row0 = i0 + hf * 64;
      const int nchunks = k0 >= p.K ? 0
                          : Cfg::HALVES ? min(2, max(0, (p.I - row0 + 31) / 32)) + min(2, max(0, (p.I - row0 - 128 + 31) / 32))
                                        : min(BN / 32, (p.I - i0 + 31) / 32);
      if (nchunks == 0) {
        // nothing to store (this warp's columns are padding): release the accumulator right away
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(acc_empty_leader);
        continue;
      }
      uint32_t v[2][32];
      tmem_ld_32x32(tbase + hf * (BN / 2), v[0]);
#pragma unroll 1
      for (int idx = 0; idx < nchunks; idx += Cfg::PREC ? 1 : 2) {
#pragma unroll
        for (int h = 0; h < (Cfg::PREC ? 1 : 2); ++h) {
          const int c = idx + h;
          if (c < nchunks) {
            // (PREC: one buffer, the logarithms want the registers of the second: R64 512x512x256 72.5 -> 63.6 us, R32 1024^3
            // 349 -> 321 us)
            if (Cfg::PREC && c > 0) tmem_ld_32x32(tbase + hf * (BN / 2) + c * 32, v[Cfg::PREC ? 0 : h]);
            tmem_ld_wait();  // chunk c is in v[h]
            if (!Cfg::PREC && c + 1 < nchunks) {
              tmem_ld_32x32(tbase + hf * (BN / 2) + (c + 1) * 32, v[h ^ 1]);
            } else if (c + 1 == nchunks) {
              // all of it is in registers: hand it back to the MMA issuer
              tc_fence_before_sync();
              __syncwarp();
              if (lane == 0) mbar_arrive_cluster(acc_empty_leader);
            }
            const int ib = row0 + c * 32 + (Cfg::HALVES && c >= 2 ? 64 : 0);
            if (Cfg::PREC) {
              // (lg2.approx of the mantissa is off by 2^-22 whatever the result, several ulp for sums near 1; it ran R32
              // 1024^3 in 308 us instead of 318 and R64 512x512x256 in 60 instead of 63.  A polynomial good to one ulp,
              // on two values per instruction: 317 and 63.)
#pragma unroll
              for (int e = 0; e < 32; ++e) {
                acc_max = max(acc_max, v[h][e]);
                v[h][e] = __float_as_uint(logf(__uint_as_float(v[h][e])));
              }
            }
            // Register e of this lane is row ib + e, column kcol of the result.  The 32 x 32 block goes through a
            // staging box (row e at byte e * 128 in the 128-byte swizzle, the 32 lanes of a store fill one row)
            // and from there as one TMA store: per-row stores straight from the registers ran at ~70 cycles per
            // row.
            if (use_tma) {
              uint8_t* stg = stg2 + (nbox & 1) * 4096;
              ++nbox;
              if (lane == 0) tma_store_wait_read<1>();  // the store before the previous one has read this box out
              __syncwarp();
#pragma unroll
              for (int e = 0; e < 32; ++e) {
                const float acc = __uint_as_float(v[h][e]);
                const float o = m + (Cfg::PREC ? acc : lg2_approx(acc) * LN2_F);
                if (Cfg::OPT) acc_max = max(acc_max, v[h][e]);
                if (Cfg::PREC) cmx = fmaxf(cmx, o);  // (rows past I hold log 0 = -inf)
                *reinterpret_cast<float*>(stg + sw128_offset(e, lane)) = o;
              }
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
                const float acc = __uint_as_float(v[h][e]);
                const float o = m + (Cfg::PREC ? acc : lg2_approx(acc) * LN2_F);
                if (Cfg::OPT) acc_max = max(acc_max, v[h][e]);
                if (Cfg::PREC) cmx = fmaxf(cmx, o);  // (rows past I hold log 0 = -inf)
                if (col_ok && e < nrows) orow[static_cast<int64_t>(e) * p.out_s1] = o;
              }
            }
          }
        }
      }
      if (warp == 4 && lane == 0) TB200_TL(8, tcount);
      }
      if (Cfg::PREC && ok && p.out_max != nullptr && col_ok) red_max_f32(p.out_max + static_cast<int64_t>(r) * p.K + kcol, cmx);
    }
    if (use_tma && lane == 0) tma_store_wait_all();  // shared memory must outlive the last box
    if (opt) {
      if (__any_sync(0xffffffffu, acc_max >= 0x7f800000u) && lane == 0) *p.opt_flag = 1;
    }
  } else if (Cfg::PREC && warp >= 8 + Cfg::NTW) {
    // ------------------------------------------------------------------ splitting: the low parts of the tile of a
    // The tile itself stays as it is (the tensor core drops the low 13 bits).
    const int t = threadIdx.x - (8 + Cfg::NTW) * 32;
    const uint32_t xf_done_leader0 = map_to_cta(smem_u32(&xf_done[0]), 0);
    uint32_t it = 0;
    bool ok = true;
    for (int tile = pair; ok && tile < p.num_tiles; tile += npairs) {
      for (int kb = 0; kb < KB; ++kb, ++it) {
        const int s = it % NS;
        if (!(ok = mbar_wait_warp(&a_full[s], (it / NS) & 1, ctl, STATUS_TIMEOUT_TRANSFORM))) break;
        write_tile_lo(a_tile(s), a_tile(s) + Cfg::A_TILE, t);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(xf_done_leader0 + static_cast<uint32_t>(s) * 8u);
      }
    }
  } else if (warp >= 8) {
    // ------------------------------------------------------------------ transform: b tile -> E^T in tensor memory
    const int q = warp & 3;         // TMEM lane quarter this warp may write
    // This warp's group takes every NG-th tile of ring 2, counted over the whole launch and not per output tile: a
    // slot of the ring (NSB is a multiple of NG) then always belongs to the same group, which has waited for the
    // slot's previous tile before it waits for the next one.  A wait by parity is only meaningful under that
    // condition: counted per output tile, an odd number of k-blocks swapped the groups' slots at every tile, a group
    // could look at a slot whose previous load (the other group's) had not landed, take the phase before that for its
    // own, and hand the slot back twice.
    const int grp = (warp - 8) >> 2;
    static_assert(NSB % Cfg::NG == 0, "a ring-2 slot belongs to one transform group");
    const int kl = q * 32 + lane;
    const uint32_t ebase = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + Cfg::E_COL0;
    const uint32_t xf_done_leader0 = map_to_cta(smem_u32(&xf_done[0]), 0);
    pdl_wait();  // m comes from the pre-pass (the producer warp is already loading operand tiles meanwhile)
    uint32_t it0 = 0, itb0 = 0, tcount = 0;  // k-blocks of ring 1 / tiles of ring 2 before this tile; tiles seen
    bool ok = true;
    for (int tile = pair; ok && tile < p.num_tiles; tile += npairs, ++tcount) {
      int r, n0, i0;
      decode(tile, r, n0, i0);
      const int kcol = n0 + static_cast<int>(rank) * BM + kl;
      // A column past K reads zero-filled values; the stabiliser +inf turns them into exact zeros.
      float m = INFINITY;
      if (!Cfg::SLOTS && kcol < p.K) m = clamp_stab(__ldg(p.m_ws + static_cast<int64_t>(r) * p.K + kcol));
      const auto first_kb = [&](uint32_t itb_tile) -> int {  // this group's first k-block of a pass that starts at ring-2 tile itb_tile
        return (grp + Cfg::NG - static_cast<int>(itb_tile % Cfg::NG)) % Cfg::NG;
      };
      const uint32_t mslot = (tcount & 1) * 4 + q;
      float* mdst = m_tile + (tcount & 1) * BM + kl;
      if (Cfg::FUSED) {
        // ---- max pass: running maximum of this lane's column over the k-blocks of this group
        float mx = -INFINITY;
        for (int kb = first_kb(itb0); kb < KB; kb += Cfg::NG) {
          const uint32_t itb = itb0 + static_cast<uint32_t>(kb);
          const int sb = itb % NSB;
          if (!(ok = mbar_wait_warp(&b_full[sb], (itb / NSB) & 1, ctl, STATUS_TIMEOUT_TRANSFORM))) break;
          const float* col = reinterpret_cast<const float*>(b_tile(sb)) + kl;
          const int jrem = p.J - kb * BK;  // rows past J are zero-filled by TMA and must not enter the maximum
#pragma unroll
          for (int x = 0; x < 32; ++x) mx = fmaxf(mx, x < jrem ? col[x * BM] : -INFINITY);
          __syncwarp();
          if (lane == 0) mbar_arrive(&b_empty[sb]);
        }
        if (!ok) break;
        itb0 += static_cast<uint32_t>(KB);
        if (grp != 0) {
          // (rewritten only after this warp has seen m_ready of the tile, i.e. after the first group read it)
          m_part[(grp - 1) * BM + kl] = mx;
          __syncwarp();
          if (lane == 0) mbar_arrive(&part_ready[(grp - 1) * 4 + q]);
        } else {
          for (int g = 1; g < Cfg::NG; ++g) {
            if (!(ok = mbar_wait_warp(&part_ready[(g - 1) * 4 + q], tcount & 1, ctl, STATUS_TIMEOUT_TRANSFORM))) break;
            mx = fmaxf(mx, m_part[(g - 1) * BM + kl]);
          }
          if (!ok) break;
          m = (kcol < p.K) ? clamp_stab(mx) : INFINITY;
          if (tcount >= 2) {
            if (!(ok = mbar_wait_warp(&m_free[mslot], ((tcount >> 1) - 1) & 1, ctl, STATUS_TIMEOUT_TRANSFORM))) break;
          }
          *mdst = m;
          __syncwarp();
          if (lane == 0) mbar_arrive(&m_ready[mslot]);
        }
      }
      // The group of k-block 0 publishes the tile's stabilisers; the other groups pick them up.  In the optimistic
      // instance that is done after the loads of the group's own first k-block are in flight (that group
      // publishes as soon as it holds k-block 0, i.e. at about the same time), not before them.
      const int kb_first = first_kb(itb0);
      bool need_m = Cfg::SLOTS && (Cfg::OPT ? kb_first != 0 : grp != 0);
      auto fetch_m = [&]() -> bool {
        if (!mbar_wait_warp(&m_ready[mslot], (tcount >> 1) & 1, ctl, STATUS_TIMEOUT_TRANSFORM)) return false;
        m = *mdst;
        __syncwarp();
        if (lane == 0) mbar_arrive(&m_free[mslot]);
        need_m = false;
        return true;
      };
      if (need_m && Cfg::FUSED) {
        if (!(ok = fetch_m())) break;
      }
      for (int kb = kb_first; kb < KB; kb += Cfg::NG) {
        const uint32_t it = it0 + static_cast<uint32_t>(kb);
        const int s = it % NS;
        const uint32_t ph = (it / NS) & 1;
        const uint32_t itb = itb0 + static_cast<uint32_t>(kb);
        const int sb = itb % NSB;
        if (!(ok = mbar_wait_warp(&b_full[sb], (itb / NSB) & 1, ctl, STATUS_TIMEOUT_TRANSFORM))) break;
        if (warp == 8 && lane == 0) TB200_TL(2, it);
        const float* col = reinterpret_cast<const float*>(b_tile(sb)) + kl;
        float v[32];
#pragma unroll
        for (int x = 0; x < 32; ++x) v[x] = col[x * BM];
        const int jrem = p.J - kb * BK;
        if (need_m) {
          if (!(ok = fetch_m())) break;
        }
        if (Cfg::OPT && kb == 0) {
          // stabiliser = maximum over the first k-block; the slot's readers of two tiles ago are done
          float mx = -INFINITY;
#pragma unroll
          for (int x = 0; x < 32; ++x) mx = fmaxf(mx, x < jrem ? v[x] : -INFINITY);
          m = (kcol < p.K) ? clamp_stab(mx) : INFINITY;
          if (tcount >= 2) {
            if (!(ok = mbar_wait_warp(&m_free[mslot], ((tcount >> 1) - 1) & 1, ctl, STATUS_TIMEOUT_TRANSFORM))) break;
          }
          *mdst = m;
          __syncwarp();
          if (lane == 0) mbar_arrive(&m_ready[mslot]);
        }
        uint32_t e[32];
        if (Cfg::PREC) {
          // (the exps stay in fp32 until the stage is free and are split there, 16 at a time: both words of all 32 do not
          // fit in the 96 registers of a thread)
#pragma unroll
          for (int x = 0; x < 32; ++x) e[x] = __float_as_uint(exp_shifted(x < jrem ? v[x] : -INFINITY, m));
        } else if (jrem >= BK) {
#pragma unroll
          for (int x = 0; x < 32; ++x) e[x] = tf32_round_bits(exp_shifted(v[x], m));
        } else {
          // rows past J are zero-filled by TMA (in log space): they enter the exp as -inf, exact zero out
#pragma unroll
          for (int x = 0; x < 32; ++x) e[x] = tf32_round_bits(exp_shifted(x < jrem ? v[x] : -INFINITY, m));
        }
        // Every lane has consumed its values of the b tile: hand the tile back to its producer.
        __syncwarp();
        if (lane == 0) mbar_arrive(&b_empty[sb]);
        // The E^T stage is free once the MMAs that read it last time have retired.  (That the tile of a the same
        // MMAs will read has landed is the watcher warp's part of xf_done.)
        if (!(ok = mbar_wait_warp(&stage_empty[s], ph ^ 1, ctl, STATUS_TIMEOUT_TRANSFORM))) break;
        if (warp == 8 && lane == 0) TB200_TL(4, it);
        tc_fence_after_sync();
        if constexpr (Cfg::PREC != 0) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float hi[16], lo[16];
#pragma unroll
            for (int x = 0; x < 16; ++x) tf32_split_rn(__uint_as_float(e[h * 16 + x]), hi[x], lo[x]);
            tmem_st_32x16(ebase + s * Cfg::E_COLS + h * 16, hi);
            tmem_st_32x16(ebase + s * Cfg::E_COLS + BK + h * 16, lo);
          }
        } else {
          tmem_st_32x32(ebase + s * Cfg::E_COLS, e);
        }
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(xf_done_leader0 + static_cast<uint32_t>(s) * 8u);
        if (warp == 8 && lane == 0) TB200_TL(6, it);
      }
      if (need_m) {  // (a group without a k-block in this tile still reads and releases the slot)
        if (!(ok = fetch_m())) break;
      }
      it0 += static_cast<uint32_t>(KB);
      itb0 += static_cast<uint32_t>(KB);
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
  if (Cfg::FUSED && p.reset_flag != nullptr && threadIdx.x == 0) {
    // A conditional launch that ran: every CTA read the flag when it started, so the CTA that finishes last may
    // put it down (the word behind it counts the finished CTAs; the optimistic launch before this one cleared it).
    __threadfence();
    if (atomicAdd(p.reset_flag + 1, 1) == static_cast<int>(gridDim.x) - 1) {
      p.reset_flag[1] = 0;
      p.reset_flag[0] = 0;
    }
  }
}

}  // namespace tb200
