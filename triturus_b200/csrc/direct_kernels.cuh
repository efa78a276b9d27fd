// Small problems: lm2exp and lt2exp for calls whose time is latency and not arithmetic.
//
// The tcgen05 kernels need some 15 us for the smallest call: barriers and tensor memory to set up, b through the ring twice, an
// accumulator that comes back through tensor memory and a staging box, all in code that runs once.  Here a block of eight
// warps takes a 32 x 32 tile of the result: what it reads goes to shared memory with asynchronous copies in one go
// (whatever the strides and alignments: 4 bytes each, 16 where the layout allows), the column maxima and exps are taken
// there once, and each warp sums its share of the contraction in registers with mma.sync m16n8k8 on tf32 operands, whose
// operands and results are plain registers; what tcgen05 has over it in rate does not show at these sizes.
// The warps' sums meet in shared memory in a fixed order, as rounded fp32 adds.
//   plain TF32: both operands rounded to nearest tf32.  3xTF32: the three products of the tcgen05 kernels, in their order.
#pragma once

#include "ptx.cuh"

namespace tb200 {

constexpr int DIRECT_THREADS = 256;
constexpr int DIRECT_PITCH = 40;  // floats between rows of 32 columns: 8 modulo 32, so that four rows x eight columns (a
                                  // B fragment) and eight rows x four pairs (results) are in different banks
constexpr int DIRECT_RED_FLOATS = 8 * 32 * DIRECT_PITCH;  // the warps' partial sums, over the operands

// Contraction length padded to whole MMAs, and the pitch of rows along it: 4 modulo 8, so that eight rows x four columns (an A
// fragment) are in different banks.
__host__ __device__ constexpr int direct_round8(int n) { return (n + 7) & ~7; }
__host__ __device__ constexpr int direct_pitch(int n) { return direct_round8(n) + 4; }

// W consecutive floats (1, 2 or 4, aligned to their size) to shared memory; zeros where !valid (the source is not read then).
template <int W>
__device__ __forceinline__ void cp_async_floats(uint32_t smem_dst, const float* src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(smem_dst), "l"(src), "n"(4 * W), "r"(valid ? 4 * W : 0) : "memory");
}

// dst[row * DIRECT_PITCH + c] = src[row * s_row + c * s_col] for row < n, c < cols, by the block.  W floats at a time: s_col = 1 if
// W > 1.  Rows and columns beyond stay as they are (direct_exp_columns writes them).
template <int W>
__device__ __forceinline__ void direct_load_columns(float* dst, const float* src, int64_t s_row, int64_t s_col, int n, int cols, int tid) {
  constexpr int LANES = 32 / W, STEP = DIRECT_THREADS / LANES;
  const int c = (tid % LANES) * W, row0 = tid / LANES;
  if (c >= cols) return;
  const float* x = src + row0 * s_row + c * s_col;
  uint32_t d = smem_u32(dst + row0 * DIRECT_PITCH + c);
#pragma unroll 4
  for (int row = row0; row < n; row += STEP, x += STEP * s_row, d += STEP * DIRECT_PITCH * 4) cp_async_floats<W>(d, x, true);
}
__device__ __forceinline__ void direct_load_columns(float* dst, const float* src, int64_t s_row, int64_t s_col, int n, int cols, int width,
                                                    int tid) {
  if (width == 4) {
    direct_load_columns<4>(dst, src, s_row, 1, n, cols, tid);
  } else if (width == 2) {
    direct_load_columns<2>(dst, src, s_row, 1, n, cols, tid);
  } else if (s_col == 1 || s_row != 1) {
    direct_load_columns<1>(dst, src, s_row, s_col, n, cols, tid);
  } else {
    // Consecutive rows, a transposed view: a warp takes eight rows of four columns, whole sectors of 32 bytes and two lanes to a
    // bank.  (A row of 32 columns at a time is a sector per value: 16 x 256^3 50 us in 3xTF32, 4 x 256^3 15.6 in TF32.)
    const int c = (tid >> 5) * 4 + ((tid >> 3) & 3);
    if (c >= cols) return;
    const float* x = src + (tid & 7) + c * s_col;
    uint32_t d = smem_u32(dst + (tid & 7) * DIRECT_PITCH + c);
#pragma unroll 4
    for (int row = tid & 7; row < n; row += 8, x += 8, d += 8 * DIRECT_PITCH * 4) cp_async_floats<1>(d, x, true);
  }
}

// dst[row * pitch + x] = src[row * s_row + x * s_x] for row < rows, x < n, zeros for n <= x < n8, by warps w of nw.  W floats at a
// time: s_x = 1 and n a multiple of W if W > 1.
template <int W>
__device__ __forceinline__ void direct_load_rows(float* dst, int pitch, const float* src, int64_t s_row, int64_t s_x, int rows, int n, int n8,
                                                 int w, int nw, int lane) {
  for (int x = lane * W; x < n8; x += 32 * W) {
    const bool ok = x < n;
    const float* v = ok ? src + w * s_row + x * s_x : src;
    const int64_t step = ok ? nw * s_row : 0;
    uint32_t d = smem_u32(dst + w * pitch + x);
#pragma unroll 4
    for (int row = w; row < rows; row += nw, v += step, d += nw * pitch * 4) cp_async_floats<W>(d, v, ok);
  }
}
__device__ __forceinline__ void direct_load_rows(float* dst, int pitch, const float* src, int64_t s_row, int64_t s_x, int rows, int n, int n8,
                                                 int width, int w, int nw, int lane) {
  if (width == 4) {
    direct_load_rows<4>(dst, pitch, src, s_row, 1, rows, n, n8, w, nw, lane);
  } else if (width == 2) {
    direct_load_rows<2>(dst, pitch, src, s_row, 1, rows, n, n8, w, nw, lane);
  } else if (s_x == 1 || s_row != 1) {
    direct_load_rows<1>(dst, pitch, src, s_row, s_x, rows, n, n8, w, nw, lane);
  } else {  // consecutive rows: a transposed view
    for (int x = w; x < n8; x += nw) {
      const bool ok = x < n && lane < rows;
      cp_async_floats<1>(smem_u32(dst + lane * pitch + x), ok ? src + lane + x * s_x : src, ok);
    }
  }
}

// x = exp(x - m) in place for rows lo <= row < hi of x[n][32 columns], m the clamped maxima over all n rows (m_in: given by the
// caller); rows n .. hi and columns from cols on become exact zeros.  part: [8][32].  Returns the m of this lane's column.
// One or two block barriers.
__device__ __forceinline__ float direct_exp_columns(float* x, int n, int lo, int hi, int cols, const float* m_in, float* part, int warp,
                                                    int lane) {
  float mx = -INFINITY;
  if (m_in != nullptr) {
    if (lane < cols) mx = __ldg(m_in + lane);
  } else {
    if (lane < cols) {
#pragma unroll 4
      for (int row = warp; row < n; row += 8) mx = fmaxf(mx, x[row * DIRECT_PITCH + lane]);
    }
    part[warp * 32 + lane] = mx;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 8; ++w) mx = fmaxf(mx, part[w * 32 + lane]);
  }
  const float m = clamp_stab(mx);
#pragma unroll 4
  for (int row = lo + warp; row < hi; row += 8) {
    const bool ok = row < n && lane < cols;
    x[row * DIRECT_PITCH + lane] = exp_shifted(ok ? x[row * DIRECT_PITCH + lane] : -INFINITY, m);
  }
  __syncthreads();
  return m;
}

// d += a * b, one 16 x 8 x 8 product of tf32 operands (a: rows i, b: columns k).
__device__ __forceinline__ void mma_tf32_16x8x8(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t to_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}

// The same of a weight, which may be as large as a float: what rounding would make infinite becomes the largest tf32 value, while
// infinity and NaN stay.  (Low bits are left in place, the tensor core ignores them; a negative weight is truncated.)
__device__ __forceinline__ uint32_t to_tf32_weight(float x) {
  const uint32_t b = __float_as_uint(x);
  return max(__viaddmin_u32(b, 0x1000u, 0x7f7fffffu), b);
}

// acc (32 rows x 32 columns over the warp) += a[32 rows][8] * e[8][32 columns]; a, e at the first of the 8 contraction values.
// Lane 4 g + t holds rows g + 8 y and, of each group n of eight columns, columns 2 t and 2 t + 1; of e column g of each group.
// SCALED: column g of group n of e is multiplied with scale[n] first.
template <int PREC, bool SCALED = false>
__device__ __forceinline__ void direct_mma_step(float (&acc)[2][4][4], const float* a, int pitch, const float* e, int g, int t,
                                                const float* scale = nullptr) {
  uint32_t bh[4][2], bl[4][2];
#pragma unroll
  for (int n = 0; n < 4; ++n) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float v = e[(t + 4 * h) * DIRECT_PITCH + n * 8 + g];
      if (SCALED) v *= scale[n];
      if (PREC) {
        float hi, lo;
        tf32_split_rn(v, hi, lo);
        bh[n][h] = __float_as_uint(hi), bl[n][h] = __float_as_uint(lo);
      } else {
        bh[n][h] = to_tf32(v);
      }
    }
  }
#pragma unroll
  for (int y = 0; y < 2; ++y) {
    uint32_t ah[4], al[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const float v = a[(y * 16 + (x & 1) * 8 + g) * pitch + t + 4 * (x >> 1)];
      if (PREC) {
        float hi, lo;
        tf32_split_trunc(v, hi, lo);
        ah[x] = __float_as_uint(hi), al[x] = __float_as_uint(lo);
      } else {
        ah[x] = to_tf32_weight(v);
      }
    }
    if (PREC) {
#pragma unroll
      for (int n = 0; n < 4; ++n) mma_tf32_16x8x8(acc[y][n], ah, bl[n][0], bl[n][1]);
#pragma unroll
      for (int n = 0; n < 4; ++n) mma_tf32_16x8x8(acc[y][n], al, bh[n][0], bh[n][1]);
    }
#pragma unroll
    for (int n = 0; n < 4; ++n) mma_tf32_16x8x8(acc[y][n], ah, bh[n][0], bh[n][1]);
  }
}

// red[warp][row][column] = this warp's sums.
__device__ __forceinline__ void direct_store_partial(float* red, const float (&acc)[2][4][4], int warp, int g, int t) {
#pragma unroll
  for (int y = 0; y < 2; ++y) {
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      float* dst = red + (warp * 32 + y * 16 + g) * DIRECT_PITCH + n * 8 + 2 * t;
      *reinterpret_cast<float2*>(dst) = make_float2(acc[y][n][0], acc[y][n][1]);
      *reinterpret_cast<float2*>(dst + 8 * DIRECT_PITCH) = make_float2(acc[y][n][2], acc[y][n][3]);
    }
  }
}

// Folds the lanes' column maxima over the warps of the block into out_max (columns of this tile; starts at -inf).
__device__ __forceinline__ void direct_fold_max(float* out_max, float cmx, int cols, float* part, int warp, int lane) {
  part[warp * 32 + lane] = cmx;
  __syncthreads();
  if (warp == 0 && lane < cols) {
#pragma unroll
    for (int w = 1; w < 8; ++w) cmx = fmaxf(cmx, part[w * 32 + lane]);
    red_max_f32(out_max + lane, cmx);
  }
}

struct DirectLmParams {
  const float* a;  // [R, I, J]
  const float* b;  // [R, J, K]
  float* out;      // [R, I, K], consecutive k
  const float* m_in;  // [R, K] column maxima of b, or nullptr
  float* out_max;     // [R, K], pre-filled with -inf: receives max_i out[r,i,k], or nullptr
  int64_t a_s0, a_s1, a_s2, b_s0, b_s1, b_s2, out_s0, out_s1;
  int I, J, K;
  int width_a, width_b;  // floats per copy: 2 or 4 where values are consecutive, and base, row length and the other strides multiples of it
};

__host__ __device__ constexpr int direct_lm_smem(int J) {
  const int need = direct_round8(J) * DIRECT_PITCH + 32 * direct_pitch(J);
  return (need > DIRECT_RED_FLOATS ? need : DIRECT_RED_FLOATS) * 4;
}

// Grid: (K / 32, I / 32, R).
template <int PREC>
__global__ void __launch_bounds__(DIRECT_THREADS, 3) lm2exp_direct_kernel(const DirectLmParams p) {
  extern __shared__ float4 direct_smem[];
  __shared__ float part[8 * 32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int k0 = blockIdx.x * 32, i0 = blockIdx.y * 32, r = blockIdx.z;
  const int cols = min(32, p.K - k0), rows = min(32, p.I - i0);
  const int J8 = direct_round8(p.J), pitch = direct_pitch(p.J);
  float* e = reinterpret_cast<float*>(direct_smem);  // [J8][DIRECT_PITCH]
  float* a = e + J8 * DIRECT_PITCH;                  // [32][pitch]

  direct_load_columns(e, p.b + r * p.b_s0 + k0 * p.b_s2, p.b_s1, p.b_s2, p.J, cols, p.width_b, tid);
  cp_async_commit();
  direct_load_rows(a, pitch, p.a + r * p.a_s0 + i0 * p.a_s1, p.a_s1, p.a_s2, rows, p.J, J8, p.width_a, warp, 8, lane);
  cp_async_commit();
  cp_async_wait<1>();
  __syncthreads();
  const int64_t col0 = static_cast<int64_t>(r) * p.K + k0;
  const float m = direct_exp_columns(e, p.J, 0, J8, cols, p.m_in != nullptr ? p.m_in + col0 : nullptr, part, warp, lane);
  cp_async_wait<0>();
  __syncthreads();

  float acc[2][4][4] = {};
  const int g = lane >> 2, t = lane & 3;
  for (int s = warp; s < J8 / 8; s += 8) direct_mma_step<PREC>(acc, a + 8 * s, pitch, e + 8 * s * DIRECT_PITCH, g, t);
  __syncthreads();
  float* red = e;
  direct_store_partial(red, acc, warp, g, t);
  __syncthreads();
  float cmx = -INFINITY;
  if (lane < cols) {
    float* out = p.out + r * p.out_s0 + i0 * p.out_s1 + k0 + lane;
    for (int row = warp; row < rows; row += 8) {
      float sum = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) sum += red[(w * 32 + row) * DIRECT_PITCH + lane];
      const float o = m + logf(sum);
      out[row * p.out_s1] = o;
      cmx = fmaxf(cmx, o);
    }
  }
  if (p.out_max != nullptr) direct_fold_max(p.out_max + col0, cmx, cols, part, warp, lane);
}

struct DirectLtParams {
  const float* w;  // [R, S, I, J]
  const float* a;  // [R, I, K]
  const float* b;  // [R, J, K]
  float* out;      // [R, S, K], consecutive k
  const float *ma_in, *mb_in;  // [R, K] column maxima of a and b, or both nullptr
  float* out_max;              // [R, K], pre-filled with -inf: receives max_s out[r,s,k], or nullptr
  int64_t w_s0, w_s1, w_s2, w_s3, a_s0, a_s1, a_s2, b_s0, b_s1, b_s2, out_s0, out_s1;
  int S, I, J, K;
  int width_w, width_a, width_b;
  int parts;  // blocks of a cluster that share the rows i of a tile
  int nbuf;   // tiles of w per warp: two where some warp takes more than one i
};

__host__ __device__ constexpr int direct_lt_smem(int I, int J, int nbuf) {
  const int need = (direct_round8(J) + I) * DIRECT_PITCH + 8 * nbuf * 32 * direct_pitch(J);
  const int red = I * DIRECT_PITCH + DIRECT_RED_FLOATS;
  return (need > red ? need : red) * 4;
}

// lt2exp as sum_i (sum_j w[s, i, j] (exp(a_i - ma) exp(b_j - mb))): the inner sums on the tensor cores, the sum over i in
// fp32.  (exp(a_i - ma) as a factor of the inner sum instead of its terms would spare a product per term, but large
// weights overflow an inner sum that the factor, zero for an impossible state, takes back.)  A warp takes one i at a time and
// fetches its 32 rows of w itself, one i ahead.  The blocks of a cluster share the i of a tile; each adds up a part of the tile's rows through
// distributed shared memory, in rank order.  Grid: (parts * K / 32, S / 32, R), clusters of `parts`.
template <int PREC>
__global__ void __launch_bounds__(DIRECT_THREADS, 2) lt2exp_direct_kernel(const DirectLtParams p) {
  extern __shared__ float4 direct_smem[];
  __shared__ float part[8 * 32];
  __shared__ float tile[32 * 32];  // this block's sums
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = static_cast<int>(cluster_ctarank());
  const int k0 = (blockIdx.x / p.parts) * 32, s0 = blockIdx.y * 32, r = blockIdx.z;
  const int cols = min(32, p.K - k0), rows = min(32, p.S - s0);
  const int J8 = direct_round8(p.J), pitch = direct_pitch(p.J);
  float* ea = reinterpret_cast<float*>(direct_smem);  // [I][DIRECT_PITCH]
  float* eb = ea + p.I * DIRECT_PITCH;                // [J8][DIRECT_PITCH]
  float* wt = eb + J8 * DIRECT_PITCH + warp * p.nbuf * 32 * pitch;  // this warp's tiles [32][pitch] of w
  const int i_lo = p.I * rank / p.parts, i_hi = p.I * (rank + 1) / p.parts;
  const float* w = p.w + r * p.w_s0 + s0 * p.w_s1;

  direct_load_columns(ea, p.a + r * p.a_s0 + k0 * p.a_s2, p.a_s1, p.a_s2, p.I, cols, p.width_a, tid);
  direct_load_columns(eb, p.b + r * p.b_s0 + k0 * p.b_s2, p.b_s1, p.b_s2, p.J, cols, p.width_b, tid);
  cp_async_commit();
  auto fetch = [&](int i, int buf) {  // (a group is committed even when there is nothing left to fetch)
    if (i < i_hi)
      direct_load_rows(wt + buf * 32 * pitch, pitch, w + i * p.w_s2, p.w_s1, p.w_s3, rows, p.J, J8, p.width_w, 0, 1, lane);
    cp_async_commit();
  };
  fetch(i_lo + warp, 0);
  cp_async_wait<1>();
  __syncthreads();
  const int64_t col0 = static_cast<int64_t>(r) * p.K + k0;
  float m = direct_exp_columns(ea, p.I, i_lo, i_hi, cols, p.ma_in != nullptr ? p.ma_in + col0 : nullptr, part, warp, lane);
  m += direct_exp_columns(eb, p.J, 0, J8, cols, p.mb_in != nullptr ? p.mb_in + col0 : nullptr, part, warp, lane);

  float acc[2][4][4] = {};
  const int g = lane >> 2, t = lane & 3;
  int buf = 0;
  for (int i = i_lo + warp; i < i_hi; i += 8, buf ^= 1) {
    fetch(i + 8, buf ^ 1);
    cp_async_wait<1>();
    __syncwarp();
    float sum[2][4][4] = {}, scale[4];
#pragma unroll
    for (int n = 0; n < 4; ++n) scale[n] = ea[i * DIRECT_PITCH + n * 8 + g];
    const float* wb = wt + buf * 32 * pitch;
    for (int s = 0; s < J8 / 8; ++s) direct_mma_step<PREC, true>(sum, wb + 8 * s, pitch, eb + 8 * s * DIRECT_PITCH, g, t, scale);
#pragma unroll
    for (int y = 0; y < 2; ++y) {
#pragma unroll
      for (int n = 0; n < 4; ++n) {
#pragma unroll
        for (int x = 0; x < 4; ++x) acc[y][n][x] += sum[y][n][x];
      }
    }
    __syncwarp();  // every lane has read the buffer that the next fetch overwrites
  }
  cp_async_wait<0>();
  __syncthreads();
  float* red = eb;
  direct_store_partial(red, acc, warp, g, t);
  __syncthreads();
  for (int row = warp; row < 32; row += 8) {
    float sum = 0.f;
#pragma unroll
    for (int x = 0; x < 8; ++x) sum += red[(x * 32 + row) * DIRECT_PITCH + lane];
    tile[row * 32 + lane] = sum;
  }
  cluster_sync_all();
  float cmx = -INFINITY;
  for (int row = rank * 8 + warp; row < rows; row += p.parts * 8) {
    float sum = 0.f;
    for (int c = 0; c < p.parts; ++c) {
      float v;
      asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(map_to_cta(smem_u32(tile + row * 32 + lane), c)) : "memory");
      sum += v;
    }
    const float o = m + logf(sum);
    if (lane < cols) {
      p.out[r * p.out_s0 + (s0 + row) * p.out_s1 + k0 + lane] = o;
      cmx = fmaxf(cmx, o);
    }
  }
  if (p.out_max != nullptr) direct_fold_max(p.out_max + col0, cmx, cols, part, warp, lane);
  cluster_sync_all();  // a block's sums stay until every block has read them
}

}  // namespace tb200
