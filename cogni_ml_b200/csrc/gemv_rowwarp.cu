// General-shape GEMV for raw GGUF blocks: one warp per output row, lane l takes element l
// of every 32-wide group, fp32 FMA accumulation, warp-shuffle reduction.
//
// This kernel accepts every legal shape (any out_dim, any in_dim that is a block multiple,
// any batch, 2-byte aligned rows) and is the path for shapes the tiled tensor-core GEMV
// does not take (Q8_0 / IQ4_NL with 16-byte aligned activations: the block kernel further down).
// It also carries the fused lm_head variant: GEMV + per-part top-1 +
// last-CTA-done reduction, all in one launch.
//
// Weight value arithmetic follows src/ml/gguf/quant_matmul.cr (w = d*sc*q - dmin*m for
// Q4_K/Q5_K, w = d*sc*(q-32) for Q6_K, w = d*q for Q8_0) in fp32 instead of f64.
#include <climits>
#include <type_traits>

#include "qmm_common.cuh"

namespace cogni {

extern int g_force_rowwarp;  // dispatch.cu

namespace {

constexpr int kWarpsPerCta = 8;
constexpr int kTop1RowsPerPart = 64;  // rows whose best key one scratch slot holds

template <int NB>
__device__ __forceinline__ void fma_cols(float w, const float *x, int64_t xs, float (&acc)[NB]) {
#pragma unroll
  for (int c = 0; c < NB; c++) acc[c] = fmaf(w, x[c * xs], acc[c]);
}

template <int TYPE, int NB> struct BlockDot;

template <int NB> struct BlockDot<kQ8_0, NB> {
  static __device__ __forceinline__ void run(const uint8_t *b, const float *x, int64_t xs, int lane,
                                             float (&acc)[NB]) {
    float d = load_half_as_float(b);
    float w = d * (float)reinterpret_cast<const int8_t *>(b + 2)[lane];
    fma_cols<NB>(w, x + lane, xs, acc);
  }
};

template <int NB> struct BlockDot<kIQ4_NL, NB> {
  static __device__ __forceinline__ void run(const uint8_t *b, const float *x, int64_t xs, int lane,
                                             float (&acc)[NB]) {
    float d = load_half_as_float(b);
    int q = b[2 + (lane & 15)];
    float w = d * (float)iq4nl_value(lane < 16 ? (q & 0x0F) : (q >> 4));
    fma_cols<NB>(w, x + lane, xs, acc);
  }
};

template <int NB> struct BlockDot<kQ4_K, NB> {
  static __device__ __forceinline__ void run(const uint8_t *b, const float *x, int64_t xs, int lane,
                                             float (&acc)[NB]) {
    float d = load_half_as_float(b), dmin = load_half_as_float(b + 2);
    const uint8_t *scales = b + 4, *qs = b + 16;
#pragma unroll
    for (int pair = 0; pair < 4; pair++) {
      int sc, m, sc2, m2;
      scale_min_k4(2 * pair, scales, sc, m);
      scale_min_k4(2 * pair + 1, scales, sc2, m2);
      int q = qs[32 * pair + lane];
      float wlo = fmaf(d * (float)sc, (float)(q & 0x0F), -(dmin * (float)m));
      float whi = fmaf(d * (float)sc2, (float)(q >> 4), -(dmin * (float)m2));
      fma_cols<NB>(wlo, x + 64 * pair + lane, xs, acc);
      fma_cols<NB>(whi, x + 64 * pair + 32 + lane, xs, acc);
    }
  }
};

template <int NB> struct BlockDot<kQ5_K, NB> {
  static __device__ __forceinline__ void run(const uint8_t *b, const float *x, int64_t xs, int lane,
                                             float (&acc)[NB]) {
    float d = load_half_as_float(b), dmin = load_half_as_float(b + 2);
    const uint8_t *scales = b + 4, *qh = b + 16, *ql = b + 48;
    int h = qh[lane];
#pragma unroll
    for (int pair = 0; pair < 4; pair++) {
      int sc, m, sc2, m2;
      scale_min_k4(2 * pair, scales, sc, m);
      scale_min_k4(2 * pair + 1, scales, sc2, m2);
      int q = ql[32 * pair + lane];
      int qlo = (q & 0x0F) + (((h >> (2 * pair)) & 1) << 4);
      int qhi = (q >> 4) + (((h >> (2 * pair + 1)) & 1) << 4);
      float wlo = fmaf(d * (float)sc, (float)qlo, -(dmin * (float)m));
      float whi = fmaf(d * (float)sc2, (float)qhi, -(dmin * (float)m2));
      fma_cols<NB>(wlo, x + 64 * pair + lane, xs, acc);
      fma_cols<NB>(whi, x + 64 * pair + 32 + lane, xs, acc);
    }
  }
};

template <int NB> struct BlockDot<kQ6_K, NB> {
  static __device__ __forceinline__ void run(const uint8_t *b, const float *x, int64_t xs, int lane,
                                             float (&acc)[NB]) {
    const uint8_t *ql = b, *qh = b + 128;
    const int8_t *sc = reinterpret_cast<const int8_t *>(b + 192);
    float d = load_half_as_float(b + 208);
    int is = lane >> 4;
#pragma unroll
    for (int half = 0; half < 2; half++) {
      int l0 = ql[64 * half + lane], l1 = ql[64 * half + 32 + lane], h = qh[32 * half + lane];
      int q1 = ((l0 & 0xF) | (((h >> 0) & 3) << 4)) - 32;
      int q2 = ((l1 & 0xF) | (((h >> 2) & 3) << 4)) - 32;
      int q3 = ((l0 >> 4) | (((h >> 4) & 3) << 4)) - 32;
      int q4 = ((l1 >> 4) | (((h >> 6) & 3) << 4)) - 32;
      const int8_t *s = sc + 8 * half + is;
      const float *xx = x + 128 * half + lane;
      fma_cols<NB>(d * (float)s[0] * (float)q1, xx, xs, acc);
      fma_cols<NB>(d * (float)s[2] * (float)q2, xx + 32, xs, acc);
      fma_cols<NB>(d * (float)s[4] * (float)q3, xx + 64, xs, acc);
      fma_cols<NB>(d * (float)s[6] * (float)q4, xx + 96, xs, acc);
    }
  }
};

template <int NB>
__device__ __forceinline__ void warp_sum(float (&acc)[NB]) {
#pragma unroll
  for (int c = 0; c < NB; c++) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], off);
  }
}

// y[b, o] = addend + W[o,:] . x[b,:] for NB batch columns starting at b0 (columns past the
// batch are clamped onto the last valid one and not stored).
template <int TYPE, int NB>
__device__ __forceinline__ void row_dot(const uint8_t *wrow, const float *x, int in_dim, int batch,
                                        int b0, int lane, float (&acc)[NB]) {
  constexpr int BE = BlockGeom<TYPE>::elems, BB = BlockGeom<TYPE>::bytes;
#pragma unroll
  for (int c = 0; c < NB; c++) acc[c] = 0.f;
  // Column c reads x row min(b0+c, batch-1); with a uniform stride this needs b0+NB <= batch,
  // so the launcher picks NB dividing the work and the tail is handled by clamping b0.
  const float *xb = x + (int64_t)b0 * in_dim;
  const int nblk = in_dim / BE;
  for (int blk = 0; blk < nblk; blk++)
    BlockDot<TYPE, NB>::run(wrow + (int64_t)blk * BB, xb + (int64_t)blk * BE, in_dim, lane, acc);
  warp_sum<NB>(acc);
}

template <int TYPE, int NB>
__global__ void __launch_bounds__(kWarpsPerCta * 32)
    gemv_rowwarp_kernel(const uint8_t *__restrict__ w, const float *__restrict__ x,
                        const float *addend, int64_t addend_stride, float *y, int in_dim,
                        int out_dim, int batch) {
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * kWarpsPerCta + (threadIdx.x >> 5);
  if (row >= out_dim) return;
  const int64_t row_bytes = (int64_t)(in_dim / BlockGeom<TYPE>::elems) * BlockGeom<TYPE>::bytes;
  const uint8_t *wrow = w + (int64_t)row * row_bytes;
  for (int b0 = 0; b0 < batch; b0 += NB) {
    int bb = b0 + NB <= batch ? b0 : batch - NB;  // last group overlaps instead of overrunning
    float acc[NB];
    row_dot<TYPE, NB>(wrow, x, in_dim, batch, bb, lane, acc);
    if (lane == 0) {
#pragma unroll
      for (int c = 0; c < NB; c++) {
        int b = bb + c;
        if (b < b0) continue;  // already written by the previous group
        float a = addend ? addend[(int64_t)b * addend_stride + row] : 0.f;
        y[(int64_t)b * out_dim + row] = a + acc[c];
      }
    }
  }
}

// Q8_0 / IQ4_NL rows of any whole number of 32-element blocks (widths that no 256-element superblock
// divides; in f32 throughout).  A row of such a matrix is a few kilobytes, so what bounds the
// row-per-warp kernel above is latency: one block after the other, two bytes a load.  Here a warp
// takes eight blocks of RPW rows at a time, four lanes per block and eight weights per lane; the
// activations are read as 16-byte vectors once for the RPW rows, and `wk` of a CTA's eight warps split
// K (partial sums meet in shared memory and are added in warp order: the same bits every time).  The
// columns of one row group are neighbouring CTAs, so the weights come from DRAM once.  Measured against
// the row-per-warp kernel (us): IQ4_NL 2053 x 2976 batch 1 / 3 / 16 14.1 -> 5.5 / 21.9 -> 6.4 / 102 ->
// 20, Q8_0 100 x 10016 batch 8 148 -> 6.2, Q8_0 20000 x 10016 batch 1 / 8 147 -> 68 (3.1 TB/s) / 855 ->
// 221 (then bound by its f32 arithmetic, 7 instructions per weight beside the multiply-adds).
constexpr int kBlockWarps = 8;
template <int TYPE>
__device__ __forceinline__ void load_quants(const uint8_t *blk, int p, uint32_t (&q)[2], float &d) {
  // 2-byte aligned addresses.  Elements 4p .. 4p+3 and 16+4p .. 16+4p+3 of the block.
  auto word = [](const uint8_t *a) {
    const unsigned short *h = reinterpret_cast<const unsigned short *>(a);
    return (uint32_t)__ldg(h) | (uint32_t)__ldg(h + 1) << 16;
  };
  d = __half2float(__ushort_as_half(__ldg(reinterpret_cast<const unsigned short *>(blk))));
  q[0] = word(blk + 2 + 4 * p);
  q[1] = TYPE == kQ8_0 ? word(blk + 18 + 4 * p) : 0u;
}
// the eight weights d * q, elements 4p .. 4p+3, then 16+4p .. 16+4p+3
template <int TYPE>
__device__ __forceinline__ void block_weights(const uint32_t (&q)[2], float d, float (&v)[8]) {
  uint32_t b[2];  // signed bytes
  if constexpr (TYPE == kQ8_0) {
    b[0] = q[0];
    b[1] = q[1];
  } else {
    auto lut4 = [](uint32_t h) {  // nibbles 0 .. 3 of h -> the four table values as bytes
      const uint32_t s7 = h & 0x7777u;
      const uint32_t lo = __byte_perm(0xBFAD9881u, 0xF6EADDCFu, s7);  // entries 0 .. 7
      const uint32_t hi = __byte_perm(0x26190D01u, 0x71594535u, s7);  // entries 8 .. 15
      return __byte_perm(lo, hi, 0x3210u | ((h >> 1) & 0x4444u));
    };
    const uint32_t e = lut4(q[0]), o = lut4(q[0] >> 16);  // (low, high) nibble pairs of bytes 0, 1 | 2, 3
    b[0] = __byte_perm(e, o, 0x6420);
    b[1] = __byte_perm(e, o, 0x7531);
  }
#pragma unroll
  for (int i = 0; i < 8; i++)  // the float is 2^23 + 128 + b, exactly
    v[i] = d * (__uint_as_float(__byte_perm(b[i >> 2] ^ 0x80808080u, 0x4B000000u, 0x7650 + (i & 3))) - 8388736.f);
}

// TAIL: the batch is no multiple of NB, so the last column group computes some columns of the one before
// again.  The addend may be y itself, so every output is stored by one CTA, that of the group which owns the
// column.  (An instance of its own: the condition moves the compiler to schedules that cost up to 25 % where
// it is not needed, Q8_0 16 x 33024 at batch 2 8.8 -> 11.1 us.)
template <int TYPE, int NB, int RPW, bool TAIL>
__global__ void __launch_bounds__(kBlockWarps * 32)
    gemv_blocks_kernel(const uint8_t *__restrict__ w, const float *__restrict__ x, const float *addend,
                       int64_t addend_stride, float *y, int in_dim, int out_dim, int batch, int bgroups,
                       int wk) {
  constexpr int BB = BlockGeom<TYPE>::bytes;
  constexpr int NP = NB == 3 ? 4 : NB > 4 ? 8 : NB, N = RPW * NP;  // sums of a warp, columns padded to a power of two
  __shared__ float s_part[kBlockWarps][N];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, p = lane & 3;
  const int nblk = in_dim >> 5;
  const int kw = warp & (wk - 1), grp = warp / wk;  // this warp's part of K, its row group of the CTA
  const int row0 = ((int)(blockIdx.x / bgroups) * (kBlockWarps / wk) + grp) * RPW;
  const int b0 = min((int)(blockIdx.x % bgroups) * NB, batch - NB);  // the last group overlaps the one before
  const long long row_bytes = (long long)nblk * BB;
  const uint8_t *wr[RPW];
#pragma unroll
  for (int r = 0; r < RPW; r++) wr[r] = w + (long long)min(row0 + r, out_dim - 1) * row_bytes;
  const float *xb = x + (long long)b0 * in_dim + 4 * p;
  float acc[N];
#pragma unroll
  for (int i = 0; i < N; i++) acc[i] = 0.f;
  for (int blk = 8 * kw + (lane >> 2); blk < nblk; blk += 8 * wk) {
    uint32_t q[RPW][2];
    float d[RPW];
#pragma unroll
    for (int r = 0; r < RPW; r++) load_quants<TYPE>(wr[r] + (long long)blk * BB, p, q[r], d[r]);
    float v[RPW][8];
#pragma unroll
    for (int r = 0; r < RPW; r++) block_weights<TYPE>(q[r], d[r], v[r]);
#pragma unroll
    for (int c = 0; c < NB; c++) {
      const float4 *xp = reinterpret_cast<const float4 *>(xb + (long long)c * in_dim + 32 * blk);
      const float4 xl = __ldg(xp), xh = __ldg(xp + 4);
#pragma unroll
      for (int r = 0; r < RPW; r++) {
        float s = fmaf(v[r][0], xl.x, acc[r * NP + c]);
        s = fmaf(v[r][1], xl.y, s);
        s = fmaf(v[r][2], xl.z, s);
        s = fmaf(v[r][3], xl.w, s);
        s = fmaf(v[r][4], xh.x, s);
        s = fmaf(v[r][5], xh.y, s);
        s = fmaf(v[r][6], xh.z, s);
        acc[r * NP + c] = fmaf(v[r][7], xh.w, s);
      }
    }
  }
  // sum over the lanes: while there are several sums, half of the lanes keep one half of them
  int n = N, off = 16;
#pragma unroll
  for (int step = 0; step < 5; step++) {
    if (n > 1) {
      n >>= 1;
      const bool up = (lane & off) != 0;
#pragma unroll
      for (int i = 0; i < N / 2; i++)
        if (i < n) {
          const float keep = up ? acc[i + n] : acc[i], give = up ? acc[i] : acc[i + n];
          acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, off);
        }
    } else {
      acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], off);
    }
    off >>= 1;
  }
  constexpr int kLanesPerSum = 32 / N;  // sum i sits in lanes i * kLanesPerSum ..
  if (lane % kLanesPerSum == 0) s_part[warp][lane / kLanesPerSum] = acc[0];
  __syncthreads();
  if (threadIdx.x < N * kBlockWarps && threadIdx.x / N < kBlockWarps / wk) {
    const int g = threadIdx.x / N, i = threadIdx.x % N, r = i / NP, c = i % NP;
    const int row = ((int)(blockIdx.x / bgroups) * (kBlockWarps / wk) + g) * RPW + r;
    float sum = 0.f;
    for (int k = 0; k < wk; k++) sum += s_part[g * wk + k][i];
    const int b = b0 + c;
    if (c < NB && (!TAIL || b >= (int)(blockIdx.x % bgroups) * NB) && row < out_dim) {
      const float a = addend ? addend[(int64_t)b * addend_stride + row] : 0.f;
      y[(int64_t)b * out_dim + row] = a + sum;
    }
  }
}

// Fused lm_head: each CTA owns kTop1RowsPerPart consecutive rows of one batch row's logits,
// keeps the best (value, index) key, stores it in its scratch slot; the CTA that takes the
// last ticket of a batch row folds all slots and writes the result.
template <int TYPE>
__global__ void __launch_bounds__(kWarpsPerCta * 32)
    gemv_top1_rowwarp_kernel(const uint8_t *__restrict__ w, const float *__restrict__ x,
                             int in_dim, int out_dim, int32_t index_base, unsigned *counters,
                             long long *part_keys, int nparts, int32_t *top_idx, float *top_val,
                             long long *top_key) {
  __shared__ long long s_best[kWarpsPerCta];
  __shared__ bool s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int b = blockIdx.y, part = blockIdx.x;
  const int64_t row_bytes = (int64_t)(in_dim / BlockGeom<TYPE>::elems) * BlockGeom<TYPE>::bytes;
  long long best = LLONG_MIN;
  const int row_end = min(out_dim, (part + 1) * kTop1RowsPerPart);
  for (int row = part * kTop1RowsPerPart + warp; row < row_end; row += kWarpsPerCta) {
    float acc[1];
    row_dot<TYPE, 1>(w + (int64_t)row * row_bytes, x, in_dim, gridDim.y, b, lane, acc);
    long long key = top1_key(acc[0], (uint32_t)(index_base + row));
    best = key > best ? key : best;
  }
  if (lane == 0) s_best[warp] = best;
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int i = 1; i < kWarpsPerCta; i++) best = s_best[i] > best ? s_best[i] : best;
    part_keys[(int64_t)b * nparts + part] = best;
    __threadfence();
    unsigned ticket = atomicAdd(&counters[b], 1u);
    s_last = (ticket == (unsigned)nparts - 1u);
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  best = LLONG_MIN;
  for (int i = threadIdx.x; i < nparts; i += blockDim.x) {
    long long k = __ldcg(&part_keys[(int64_t)b * nparts + i]);
    best = k > best ? k : best;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    long long o = __shfl_xor_sync(0xffffffffu, best, off);
    best = o > best ? o : best;
  }
  __syncthreads();
  if (lane == 0) s_best[warp] = best;
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int i = 1; i < kWarpsPerCta; i++) best = s_best[i] > best ? s_best[i] : best;
    float v;
    uint32_t idx;
    top1_unkey(best, v, idx);
    top_idx[b] = (int32_t)idx;
    top_val[b] = v;
    if (top_key) top_key[b] = best;
    counters[b] = 0u;  // ready for the next call on this scratch buffer
  }
}

// Four rows a warp share the activations' loads; matrices of few rows take one row a warp, so that
// two CTAs per SM remain.  Short rows are split over fewer warps: a part has at least one step of
// eight blocks, two where the matrix has rows enough to fill the SMs.
template <int TYPE, int NB, int RPW>
int run_blocks_rows(const void *d_w, const float *d_x, const float *d_addend, int64_t addend_stride, float *d_y,
                    int in_dim, int out_dim, int batch, int bgroups, cudaStream_t s) {
  const int groups = (out_dim + RPW - 1) / RPW, steps = (in_dim / 32 + 7) / 8;
  int wk = kBlockWarps;
  while (wk > 1 && (wk / 2 >= steps ||
                    (wk >= steps && (long long)groups * bgroups * wk / 2 >= 148LL * 4 * kBlockWarps)))
    wk /= 2;
  const int per_cta = kBlockWarps / wk;
  const unsigned ctas = (unsigned)((groups + per_cta - 1) / per_cta) * (unsigned)bgroups;
  auto launch = [&](auto tail) {
    gemv_blocks_kernel<TYPE, NB, RPW, decltype(tail)::value><<<ctas, kBlockWarps * 32, 0, s>>>(
        static_cast<const uint8_t *>(d_w), d_x, d_addend, addend_stride, d_y, in_dim, out_dim, batch, bgroups, wk);
  };
  if (NB > 2 && batch % NB != 0) launch(std::integral_constant<bool, (NB > 2)>{});  // one or two columns are one group
  else launch(std::false_type{});
  return (int)cudaGetLastError();
}
template <int TYPE, int NB>
int run_blocks(const void *d_w, const float *d_x, const float *d_addend, int64_t addend_stride, float *d_y,
               int in_dim, int out_dim, int batch, int bgroups, cudaStream_t s) {
  if (NB > 4 || (long long)((out_dim + 3) / 4) * bgroups >= 2 * 148)
    return run_blocks_rows<TYPE, NB, 4>(d_w, d_x, d_addend, addend_stride, d_y, in_dim, out_dim, batch, bgroups, s);
  return run_blocks_rows<TYPE, (NB > 4 ? 4 : NB), (NB > 4 ? 4 : 1)>(d_w, d_x, d_addend, addend_stride, d_y, in_dim, out_dim, batch, bgroups, s);
}

// Rows of so few blocks that the block kernel's reductions across lanes and warps cost more than the
// row-per-warp kernel's passes over them (of four columns, or two).  Measured, us, row-per-warp / block:
// Q8_0 600 x 192 at batch 1 2.11 / 2.24, 600 x 224 2.41 / 2.25; at batch 2 Q8_0 100 x 96 2.01 / 2.41, 100 x 128
// 2.23 / 2.28, IQ4_NL 100 x 128 1.95 / 2.54; Q8_0 100 x 96 at batch 4 2.19 / 2.53, 100 x 128 2.68 / 2.66; 600 x 32
// at batch 5 2.42 / 2.70.  On many rows the weights' bytes decide, and the block kernel's wider loads: IQ4_NL
// 20000 x 32 at batch 1 3.73 / 4.52, 20000 x 96 4.98 / 4.65.
bool short_rows(int type, int blocks, int out_dim, int batch) {
  if (out_dim > (batch <= 2 || batch == 4 ? 5000 : 2500)) return batch <= 2 && blocks == 1;
  if (batch <= 2) return blocks <= (type == kQ8_0 && batch == 2 ? 3 : 6);
  return batch <= 8 && blocks * (batch == 4 ? 1 : 2) <= 3;
}

template <int TYPE>
int run_gemv(const void *d_w, const float *d_x, const float *d_addend, int64_t addend_stride,
             float *d_y, int in_dim, int out_dim, int batch, cudaStream_t s) {
  const uint8_t *w = static_cast<const uint8_t *>(d_w);
  if constexpr (TYPE == kQ8_0 || TYPE == kIQ4_NL) {
    // Up to four columns a CTA; on many rows the unpacked weights serve up to eight (Q8_0: six, its
    // weights take more registers until they are unpacked; 20000 x 10016 at batch 5 / 8: 166 -> 143 /
    // 221 -> 259 us with one group of 5 / 8 against 3 + 3 / 4 + 4, IQ4_NL 196 -> 165 / 219 -> 191).
    const int most = batch > 4 && out_dim >= 4 * 148 * 8 ? (TYPE == kIQ4_NL ? 8 : 6) : 4;
    const int bg = (batch + most - 1) / most, nb = (batch + bg - 1) / bg;  // 5 rows: 3 + 3, 9: 3 + 3 + 3
    // 16-byte loads of x: rows are whole 128-byte blocks, so its base decides
    if (g_force_rowwarp == 0 && !short_rows(TYPE, in_dim / 32, out_dim, batch) &&
        (reinterpret_cast<uintptr_t>(d_x) & 15) == 0 && (long long)out_dim * bg <= 0x7fffffffLL) {
      if (nb == 1) return run_blocks<TYPE, 1>(d_w, d_x, d_addend, addend_stride, d_y, in_dim, out_dim, batch, bg, s);
      if (nb == 2) return run_blocks<TYPE, 2>(d_w, d_x, d_addend, addend_stride, d_y, in_dim, out_dim, batch, bg, s);
      if (nb == 3) return run_blocks<TYPE, 3>(d_w, d_x, d_addend, addend_stride, d_y, in_dim, out_dim, batch, bg, s);
      if (nb == 4) return run_blocks<TYPE, 4>(d_w, d_x, d_addend, addend_stride, d_y, in_dim, out_dim, batch, bg, s);
      if (nb == 5) return run_blocks<TYPE, 5>(d_w, d_x, d_addend, addend_stride, d_y, in_dim, out_dim, batch, bg, s);
      if (nb == 6) return run_blocks<TYPE, 6>(d_w, d_x, d_addend, addend_stride, d_y, in_dim, out_dim, batch, bg, s);
      if (nb == 7) return run_blocks<TYPE, 7>(d_w, d_x, d_addend, addend_stride, d_y, in_dim, out_dim, batch, bg, s);
      return run_blocks<TYPE, 8>(d_w, d_x, d_addend, addend_stride, d_y, in_dim, out_dim, batch, bg, s);
    }
  }
  dim3 grid((out_dim + kWarpsPerCta - 1) / kWarpsPerCta), block(kWarpsPerCta * 32);
  if (batch >= 4)
    gemv_rowwarp_kernel<TYPE, 4><<<grid, block, 0, s>>>(w, d_x, d_addend, addend_stride, d_y,
                                                        in_dim, out_dim, batch);
  else if (batch >= 2)
    gemv_rowwarp_kernel<TYPE, 2><<<grid, block, 0, s>>>(w, d_x, d_addend, addend_stride, d_y,
                                                        in_dim, out_dim, batch);
  else
    gemv_rowwarp_kernel<TYPE, 1><<<grid, block, 0, s>>>(w, d_x, d_addend, addend_stride, d_y,
                                                        in_dim, out_dim, batch);
  return (int)cudaGetLastError();
}

template <int TYPE>
int run_top1(const void *d_w, const float *d_x, int in_dim, int out_dim, int batch,
             int32_t index_base, void *d_scratch, int32_t *d_idx, float *d_val, long long *d_key,
             cudaStream_t s) {
  int nparts = (out_dim + kTop1RowsPerPart - 1) / kTop1RowsPerPart;
  unsigned *counters = static_cast<unsigned *>(d_scratch);
  long long *keys = reinterpret_cast<long long *>(static_cast<char *>(d_scratch) +
                                                  (((size_t)batch * 4 + 7) & ~(size_t)7));
  // A call of a smaller batch, or of the tiled kernel (one counter), on the same scratch buffer has its
  // part keys where this one's counters lie.
  const cudaError_t e = cudaMemsetAsync(counters, 0, (size_t)batch * sizeof(unsigned), s);
  if (e != cudaSuccess) return (int)e;
  dim3 grid(nparts, batch), block(kWarpsPerCta * 32);
  gemv_top1_rowwarp_kernel<TYPE><<<grid, block, 0, s>>>(static_cast<const uint8_t *>(d_w), d_x,
                                                         in_dim, out_dim, index_base, counters,
                                                         keys, nparts, d_idx, d_val, d_key);
  return (int)cudaGetLastError();
}

}  // namespace

size_t top1_scratch_bytes(int out_dim, int batch) {
  // one slot per 64 rows, and never fewer than 256 so a one-CTA-per-SM kernel always has a slot
  size_t nparts = ((size_t)out_dim + kTop1RowsPerPart - 1) / kTop1RowsPerPart;
  if (nparts < 256) nparts = 256;
  return (((size_t)batch * 4 + 7) & ~(size_t)7) + (size_t)batch * nparts * 8;
}

int launch_gemv_rowwarp(int type, const void *d_w, const float *d_x, const float *d_addend,
                        int64_t addend_stride, float *d_y, int in_dim, int out_dim, int batch,
                        cudaStream_t s) {
  switch (type) {
    case kQ8_0: return run_gemv<kQ8_0>(d_w, d_x, d_addend, addend_stride, d_y, in_dim, out_dim, batch, s);
    case kIQ4_NL: return run_gemv<kIQ4_NL>(d_w, d_x, d_addend, addend_stride, d_y, in_dim, out_dim, batch, s);
    case kQ4_K: return run_gemv<kQ4_K>(d_w, d_x, d_addend, addend_stride, d_y, in_dim, out_dim, batch, s);
    case kQ5_K: return run_gemv<kQ5_K>(d_w, d_x, d_addend, addend_stride, d_y, in_dim, out_dim, batch, s);
    case kQ6_K: return run_gemv<kQ6_K>(d_w, d_x, d_addend, addend_stride, d_y, in_dim, out_dim, batch, s);
    default: return COGNI_QMM_ERR_TYPE;
  }
}

int launch_gemv_top1_rowwarp(int type, const void *d_w, const float *d_x, int in_dim, int out_dim,
                             int batch, int32_t index_base, void *d_scratch, int32_t *d_idx,
                             float *d_val, long long *d_key, cudaStream_t s) {
  switch (type) {
    case kQ8_0: return run_top1<kQ8_0>(d_w, d_x, in_dim, out_dim, batch, index_base, d_scratch, d_idx, d_val, d_key, s);
    case kIQ4_NL: return run_top1<kIQ4_NL>(d_w, d_x, in_dim, out_dim, batch, index_base, d_scratch, d_idx, d_val, d_key, s);
    case kQ4_K: return run_top1<kQ4_K>(d_w, d_x, in_dim, out_dim, batch, index_base, d_scratch, d_idx, d_val, d_key, s);
    case kQ5_K: return run_top1<kQ5_K>(d_w, d_x, in_dim, out_dim, batch, index_base, d_scratch, d_idx, d_val, d_key, s);
    case kQ6_K: return run_top1<kQ6_K>(d_w, d_x, in_dim, out_dim, batch, index_base, d_scratch, d_idx, d_val, d_key, s);
    default: return COGNI_QMM_ERR_TYPE;
  }
}

}  // namespace cogni
