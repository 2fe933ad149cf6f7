// Bulk dequantisation of raw GGUF blocks to f32 on the device.
//
// Bit-exact against the reference's CPU dequantiser (src/ml/gguf/dequant.cr): the same f32
// operations in the same order, written with the explicit round-to-nearest intrinsics so
// the compiler cannot contract a multiply and a subtract into one fused operation:
//   Q4_K/Q5_K  d1 = d*sc; m1 = dmin*m; w = d1*q - m1     (dequant.cr:120-133, 168-185)
//   Q6_K       w = (d*sc)*q                              (dequant.cr:224-227)
//   Q8_0       w = d*q                                   (dequant.cr:66-68)
//   IQ4_NL     w = d*table[nibble]                       (dequant.cr:76-101)
// HBM-bound: 4 B written per element against 0.56-1.06 B read.
#include "qmm_common.cuh"

namespace cogni {
namespace {

template <int TYPE>
__device__ __forceinline__ void expand_block(const uint8_t *b, float *y, int lane);

template <>
__device__ __forceinline__ void expand_block<kQ8_0>(const uint8_t *b, float *y, int lane) {
  float d = load_half_as_float(b);
  int q = reinterpret_cast<const int8_t *>(b + 2)[lane];
  y[lane] = __fmul_rn(d, (float)q);
}

template <>
__device__ __forceinline__ void expand_block<kIQ4_NL>(const uint8_t *b, float *y, int lane) {
  float d = load_half_as_float(b);
  int q = b[2 + (lane & 15)];
  y[lane] = __fmul_rn(d, (float)iq4nl_value(lane < 16 ? (q & 0x0F) : (q >> 4)));
}

template <>
__device__ __forceinline__ void expand_block<kQ4_K>(const uint8_t *b, float *y, int lane) {
  float d = load_half_as_float(b), dmin = load_half_as_float(b + 2);
  const uint8_t *scales = b + 4, *qs = b + 16;
#pragma unroll
  for (int pair = 0; pair < 4; pair++) {
    int sc, m, sc2, m2;
    scale_min_k4(2 * pair, scales, sc, m);
    scale_min_k4(2 * pair + 1, scales, sc2, m2);
    float d1 = __fmul_rn(d, (float)sc), m1 = __fmul_rn(dmin, (float)m);
    float d2 = __fmul_rn(d, (float)sc2), m2f = __fmul_rn(dmin, (float)m2);
    int q = qs[32 * pair + lane];
    y[64 * pair + lane] = __fsub_rn(__fmul_rn(d1, (float)(q & 0x0F)), m1);
    y[64 * pair + 32 + lane] = __fsub_rn(__fmul_rn(d2, (float)(q >> 4)), m2f);
  }
}

template <>
__device__ __forceinline__ void expand_block<kQ5_K>(const uint8_t *b, float *y, int lane) {
  float d = load_half_as_float(b), dmin = load_half_as_float(b + 2);
  const uint8_t *scales = b + 4, *qh = b + 16, *ql = b + 48;
  int h = qh[lane];
#pragma unroll
  for (int pair = 0; pair < 4; pair++) {
    int sc, m, sc2, m2;
    scale_min_k4(2 * pair, scales, sc, m);
    scale_min_k4(2 * pair + 1, scales, sc2, m2);
    float d1 = __fmul_rn(d, (float)sc), m1 = __fmul_rn(dmin, (float)m);
    float d2 = __fmul_rn(d, (float)sc2), m2f = __fmul_rn(dmin, (float)m2);
    int q = ql[32 * pair + lane];
    int qlo = (q & 0x0F) + (((h >> (2 * pair)) & 1) << 4);
    int qhi = (q >> 4) + (((h >> (2 * pair + 1)) & 1) << 4);
    y[64 * pair + lane] = __fsub_rn(__fmul_rn(d1, (float)qlo), m1);
    y[64 * pair + 32 + lane] = __fsub_rn(__fmul_rn(d2, (float)qhi), m2f);
  }
}

template <>
__device__ __forceinline__ void expand_block<kQ6_K>(const uint8_t *b, float *y, int lane) {
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
    float *yy = y + 128 * half + lane;
    yy[0] = __fmul_rn(__fmul_rn(d, (float)s[0]), (float)q1);
    yy[32] = __fmul_rn(__fmul_rn(d, (float)s[2]), (float)q2);
    yy[64] = __fmul_rn(__fmul_rn(d, (float)s[4]), (float)q3);
    yy[96] = __fmul_rn(__fmul_rn(d, (float)s[6]), (float)q4);
  }
}

// Any 2-byte aligned weights, any 4-byte aligned output, and small tensors: one warp per block, lane l
// writes element l of every 32-wide group.
template <int TYPE>
__global__ void __launch_bounds__(256) dequantize_blocks_kernel(const uint8_t *__restrict__ w,
                                                                float *__restrict__ out,
                                                                long long nblocks) {
  const int lane = threadIdx.x & 31;
  long long warp = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const long long nwarps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long blk = warp; blk < nblocks; blk += nwarps)
    expand_block<TYPE>(w + blk * BlockGeom<TYPE>::bytes, out + blk * BlockGeom<TYPE>::elems, lane);
}

// 16-byte aligned weights and output.  A thread takes the quant words that lie at one four-element
// position of a block and writes everything they hold as 16-byte stores: per word the low and the
// high nibbles, for Q5_K / Q6_K all groups that share its qh word.  LANES threads cover a block, a
// store instruction writes whole 64- or 128-byte runs, and a thread's loads are all independent.
// 4096 x 4096 in us, before (a 4-byte store per element) -> now, GB/s: Q4_K 16.4 -> 12.3 (6240), Q5_K
// 17.8 -> 13.0 (6060), Q6_K 15.7 -> 14.4 (5640), Q8_0 23.2 -> 17.1 (4980), IQ4_NL 28.0 -> 14.4 (5340).
template <int TYPE> constexpr int kQuadLanes = TYPE == kQ6_K ? 16 : TYPE == kIQ4_NL ? 4 : 8;

// four consecutive bytes at a 2-byte aligned address
__device__ __forceinline__ uint32_t ldg_word2(const uint8_t *p) {
  const unsigned short *h = reinterpret_cast<const unsigned short *>(p);
  return (uint32_t)__ldg(h) | (uint32_t)__ldg(h + 1) << 16;
}
__device__ __forceinline__ uint32_t ldg_word4(const uint8_t *p) { return __ldg(reinterpret_cast<const uint32_t *>(p)); }
__device__ __forceinline__ float ldg_half(const uint8_t *p) {
  return __half2float(__ushort_as_half(__ldg(reinterpret_cast<const unsigned short *>(p))));
}
__device__ __forceinline__ void put4(float *y, float a, float b, float c, float d) {
  *reinterpret_cast<float4 *>(y) = make_float4(a, b, c, d);
}

template <int TYPE>
__device__ __forceinline__ void expand_quads(const uint8_t *b, float *y, int i) {
  if constexpr (TYPE == kQ8_0) {
    const uint32_t q = ldg_word2(b + 2 + 4 * i);
    const float d = ldg_half(b);
    put4(y + 4 * i, __fmul_rn(d, (float)(int8_t)q), __fmul_rn(d, (float)(int8_t)(q >> 8)),
         __fmul_rn(d, (float)(int8_t)(q >> 16)), __fmul_rn(d, (float)(int8_t)(q >> 24)));
  } else if constexpr (TYPE == kIQ4_NL) {
    const uint32_t q = ldg_word2(b + 2 + 4 * i);
    const float d = ldg_half(b);
    float v[8];
#pragma unroll
    for (int e = 0; e < 8; e++) v[e] = __fmul_rn(d, (float)iq4nl_value((q >> (4 * e)) & 15));
    put4(y + 4 * i, v[0], v[2], v[4], v[6]);
    put4(y + 16 + 4 * i, v[1], v[3], v[5], v[7]);
  } else if constexpr (TYPE == kQ6_K) {
    const int half = i >> 3, l = 4 * (i & 7);
    const uint32_t q0 = ldg_word2(b + 64 * half + l), q1 = ldg_word2(b + 64 * half + 32 + l);
    const uint32_t h = ldg_word2(b + 128 + 32 * half + l);
    const uint8_t *s = b + 192 + 8 * half + (l >> 4);
    const float d = ldg_half(b + 208);
    float *yy = y + 128 * half + l;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint32_t lo = ((k & 1 ? q1 : q0) >> (k & 2 ? 4 : 0)) & 0x0f0f0f0fu;
      const uint32_t q = lo | ((h >> (2 * k)) & 0x03030303u) << 4;
      const float ds = __fmul_rn(d, (float)(int8_t)__ldg(s + 2 * k));
      put4(yy + 32 * k, __fmul_rn(ds, (float)((int)(q & 255) - 32)), __fmul_rn(ds, (float)((int)(q >> 8 & 255) - 32)),
           __fmul_rn(ds, (float)((int)(q >> 16 & 255) - 32)), __fmul_rn(ds, (float)((int)(q >> 24) - 32)));
    }
  } else {
    constexpr int QS = TYPE == kQ5_K ? 48 : 16;
    const uint4 hdr = __ldg(reinterpret_cast<const uint4 *>(b));
    uint32_t qs[4], h = 0;
#pragma unroll
    for (int p = 0; p < 4; p++) qs[p] = ldg_word4(b + QS + 32 * p + 4 * i);
    if (TYPE == kQ5_K) h = ldg_word4(b + 16 + 4 * i);
    const __half2 dd = *reinterpret_cast<const __half2 *>(&hdr.x);
    const float d = __low2float(dd), dmin = __high2float(dd);
    // the eight 6-bit scales / mins as bytes (dequant.cr:240-249, four at a time)
    const uint32_t sc[2] = {hdr.y & 0x3f3f3f3fu, (hdr.w & 0x0f0f0f0fu) | ((hdr.y >> 2) & 0x30303030u)};
    const uint32_t mn[2] = {hdr.z & 0x3f3f3f3fu, ((hdr.w >> 4) & 0x0f0f0f0fu) | ((hdr.z >> 2) & 0x30303030u)};
#pragma unroll
    for (int g = 0; g < 8; g++) {
      const float dg = __fmul_rn(d, (float)(sc[g >> 2] >> (8 * (g & 3)) & 255u));
      const float mg = __fmul_rn(dmin, (float)(mn[g >> 2] >> (8 * (g & 3)) & 255u));
      uint32_t q = (qs[g >> 1] >> (4 * (g & 1))) & 0x0f0f0f0fu;
      if (TYPE == kQ5_K) q |= ((h >> g) & 0x01010101u) << 4;
      put4(y + 32 * g + 4 * i, __fsub_rn(__fmul_rn(dg, (float)(q & 255u)), mg),
           __fsub_rn(__fmul_rn(dg, (float)(q >> 8 & 255u)), mg), __fsub_rn(__fmul_rn(dg, (float)(q >> 16 & 255u)), mg),
           __fsub_rn(__fmul_rn(dg, (float)(q >> 24)), mg));
    }
  }
}

// UNROLL blocks of a thread are a CTA's LANES-wide strides apart; their loads go out together.
template <int TYPE> constexpr int kQuadUnroll = TYPE == kQ8_0 ? 4 : 2;
template <int TYPE>
__global__ void __launch_bounds__(256) dequantize_quads_kernel(const uint8_t *__restrict__ w, float *__restrict__ out,
                                                               long long nblocks) {
  constexpr int L = kQuadLanes<TYPE>, PER = 256 / L, U = kQuadUnroll<TYPE>;
  const int i = threadIdx.x % L;
  const long long blk0 = (long long)blockIdx.x * PER * U + threadIdx.x / L;
#pragma unroll
  for (int u = 0; u < U; u++) {
    const long long blk = blk0 + u * PER;
    if (blk < nblocks)
      expand_quads<TYPE>(w + blk * BlockGeom<TYPE>::bytes, out + blk * BlockGeom<TYPE>::elems, i);
  }
}

// Token-embedding gather: out[t, :] = dequant(row token_ids[t] of the table), the same block
// expansion as the bulk dequantiser (bit-exact against Dequant.dequantize of that row,
// src/ml/gguf/qwen35_cpu.cr:3305-3332).  One warp per block of a token's row.  An id outside
// [0, vocab) yields a row of zeros and raises *status to 1 + the index of such a token.
template <int TYPE>
__global__ void __launch_bounds__(256) embedding_rows_kernel(const uint8_t *__restrict__ table,
                                                             const int32_t *__restrict__ token_ids,
                                                             int n_tokens, int vocab, int blocks_per_row,
                                                             float *__restrict__ out, int32_t *status) {
  constexpr int BE = BlockGeom<TYPE>::elems, BB = BlockGeom<TYPE>::bytes;
  const int lane = threadIdx.x & 31;
  const long long total = (long long)n_tokens * blocks_per_row;
  const long long nwarps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long i = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < total; i += nwarps) {
    const int t = (int)(i / blocks_per_row), blk = (int)(i - (long long)t * blocks_per_row);
    const int id = token_ids[t];
    float *y = out + ((long long)t * blocks_per_row + blk) * BE;
    if (id < 0 || id >= vocab) {
      for (int e = lane; e < BE; e += 32) y[e] = 0.f;
      if (status && blk == 0 && lane == 0) atomicMax(status, t + 1);
      continue;
    }
    expand_block<TYPE>(table + ((long long)id * blocks_per_row + blk) * BB, y, lane);
  }
}

template <int TYPE>
int run_embedding(const void *d_table, const int32_t *d_ids, int n_tokens, int vocab, int n_embd,
                  float *d_out, int32_t *d_status, cudaStream_t s) {
  const int bpr = n_embd / BlockGeom<TYPE>::elems;
  const long long want = ((long long)n_tokens * bpr + 7) / 8;
  if (want == 0) return COGNI_QMM_OK;
  const int grid = (int)(want < 148LL * 16 ? want : 148LL * 16);
  embedding_rows_kernel<TYPE><<<grid, 256, 0, s>>>(static_cast<const uint8_t *>(d_table), d_ids,
                                                  n_tokens, vocab, bpr, d_out, d_status);
  return (int)cudaGetLastError();
}

// Elements from which the 16-byte stores pay: below, their few CTAs each expand a chain of blocks while SMs
// idle, and a warp per block is done first.  Measured, us, warp per block / 16-byte stores (graph replay):
// Q8_0 64 K 1.77 / 2.40, 256 K 2.53 / 2.54, 512 K 3.32 / 2.43; IQ4_NL 128 K 2.07 / 2.14, 256 K 2.49 / 2.16; Q4_K 256 K
// 1.93 / 2.80, 1.5 M 3.02 / 2.97; Q5_K 256 K 1.96 / 2.91, 2 M 3.49 / 3.69, 3 M 5.49 / 5.13; Q6_K 256 K 1.92 / 2.52, 2 M
// 3.74 / 3.75, 3 M 4.92 / 4.81.
template <int TYPE>
constexpr int64_t kQuadsFrom = TYPE == kQ8_0 ? 1 << 18 : TYPE == kIQ4_NL ? 3 << 16 : TYPE == kQ4_K ? 3 << 19 : 3 << 20;

template <int TYPE>
int run(const void *d_w, int64_t n, float *d_out, cudaStream_t s) {
  long long nblocks = n / BlockGeom<TYPE>::elems;
  if (nblocks == 0) return COGNI_QMM_OK;
  if (n >= kQuadsFrom<TYPE> && ((reinterpret_cast<uintptr_t>(d_w) | reinterpret_cast<uintptr_t>(d_out)) & 15) == 0) {
    constexpr int per_cta = 256 / kQuadLanes<TYPE> * kQuadUnroll<TYPE>;
    const long long ctas = (nblocks + per_cta - 1) / per_cta;
    if (ctas <= 0x7fffffffLL) {
      dequantize_quads_kernel<TYPE><<<(unsigned)ctas, 256, 0, s>>>(static_cast<const uint8_t *>(d_w), d_out, nblocks);
      return (int)cudaGetLastError();
    }
  }
  long long want = (nblocks + 7) / 8;
  int grid = (int)(want < 148LL * 16 ? want : 148LL * 16);
  dequantize_blocks_kernel<TYPE><<<grid, 256, 0, s>>>(static_cast<const uint8_t *>(d_w), d_out,
                                                     nblocks);
  return (int)cudaGetLastError();
}

}  // namespace

int launch_dequantize(int type, const void *d_w, int64_t n, float *d_out, cudaStream_t s) {
  switch (type) {
    case kQ8_0: return run<kQ8_0>(d_w, n, d_out, s);
    case kIQ4_NL: return run<kIQ4_NL>(d_w, n, d_out, s);
    case kQ4_K: return run<kQ4_K>(d_w, n, d_out, s);
    case kQ5_K: return run<kQ5_K>(d_w, n, d_out, s);
    case kQ6_K: return run<kQ6_K>(d_w, n, d_out, s);
    default: return COGNI_QMM_ERR_TYPE;
  }
}

int launch_embedding_rows(int type, const void *d_table, const int32_t *d_ids, int n_tokens, int vocab,
                          int n_embd, float *d_out, int32_t *d_status, cudaStream_t s) {
  switch (type) {
    case kQ8_0: return run_embedding<kQ8_0>(d_table, d_ids, n_tokens, vocab, n_embd, d_out, d_status, s);
    case kIQ4_NL: return run_embedding<kIQ4_NL>(d_table, d_ids, n_tokens, vocab, n_embd, d_out, d_status, s);
    case kQ4_K: return run_embedding<kQ4_K>(d_table, d_ids, n_tokens, vocab, n_embd, d_out, d_status, s);
    case kQ5_K: return run_embedding<kQ5_K>(d_table, d_ids, n_tokens, vocab, n_embd, d_out, d_status, s);
    case kQ6_K: return run_embedding<kQ6_K>(d_table, d_ids, n_tokens, vocab, n_embd, d_out, d_status, s);
    default: return COGNI_QMM_ERR_TYPE;
  }
}

}  // namespace cogni
