// decoder.cuh -- the map decoder of the surrogate network (mlp.cu).
//
// The network's last dense layer emits, besides its dense outputs, a latent
// grid of S0 x S0 cells with C0 channels (row-major, channels fastest: NHWC).
// The decoder takes it through a ReLU and then through levels that each
// upsample by 2 (nearest neighbour) and apply a 3x3 convolution with zero
// padding and a bias; every level but the last applies a ReLU, the last has
// one output channel: the map.  Activations are BF16 in NHWC, weights BF16 as
// [Cout][9*Cin] with the tap (ty*3+tx) major and the input channel minor,
// padded with zeros to a multiple of 16.
//
// Forward, level l with 16 or more output channels: im2col of the upsampled
// input (k_im2col_up, never materialising the upsampled grid) and the
// tensor-core product (im2col x W^T, bias and ReLU in the epilogue).  A level
// with fewer output channels (the map's one, or 8) is below the tensor
// cores' narrowest tile and runs as a direct convolution (k_dec_conv).
// Backward: the map's gradient in BF16 (k_to_bf16); per level the weight and
// bias gradients by k_dec_dw (k_dec_dw1 for the map's level; per chunk of input
// cells, FP32 sums of the output gradient over the pixels that a cell reaches
// through a tap, times the cell, then summed over the chunks) and the input
// gradient by k_dec_dx (k_dec_dx1; FP32 sums of BF16 products over the taps and
// the 2x2 upsampled cells), in BF16 rows that are the next level's output
// gradient.  The convolution and the input gradient keep the weights in shared
// memory as FP32.  Every sum runs in a fixed order, so training is deterministic.
#pragma once
#include <cuda_bf16.h>

#include <algorithm>
#include <cstdint>

namespace cliffs_nn {

// Two FP32 values in a register pair and Blackwell's packed operations on
// them: each half rounds as the scalar operation does.
using fpair = unsigned long long;
__device__ __forceinline__ fpair pair_of(uint32_t lo, uint32_t hi) {
  return (fpair)hi << 32 | lo;
}
__device__ __forceinline__ fpair pair_add(fpair a, fpair b) {
  fpair r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ void pair_fma(fpair& acc, fpair a, fpair b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float pair_lo(fpair a) { return __uint_as_float((uint32_t)a); }
__device__ __forceinline__ float pair_hi(fpair a) { return __uint_as_float((uint32_t)(a >> 32)); }
// Two BF16 values as FP32.
__device__ __forceinline__ fpair pair_bf16(uint32_t w) { return pair_of(w << 16, w & 0xffff0000u); }

// im2col of the 2x upsampled input: row p = (b, Y, X) of the output grid
// (side 2S), column k = tap * Cin + c < 9 Cin, columns up to kp zero.  The
// upsampled cell (Y', X') = (Y + ty - 1, X + tx - 1) reads input cell
// (Y' / 2, X' / 2); outside [0, 2S) it is zero padding.  dst [P][kp].  A block
// per (b, Y); a thread keeps its 8 columns (one tap, 8 channels: C and kp are
// multiples of 8) and walks along X, one 16-byte load and store a pixel, so that
// the divisions are done once.  Blocks of im2col_threads(kp).  302 MB written at a
// batch of 512: a warp per pixel, 28 of 32 lanes idle in every second round of the
// surrogate's 36 groups, took 171 us, a thread per 8 columns 95, this 56.
__host__ __device__ constexpr int im2col_threads(int kp) { return 256 / (kp / 8) * (kp / 8); }
__global__ void __launch_bounds__(256) k_im2col_up(int S, int C, const __nv_bfloat16* __restrict__ x, int kp,
                                                   __nv_bfloat16* dst) {
  const int S2 = 2 * S, per = kp / 8, step = (int)blockDim.x / per;
  const int b = blockIdx.x / S2, Y = blockIdx.x % S2;
  const int g = (int)threadIdx.x % per, tap = 8 * g / C, c = 8 * g % C;
  const int Yu = Y + tap / 3 - 1, dx = tap % 3 - 1;
  const bool row = tap < 9 && Yu >= 0 && Yu < S2;
  const __nv_bfloat16* src = x + (((size_t)b * S + (row ? Yu >> 1 : 0)) * S) * C + c;
  uint4* out = reinterpret_cast<uint4*>(dst) + (size_t)blockIdx.x * S2 * per + g;
#pragma unroll 4
  for (int X = (int)threadIdx.x / per; X < S2; X += step) {
    const int Xu = X + dx;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (row && Xu >= 0 && Xu < S2) v = __ldg(reinterpret_cast<const uint4*>(src + (size_t)(Xu >> 1) * C));
    out[(size_t)X * per] = v;
  }
}

// The decoder's input: ReLU of the latent columns [col0, col0 + n) of the
// dense output (rows of ld floats) in BF16.
__global__ void k_dec_input(int B, int n, const float* __restrict__ y, int ld, int col0, __nv_bfloat16* x) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= B * n) return;
  const int b = t / n, j = t % n;
  x[t] = __float2bfloat16(fmaxf(y[(size_t)b * ld + col0 + j], 0.f));
}

// Squared-error loss of one output block: y rows (ld_y floats, from column
// y0) against target rows idx[r] (or r) of tg (ld_t floats, from column t0),
// n values per row.  dy (ld_d floats per row, from column d0) gets
// scale (y - t); part[blockIdx.x] a partial sum of (y - t)^2 in a fixed order.
__global__ void __launch_bounds__(256) k_mse_block(int B, int n, const float* __restrict__ y, int ld_y, int y0,
                                                   const float* __restrict__ tg, int ld_t, int t0,
                                                   const int* __restrict__ idx, float* dy, int ld_d, int d0,
                                                   float scale, float* part) {
  __shared__ float s[256];
  float acc = 0.f;
  const int total = B * n;  // < 2^31
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < total; k += gridDim.x * blockDim.x) {
    const int r = k / n, j = k % n;
    const int tr = idx ? idx[r] : r;
    const float d = y[(size_t)r * ld_y + y0 + j] - tg[(size_t)tr * ld_t + t0 + j];
    dy[(size_t)r * ld_d + d0 + j] = scale * d;
    acc += d * d;
  }
  s[threadIdx.x] = acc;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) s[threadIdx.x] += s[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = s[0];
}

// Partial sums [splits][rows][ldp] summed into out [rows][cols] (cols <=
// ldp): block (32 outputs) x (kStrands strands); strand s adds the splits
// z = s, s + kStrands, ... in order, and the strand sums are added in strand
// order, so the result does not depend on the launch.  Column sums of a
// matrix [R][N] are the case rows = 1, cols = ldp = N, splits = R.
constexpr int kStrands = 16;
__global__ void __launch_bounds__(32 * kStrands) k_reduce_wgrad(int rows, int cols, int ldp, int splits,
                                                               const float* __restrict__ part, float* out) {
  __shared__ float sh[kStrands][33];
  const int lane = threadIdx.x & 31, strand = threadIdx.x >> 5;
  const int k = blockIdx.x * 32 + lane;
  const bool in = k < rows * cols;
  float s = 0.f;
  if (in) {
    const int r = k / cols, c = k % cols;
    const float* at = part + (size_t)r * ldp + c;
    const size_t split = (size_t)rows * ldp;
    int z = strand;
    for (; z + 7 * kStrands < splits; z += 8 * kStrands) {  // 8 loads in flight, added in order
      float v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = __ldg(at + (size_t)(z + i * kStrands) * split);
#pragma unroll
      for (int i = 0; i < 8; ++i) s += v[i];
    }
    for (; z < splits; z += kStrands) s += __ldg(at + (size_t)z * split);
  }
  sh[strand][lane] = s;
  __syncthreads();
  if (strand == 0 && in) {
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < kStrands; ++i) t += sh[i][lane];
    out[k] = t;
  }
}

// FP32 to BF16, n values, four a thread (both arrays 16-byte aligned).
__global__ void k_to_bf16(int n, const float* __restrict__ src, __nv_bfloat16* dst) {
  const int t = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (t + 3 < n) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(src + t));
    const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(dst + t) =
        make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
  } else {
    for (int i = t; i < n; ++i) dst[i] = __float2bfloat16(src[i]);
  }
}

// The 8 BF16 values of a 16-byte load as FP32.
__device__ __forceinline__ void unpack8(const uint4 q, float (&v)[8]) {
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] = __uint_as_float(w[i] << 16);
    v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}

// The weights w [co][kp] (BF16, columns k = tap * C + c) into shared memory
// as FP32, [tap][C][co] or (CLAST) [tap][co][C], 8 columns at a time (C and kp
// are multiples of 8).  The whole block calls it; true if every weight is finite.
// A value at a time, 64 x 64 channels took most of a small batch's input gradient:
// the training step below, of a batch of 16 with a map of 8 x 8, 600 us, 469 now.
template <bool CLAST>
__device__ __forceinline__ bool stage_weights(float* sw, int C, int co, const __nv_bfloat16* __restrict__ w, int kp) {
  bool finite = true;
  for (int t = threadIdx.x; t < 9 * C / 8 * co; t += blockDim.x) {
    const int o = CLAST ? t / (C / 8) % co : t % co, k = CLAST ? t / (C / 8 * co) * C + t % (C / 8) * 8 : t / co * 8;
    float v[8];
    unpack8(__ldg(reinterpret_cast<const uint4*>(w + (size_t)o * kp + k)), v);
#pragma unroll
    for (int i = 0; i < 8; ++i) finite = finite && isfinite(v[i]);
    if (CLAST) {
      float4* to = reinterpret_cast<float4*>(sw + 8 * t);
      to[0] = make_float4(v[0], v[1], v[2], v[3]);
      to[1] = make_float4(v[4], v[5], v[6], v[7]);
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) sw[(k + i) * co + o] = v[i];
    }
  }
  return __syncthreads_and(finite);
}

// Direct forward convolution of a level with CO = 1 or 8 output channels: a
// thread per input cell (b, y0, x0), whose 2 x 2 output pixels share the
// weights' reads and, upsampled from 3 x 3 input cells, most of the inputs'.
// Per pixel FP32 sums over the taps (in order) and the input channels, bias
// added; then either ReLU and a BF16 row of CO values (out16, NHWC) or the FP32
// value of the one-channel map (out32).  A tap in the zero padding adds
// products with 0, which leave a sum as it is; with weights that are not
// finite (GUARD) it is passed over.  C a multiple of 8.  Dynamic shared memory:
// 9 C CO floats.  Bound by the FP32 issue (36 C CO products a cell, two to an
// instruction for CO = 8).  A thread per pixel read the weights four times as
// often: at a batch of 512, 212 us for the map's level and 170 us for the
// 8-channel one, against 51 and 107 here (the map's
// level with 8 channels unpacks each of the nine cells once; unpacked at every tap 69)
template <int CO, bool GUARD>
__device__ __forceinline__ void conv_cell(int S, int C, int b, int y0, int x0, const __nv_bfloat16* __restrict__ x,
                                          const float* sw, const float* __restrict__ bias, __nv_bfloat16* out16,
                                          float* out32) {
  constexpr int NP = CO == 8 ? 4 : 1;
  const int S2 = 2 * S;
  fpair acc2[4][NP];
  float acc[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    acc[i] = 0.f;
#pragma unroll
    for (int o = 0; o < NP; ++o) acc2[i][o] = 0;
  }
  if (CO == 1 && !GUARD && C == 8) {  // all taps of the nine cells, each unpacked once
    float xv[9][8];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const int yy = y0 + k / 3 - 1, xx = x0 + k % 3 - 1;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (yy >= 0 && yy < S && xx >= 0 && xx < S)
        v = __ldg(reinterpret_cast<const uint4*>(x) + ((size_t)b * S + yy) * S + xx);
      unpack8(v, xv[k]);
    }
#pragma unroll
    for (int tap = 0; tap < 9; ++tap) {
      const float4 w0 = *reinterpret_cast<const float4*>(sw + 8 * tap);
      const float4 w1 = *reinterpret_cast<const float4*>(sw + 8 * tap + 4);
      const float f[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int k = ((i >> 1) + tap / 3 + 1) / 2 * 3 + ((i & 1) + tap % 3 + 1) / 2;
#pragma unroll
        for (int g = 0; g < 8; ++g) acc[i] = fmaf(xv[k][g], f[g], acc[i]);
      }
    }
    C = 0;  // done
  }
#pragma unroll
  for (int tap = 0; tap < 9; ++tap) {
    const int ty = tap / 3, tx = tap % 3;
#pragma unroll 1
    for (int c8 = 0; c8 < C; c8 += 8) {
      uint4 v[4];  // pixel (a, e) = i reads input cell (y0 + dy, x0 + dx) through the tap
      bool in[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int a = i >> 1, e = i & 1;
        const int yy = y0 + (a + ty + 1) / 2 - 1, xx = x0 + (e + tx + 1) / 2 - 1;
        if (e == 1 && tx != 0 && tx != 2) {
          v[i] = v[i - 1], in[i] = in[i - 1];  // the cell of the pixel to the left
        } else if (a == 1 && ty == 1) {
          v[i] = v[i - 2], in[i] = in[i - 2];  // of the pixel above
        } else {
          v[i] = make_uint4(0u, 0u, 0u, 0u);
          in[i] = yy >= 0 && yy < S && xx >= 0 && xx < S;
          if (in[i]) v[i] = __ldg(reinterpret_cast<const uint4*>(x + (((size_t)b * S + yy) * S + xx) * C + c8));
        }
      }
      const float* wt = sw + (tap * C + c8) * CO;
      if constexpr (CO == 8) {
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          const ulonglong2 w0 = *reinterpret_cast<const ulonglong2*>(wt + g * 8);
          const ulonglong2 w1 = *reinterpret_cast<const ulonglong2*>(wt + g * 8 + 4);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t q = g < 2 ? v[i].x : g < 4 ? v[i].y : g < 6 ? v[i].z : v[i].w;
            const uint32_t f = g & 1 ? q & 0xffff0000u : q << 16;
            const fpair d = pair_of(f, f);
            if (!GUARD || in[i]) {
              pair_fma(acc2[i][0], d, w0.x);
              pair_fma(acc2[i][1], d, w0.y);
              pair_fma(acc2[i][2], d, w1.x);
              pair_fma(acc2[i][3], d, w1.y);
            }
          }
        }
      } else {
        const float4 w0 = *reinterpret_cast<const float4*>(wt), w1 = *reinterpret_cast<const float4*>(wt + 4);
        const float f[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float xv[8];
          unpack8(v[i], xv);
          if (!GUARD || in[i]) {
#pragma unroll
            for (int g = 0; g < 8; ++g) acc[i] = fmaf(xv[g], f[g], acc[i]);
          }
        }
      }
    }
  }
#pragma unroll
  for (int a = 0; a < 2; ++a) {
    const size_t p = ((size_t)b * S2 + 2 * y0 + a) * S2 + 2 * x0;
    if constexpr (CO == 8) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        uint32_t w[4];
#pragma unroll
        for (int o = 0; o < 4; ++o) {
          const fpair r = acc2[2 * a + e][o];
          const __nv_bfloat162 h = __floats2bfloat162_rn(fmaxf(pair_lo(r) + bias[2 * o], 0.f),
                                                         fmaxf(pair_hi(r) + bias[2 * o + 1], 0.f));
          w[o] = *reinterpret_cast<const uint32_t*>(&h);
        }
        *reinterpret_cast<uint4*>(out16 + (p + e) * 8) = make_uint4(w[0], w[1], w[2], w[3]);
      }
    } else {
      *reinterpret_cast<float2*>(out32 + p) = make_float2(acc[2 * a] + bias[0], acc[2 * a + 1] + bias[0]);
    }
  }
}
template <int CO>
__global__ void __launch_bounds__(256) k_dec_conv(int B, int S, int C, const __nv_bfloat16* __restrict__ x,
                                                  const __nv_bfloat16* __restrict__ w, int kp,
                                                  const float* __restrict__ bias, __nv_bfloat16* out16, float* out32) {
  extern __shared__ __align__(16) float sw[];
  const bool finite = stage_weights<false>(sw, C, CO, w, kp);
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= B * S * S) return;
  const int b = q / (S * S), y0 = (q / S) % S, x0 = q % S;
  if (finite)
    conv_cell<CO, false>(S, C, b, y0, x0, x, sw, bias, out16, out32);
  else
    conv_cell<CO, true>(S, C, b, y0, x0, x, sw, bias, out16, out32);
}

// The weight gradients of a level are sums over the input cells.  The 2x upsampling
// makes four upsampled cells of an input cell (y0, x0), and through tap (ty, tx)
// these are read by the four output pixels in rows 2 y0 + 1 - ty, 2 y0 + 2 - ty
// and columns 2 x0 + 1 - tx, 2 x0 + 2 - tx.  So with D[tap][o] the sum of the
// output gradient over those four pixels (inside the grid),
//   dW[o][tap][c] = sum over cells of D[tap][o] x[c]
//   db[o]         = sum over cells of D[centre][o]
// a quarter of the products of the sums over output pixels, and the nine D of a
// cell come from one window of 4 x 4 pixels.

// The 8 gradients o0 .. o0 + 7 of pixel (Y, X), as FP32 pairs; 0 outside.
__device__ __forceinline__ void dz_pixel(const __nv_bfloat16* __restrict__ dz, int b, int S2, int Y, int X, int co,
                                         int o0, fpair (&v)[4]) {
  uint4 q = make_uint4(0u, 0u, 0u, 0u);
  if (Y >= 0 && Y < S2 && X >= 0 && X < S2)
    q = __ldg(reinterpret_cast<const uint4*>(dz + (((size_t)b * S2 + Y) * S2 + X) * co + o0));
  v[0] = pair_bf16(q.x);
  v[1] = pair_bf16(q.y);
  v[2] = pair_bf16(q.z);
  v[3] = pair_bf16(q.w);
}

// Columns X .. X + N + 1 of row Y of the one-channel gradient, 0 outside; X odd,
// N even: the N in the middle are read in pairs.
template <int N>
__device__ __forceinline__ void dz_row(const __nv_bfloat16* __restrict__ dz, int b, int S2, int Y, int X,
                                       float (&v)[N + 2]) {
#pragma unroll
  for (int j = 0; j < N + 2; ++j) v[j] = 0.f;
  if (Y < 0 || Y >= S2) return;
  const __nv_bfloat16* r = dz + ((size_t)b * S2 + Y) * S2;
  if (X >= 0) v[0] = __bfloat162float(r[X]);
#pragma unroll
  for (int j = 1; j < N + 1; j += 2)
    if (X + j < S2) {
      const uint32_t q = __ldg(reinterpret_cast<const unsigned int*>(r + X + j));
      v[j] = __uint_as_float(q << 16);
      v[j + 1] = __uint_as_float(q & 0xffff0000u);
    }
  if (X + N + 1 < S2) v[N + 1] = __bfloat162float(r[X + N + 1]);
}

// Partial weight and bias gradients of a level with co (a multiple of 8) output
// channels over one chunk of input cells (block z: cells [z chunk, (z+1) chunk)).
// Per run of STAGE cells the block puts D and x as FP32 into shared memory, a row
// of STAGE + 4 floats for each of the 9 co (tap, o) and of its channels, and
// multiplies them: thread (slot, mm, nn) holds the 8 x 4 sums of rows mm + i mt
// and channels nn + j nb (mt = 9 co / 8; neighbouring threads read neighbouring
// rows, in other banks), and takes every NS-th group of 4 cells, two cells to a
// packed product.  12 16-byte reads of shared memory feed 128 products.  The
// slots' sums are then added in slot order.  Channels beyond 4 nb go to further
// blockIdx.y.  part [blocks][co][9C], part_b [blocks][co] (from blockIdx.y = 0).
// At a batch of 512, 32 -> 16 and 16 -> 8 channels took 322 and 323 us with a
// thread per column that walked the output pixels; 75 each here, most
// of it staging and the reads of shared memory (604 M products each).
constexpr int kDwTiles = 512;    // most threads of a slot
constexpr int kDwThreads = 160;  // threads wanted in a block: at 128 registers, three blocks an SM
constexpr int dw_stage(int co) { return co <= 8 ? 128 : 64; }
struct DwPlan {  // of co output and C input channels
  int nb, slots, threads, smem;
};
inline DwPlan dw_plan(int co, int C) {
  const int mt = 9 * co / 8, stage = dw_stage(co);
  DwPlan p;
  p.nb = std::min(C / 4, kDwTiles / mt) & ~1;  // at least 2 (mt <= 72): whole groups of 8 channels
  p.slots = std::max(1, std::min(stage / 4, kDwThreads / (mt * p.nb)));
  p.threads = (mt * p.nb * p.slots + 31) / 32 * 32;
  p.smem = std::max((9 * co + 4 * p.nb) * (stage + 4), p.slots > 1 ? mt * p.nb * 33 : 0) * 4 + co * 4;
  return p;
}
template <int STAGE>
__global__ void __launch_bounds__(kDwTiles) k_dec_dw(int cells, int S, int C, int co, int nb, int slots,
                                                     const __nv_bfloat16* __restrict__ dz,
                                                     const __nv_bfloat16* __restrict__ x, int chunk, float* part,
                                                     float* part_b) {
  constexpr int LD = STAGE + 4;
  extern __shared__ __align__(16) float sm[];
  const int M = 9 * co, mt = M / 8, T = mt * nb, S2 = 2 * S;
  const int cb = blockIdx.y * 4 * nb, cn = min(4 * nb, C - cb), nl = cn / 4;  // this block's channels
  float* sb = sm;                    // [co] bias sums
  float* sd = sm + co;               // [M][LD]
  float* sx = sd + (size_t)M * LD;   // [cn][LD]
  const int t = threadIdx.x, slot = t / T, tt = t % T, mm = tt % mt, nn = tt / mt;
  const bool worker = slot < slots && nn < nl;
  const int q0 = blockIdx.x * chunk, n = min(chunk, cells - q0);
  fpair acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0;
  for (int o = t; o < co; o += blockDim.x) sb[o] = 0.f;
  for (int r0 = 0; r0 < n; r0 += STAGE) {
    __syncthreads();  // the previous run is consumed
    const int nd = STAGE * (co / 8), all = nd + STAGE * (cn / 8);
    for (int k = t; k < all; k += blockDim.x) {
      const bool isd = k < nd;
      const int j = k % STAGE, g = 8 * ((isd ? k : k - nd) / STAGE);  // cell, first of 8 channels
      const int q = q0 + r0 + j;
      const bool in = r0 + j < n;
      if (isd) {
        const int b = q / (S * S), y0 = (q / S) % S, x0 = q % S;
        float* to = sd + (size_t)g * LD + j;
        fpair h[3][4];  // sums of neighbouring columns, the row above
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          fpair p[4][4];
#pragma unroll
          for (int e = 0; e < 4; ++e)
            dz_pixel(dz, b, S2, in ? 2 * y0 - 1 + r : -1, 2 * x0 - 1 + e, co, g, p[e]);
#pragma unroll
          for (int e = 0; e < 3; ++e)
#pragma unroll
            for (int o = 0; o < 4; ++o) {
              const fpair s = pair_add(p[e][o], p[e + 1][o]);
              if (r > 0) {
                const fpair d = pair_add(h[e][o], s);  // tap (3 - r, 2 - e)
                float* at = to + (size_t)((3 * (3 - r) + 2 - e) * co + 2 * o) * LD;
                at[0] = pair_lo(d);
                at[LD] = pair_hi(d);
              }
              h[e][o] = s;
            }
        }
      } else {
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (in) v = __ldg(reinterpret_cast<const uint4*>(x + (size_t)q * C + cb + g));
        float f[8];
        unpack8(v, f);
        float* to = sx + (size_t)g * LD + j;
#pragma unroll
        for (int i = 0; i < 8; ++i) to[i * LD] = f[i];
      }
    }
    __syncthreads();
    if (blockIdx.y == 0)  // db: the centre tap's sums, a warp per channel
      for (int o = t >> 5; o < co; o += blockDim.x >> 5) {
        const float* d = sd + (size_t)(4 * co + o) * LD;
        float s = 0.f;
#pragma unroll
        for (int j = 0; j < STAGE; j += 32) s += d[j + (t & 31)];
#pragma unroll
        for (int k = 16; k > 0; k >>= 1) s += __shfl_xor_sync(0xffffffffu, s, k);
        if ((t & 31) == 0) sb[o] += s;
      }
    if (worker) {
      const float* d0 = sd + (size_t)mm * LD;
      const float* x0 = sx + (size_t)nn * LD;
#pragma unroll 1
      for (int k = 4 * slot; k < STAGE; k += 4 * slots) {
        ulonglong2 xv[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) xv[j] = *reinterpret_cast<const ulonglong2*>(x0 + (size_t)j * nl * LD + k);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const ulonglong2 d = *reinterpret_cast<const ulonglong2*>(d0 + (size_t)i * mt * LD + k);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            pair_fma(acc[i][j], d.x, xv[j].x);
            pair_fma(acc[i][j], d.y, xv[j].y);
          }
        }
      }
    }
  }
  float v[32];
#pragma unroll
  for (int k = 0; k < 32; ++k) v[k] = pair_lo(acc[k / 4][k % 4]) + pair_hi(acc[k / 4][k % 4]);
  __syncthreads();
  if (blockIdx.y == 0)
    for (int o = t; o < co; o += blockDim.x) part_b[(size_t)blockIdx.x * co + o] = sb[o];
  if (slots > 1) {  // added in slot order
    float* sacc = sd + tt * 33;
    for (int s = 0; s < slots; ++s) {
      if (worker && slot == s)
#pragma unroll
        for (int k = 0; k < 32; ++k) {
          if (s > 0) v[k] += sacc[k];
          sacc[k] = v[k];
        }
      __syncthreads();
    }
  }
  if (worker && slot == slots - 1)
#pragma unroll
    for (int k = 0; k < 32; ++k) {
      const int row = mm + k / 4 * mt, c = cb + nn + k % 4 * nl;
      part[((size_t)blockIdx.x * co + row % co) * 9 * C + row / co * C + c] = v[k];
    }
}

// The same for one output channel (the map's level): a thread per input cell of
// the chunk, stepping by the block, and the 8 channels from 8 blockIdx.y; its 72
// sums stay in registers, then the block's are added in a fixed order.  278 us at
// a batch of 512 before, 55 here (151 M products; loads of pairs and single values).
constexpr int kDw1Threads = 160;
__global__ void __launch_bounds__(kDw1Threads) k_dec_dw1(int cells, int S, int C, const __nv_bfloat16* __restrict__ dz,
                                                         const __nv_bfloat16* __restrict__ x, int chunk, float* part,
                                                         float* part_b) {
  __shared__ float red[kDw1Threads / 32][73];
  const int S2 = 2 * S, cb = 8 * blockIdx.y;
  const int q0 = blockIdx.x * chunk, q1 = min(q0 + chunk, cells);
  float acc[73];  // [tap][channel], then the bias
#pragma unroll
  for (int k = 0; k < 73; ++k) acc[k] = 0.f;
  for (int q = q0 + threadIdx.x; q < q1; q += kDw1Threads) {
    const int b = q / (S * S), y0 = (q / S) % S, x0 = q % S;
    float xv[8];
    unpack8(__ldg(reinterpret_cast<const uint4*>(x + (size_t)q * C + cb)), xv);
    float p[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r) dz_row<2>(dz, b, S2, 2 * y0 - 1 + r, 2 * x0 - 1, p[r]);
#pragma unroll
    for (int ty = 0; ty < 3; ++ty)
#pragma unroll
      for (int tx = 0; tx < 3; ++tx) {
        const int r = 2 - ty, e = 2 - tx;
        const float d = (p[r][e] + p[r][e + 1]) + (p[r + 1][e] + p[r + 1][e + 1]);
        if (ty == 1 && tx == 1) acc[72] += d;
#pragma unroll
        for (int g = 0; g < 8; ++g) acc[(ty * 3 + tx) * 8 + g] = fmaf(d, xv[g], acc[(ty * 3 + tx) * 8 + g]);
      }
  }
#pragma unroll
  for (int k = 0; k < 73; ++k) {
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], w);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][k] = acc[k];
  }
  __syncthreads();
  const int k = threadIdx.x;
  if (k < 73) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < kDw1Threads / 32; ++w) s += red[w][k];
    if (k < 72)
      part[(size_t)blockIdx.x * 9 * C + k / 8 * C + cb + k % 8] = s;
    else if (blockIdx.y == 0)
      part_b[blockIdx.x] = s;
  }
}

// Writes the gradients of N (4 or 8) channels of an input cell: the ReLU
// derivative applied (mask: x's own values, x > 0), as a BF16 row (the output
// gradient of the level above) or as FP32.
template <int N>
__device__ __forceinline__ void dx_store(const float (&v)[N], const __nv_bfloat16* mask, size_t at, size_t to,
                                         __nv_bfloat16* dx16, float* dx32) {
  uint32_t w[N / 2];
  float r[N];
  if constexpr (N == 8) {
    const uint4 q = __ldg(reinterpret_cast<const uint4*>(mask + at));
    w[0] = q.x, w[1] = q.y, w[2] = q.z, w[3] = q.w;
  } else {
    const uint2 q = __ldg(reinterpret_cast<const uint2*>(mask + at));
    w[0] = q.x, w[1] = q.y;
  }
#pragma unroll
  for (int g = 0; g < N; ++g)
    r[g] = __uint_as_float(g & 1 ? w[g / 2] & 0xffff0000u : w[g / 2] << 16) > 0.f ? v[g] : 0.f;
  if (dx16) {
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
      const __nv_bfloat162 h = __floats2bfloat162_rn(r[2 * i], r[2 * i + 1]);
      w[i] = *reinterpret_cast<const uint32_t*>(&h);
    }
    if constexpr (N == 8)
      *reinterpret_cast<uint4*>(dx16 + at) = make_uint4(w[0], w[1], w[2], w[3]);
    else
      *reinterpret_cast<uint2*>(dx16 + at) = make_uint2(w[0], w[1]);
  } else {
#pragma unroll
    for (int g = 0; g < N; ++g) dx32[to + g] = r[g];
  }
}

// Gradient of the level input x (B, S, S, C) from the output gradient dz (B, 2S,
// 2S pixels of co BF16 values) and the weights w [co][kp], with x's ReLU
// derivative: BF16 rows (dx16), or FP32 with sample b's S S C values at dx32 +
// b ld + col0.  The 3x3 correlation transposed, summed over the 2x2 upsampled
// cells of each input cell: FP32 sums over (cell, tap, o) in order, a channel
// each (the sums over D above would round otherwise, and what is rounded here
// goes through every layer below).  A thread takes two cells, one below the
// other, so that neighbouring lanes read neighbouring pixels, and G channels (16,
// or 8 where C is no multiple of 16; fewer where so few cells leave SMs without a
// block, dx_group): 16 bytes of weights from shared memory serve 8 products.  A pixel in the zero padding adds products with 0, which leave a sum
// as it is; with weights that are not finite (GUARD) it is passed over.  Dynamic
// shared memory: 9 C co floats, [tap][o][c].  36 C co products a cell, 65 us of
// FP32 issue at a batch of 512 for 32 <- 16 and for 16 <- 8 channels; these took
// 432 and 230 us with a cell and 2 or 4 channels a thread, 165 and 144 here.  Two
// cells side by side: 187 and 141; 8 channels: 190 and 156; four cells: 185 and 142;
// packed products: 157 each, the copies into pairs costing what they save.
constexpr int kDxThreads = 128, kDxCells = 2;
// Channels a thread: 16, or half and a quarter of that while the blocks, which
// hold an SM each where there are many channels, still all run at once on 152
// SMs: a block lasts as long as a thread's products.  A training step of a batch
// of 16 with 64 channels throughout and a map of 8 x 8 (16 x 16, 32 x 32) took 682
// us (752, 850) with 16 channels always, 600 (663, 760) this way; where 8 channels
// make more than 152 blocks they lose (batch of 128, 32 x 32: 911 us against 830).
constexpr int kDxFill = 152;
inline int dx_group(long long runs, int C) {
  int g = C % 16 ? 8 : 16;
  while (g > 4 && (runs * (C / (g / 2)) + kDxThreads - 1) / kDxThreads <= kDxFill) g /= 2;
  return g;
}
template <int G, bool GUARD>
__device__ __forceinline__ void dx_cells(int S, int C, int co, int b, int y0, int x0, int c0,
                                         const __nv_bfloat16* __restrict__ dz, const float* sw, float (&acc)[kDxCells][G]) {
  const int S2 = 2 * S;
#pragma unroll 1
  for (int ae = 0; ae < 4; ++ae) {
    const int Yu = 2 * y0 + (ae >> 1), Xu = 2 * x0 + (ae & 1);  // the upsampled cell
#pragma unroll 1
    for (int ty = 0; ty < 3; ++ty) {
      const int Y = Yu - (ty - 1);  // output row that read it through tap ty
#pragma unroll
      for (int tx = 0; tx < 3; ++tx) {
        const int X = Xu - (tx - 1);
        const __nv_bfloat16* px = dz + (((ptrdiff_t)b * S2 + Y) * S2 + X) * co;
        bool in[kDxCells];
#pragma unroll
        for (int m = 0; m < kDxCells; ++m) in[m] = Y + 2 * m >= 0 && Y + 2 * m < S2 && X >= 0 && X < S2;
        const float* wt = sw + (ty * 3 + tx) * co * C + c0;
#pragma unroll 1
        for (int o8 = 0; o8 < co; o8 += 8) {
          uint4 q[kDxCells];
#pragma unroll
          for (int m = 0; m < kDxCells; ++m) {
            q[m] = make_uint4(0u, 0u, 0u, 0u);
            if (in[m]) q[m] = __ldg(reinterpret_cast<const uint4*>(px + (ptrdiff_t)(2 * m) * S2 * co + o8));
          }
#pragma unroll
          for (int o = 0; o < 8; ++o) {
            const float4* wp = reinterpret_cast<const float4*>(wt + (o8 + o) * C);
            float f[G];
#pragma unroll
            for (int k = 0; k < G / 4; ++k) {
              const float4 v = wp[k];
              f[4 * k] = v.x, f[4 * k + 1] = v.y, f[4 * k + 2] = v.z, f[4 * k + 3] = v.w;
            }
#pragma unroll
            for (int m = 0; m < kDxCells; ++m) {
              const uint32_t h = o < 2 ? q[m].x : o < 4 ? q[m].y : o < 6 ? q[m].z : q[m].w;
              const float d = __uint_as_float(o & 1 ? h & 0xffff0000u : h << 16);
              if (!GUARD || in[m]) {
#pragma unroll
                for (int k = 0; k < G; ++k) acc[m][k] = fmaf(d, f[k], acc[m][k]);
              }
            }
          }
        }
      }
    }
  }
}
template <int G>
__global__ void __launch_bounds__(kDxThreads) k_dec_dx(int B, int S, int C, int co,
                                                       const __nv_bfloat16* __restrict__ dz,
                                                       const __nv_bfloat16* __restrict__ w, int kp,
                                                       const __nv_bfloat16* __restrict__ x, __nv_bfloat16* dx16,
                                                       float* dx32, int ld, int col0) {
  constexpr int N = G < 8 ? G : 8;  // of a store
  extern __shared__ __align__(16) float sw[];
  const bool finite = stage_weights<true>(sw, C, co, w, kp);
  const int pr = (S + kDxCells - 1) / kDxCells, runs = B * S * pr;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= runs * (C / G)) return;
  const int c0 = t / runs * G, u = t % runs;
  const int x0 = u % S, y0 = (u / S) % pr * kDxCells, b = u / (pr * S);
  float acc[kDxCells][G];
#pragma unroll
  for (int m = 0; m < kDxCells; ++m)
#pragma unroll
    for (int g = 0; g < G; ++g) acc[m][g] = 0.f;
  if (finite)
    dx_cells<G, false>(S, C, co, b, y0, x0, c0, dz, sw, acc);
  else
    dx_cells<G, true>(S, C, co, b, y0, x0, c0, dz, sw, acc);
#pragma unroll
  for (int m = 0; m < kDxCells; ++m) {
    if (y0 + m >= S) break;
    const size_t cell = (size_t)(y0 + m) * S + x0;
#pragma unroll
    for (int h = 0; h < G; h += N) {
      float v[N];
#pragma unroll
      for (int g = 0; g < N; ++g) v[g] = acc[m][h + g];
      dx_store<N>(v, x, ((size_t)b * S * S + cell) * C + c0 + h, (size_t)b * ld + col0 + cell * C + c0 + h, dx16, dx32);
    }
  }
}

// The same for one output channel (the map's level), the window of 4 x 6 pixels
// in registers: 105 us at a batch of 512 before, 58 here (two cells and 128 threads: with 256 one block of 158 registers an SM, 92).
template <bool GUARD>
__device__ __forceinline__ void dx1_cells(int S, int y0, int x0, const float (&p)[4][6], const float* wt, int C,
                                          fpair (&acc)[2][4]) {
#pragma unroll
  for (int ae = 0; ae < 4; ++ae)
#pragma unroll
    for (int tap = 0; tap < 9; ++tap) {
      const int r = (ae >> 1) - tap / 3 + 2, e = (ae & 1) - tap % 3 + 2;  // row, column in the window
      const ulonglong2* wp = reinterpret_cast<const ulonglong2*>(wt + tap * C);
      const ulonglong2 f0 = wp[0], f1 = wp[1];
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const uint32_t h = __float_as_uint(p[r][e + 2 * m]);
        const fpair d = pair_of(h, h);
        const int Y = 2 * y0 - 1 + r, X = 2 * x0 - 1 + e + 2 * m;
        if (!GUARD || (Y >= 0 && Y < 2 * S && X >= 0 && X < 2 * S)) {
          pair_fma(acc[m][0], d, f0.x);
          pair_fma(acc[m][1], d, f0.y);
          pair_fma(acc[m][2], d, f1.x);
          pair_fma(acc[m][3], d, f1.y);
        }
      }
    }
}
__global__ void __launch_bounds__(kDxThreads, 4) k_dec_dx1(int B, int S, int C, const __nv_bfloat16* __restrict__ dz,
                                                 const __nv_bfloat16* __restrict__ w, int kp,
                                                 const __nv_bfloat16* __restrict__ x, __nv_bfloat16* dx16) {
  extern __shared__ __align__(16) float sw[];
  const bool finite = stage_weights<true>(sw, C, 1, w, kp);
  const int pr = (S + 1) / 2, runs = B * S * pr, S2 = 2 * S;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= runs * (C / 8)) return;
  const int c0 = t / runs * 8, u = t % runs;
  const int x0 = u % pr * 2, y0 = (u / pr) % S, b = u / (pr * S);
  float p[4][6];
  fpair acc[2][4] = {};
#pragma unroll
  for (int r = 0; r < 4; ++r) dz_row<4>(dz, b, S2, 2 * y0 - 1 + r, 2 * x0 - 1, p[r]);
  if (finite)
    dx1_cells<false>(S, y0, x0, p, sw + c0, C, acc);
  else
    dx1_cells<true>(S, y0, x0, p, sw + c0, C, acc);
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    float v[8];
#pragma unroll
    for (int g = 0; g < 4; ++g) v[2 * g] = pair_lo(acc[m][g]), v[2 * g + 1] = pair_hi(acc[m][g]);
    if (x0 + m < S) dx_store<8>(v, x, (((size_t)b * S + y0) * S + x0 + m) * C + c0, 0, dx16, nullptr);
  }
}

}  // namespace cliffs_nn
