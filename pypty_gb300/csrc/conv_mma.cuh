// 3x3 convolutions of the warm-start network on the tensor cores (tcgen05), as implicit GEMMs.
//
// Staging. Activations are BF16 NCHW in global memory; a tile with its halo is staged in shared
// memory as [chunk of 8 channels][pixel][8 channels], 16 bytes per (chunk, pixel). That is the
// unswizzled core-matrix order of tcgen05 both with channels along K (forward and data gradient:
// rows are pixels, K-major) and with pixels along K (weight gradient: MN-major), and a tap
// (dy, dx) of the kernel is a constant offset of (dy * pitch + dx) * 16 bytes of the start
// address: the tile is staged once for all nine taps, and no image is expanded.
//
// Precision. The FP32 weights are split into three BF16 terms (8 + 8 + 8 bits: every bit of the
// weight), whose products with BF16 activations are exact; the three terms have accumulators of
// their own, added in FP32 at the end. The weight gradient's operands are BF16 as they are; the
// tensor core's accumulation truncates, so its FP32 accumulators hold the sum of 128 pixels at a
// time and are drained into registers by round-to-nearest adds: 1.0e-7 to 1.3e-7 of the norm from
// the FP64 sum where FP32 FMAs in pixel order were 1.1e-7 to 1.9e-7 (256 pixels at a time:
// 1.5e-7 to 1.7e-7).
//
// What bounds it: staging (global loads, the split of the weights, shared-memory stores); the MMAs
// take about a fifth of the time, two CTAs per SM overlap one's staging with the other's MMAs. On
// CUDA cores, 4 x 64 -> 64 channels x 128 x 128: forward 209, data gradient 207, weight gradient
// 490 us; here 39, 33 and 47 us (the weight gradient with one MMA per tap and N = 16: 61 us;
// the forward reading the weights as single floats: 67 us).
#pragma once
#include "plan.h"
#include "umma.cuh"

namespace pty {
namespace nn {

typedef __nv_bfloat16 bf16;

// unswizzled descriptor: `lbo` the stride between core matrices along the 16-byte direction's
// neighbour (K-major: K; MN-major: K groups of 8), `sbo` the other (K-major: groups of 8 rows;
// MN-major: chunks of 8 along MN)
__device__ __forceinline__ uint64_t desc_plain(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) |
         ((uint64_t)1 << 46);
}

__device__ __forceinline__ bool nonfinite_pair(uint32_t p) {   // two BF16
  return (p & 0x7F80u) == 0x7F80u || (p & 0x7F800000u) == 0x7F800000u;
}

// two neighbouring BF16 of a row; `wide`: the tensor's base is 4-byte aligned (rows are, being
// multiples of 32 pixels)
__device__ __forceinline__ uint32_t ld_pair(const bf16* p, bool wide) {
  if (wide) return *reinterpret_cast<const uint32_t*>(p);
  const uint16_t* q = reinterpret_cast<const uint16_t*>(p);
  return (uint32_t)q[0] | ((uint32_t)q[1] << 16);
}

// Stage channels [c0, c0 + 8 * CH) of a tile with its halo (origin y0 - 1, x0 - 2; PITCH pixels a row,
// ROWS rows; zero outside the image and beyond C channels) by `nth` threads. COPIES = 0: as
// [chunk][row][PITCH]. COPIES = TW: as three tiles shifted by one pixel, [dx][chunk][row][TW] with
// pixel x0 - 1 + dx first, so that the taps of a row are neighbours along an MMA's N. Returns
// whether this thread met a non-finite value.
template <int CH, int PITCH, int ROWS, int COPIES = 0>
__device__ __forceinline__ bool stage_tile(unsigned char* dst, const bf16* __restrict__ src, int c0, int C, int H,
                                           int Wd, int y0, int x0, bool wide, int nth) {
  constexpr int PAIRS = PITCH / 2, PER = ROWS * PAIRS;
  const size_t plane = (size_t)H * Wd;
  bool bad = false;
  for (int e = threadIdx.x; e < CH * PER; e += nth) {
    const int ch = e / PER, r = (e % PER) / PAIRS, cp = e % PAIRS;
    const int y = y0 - 1 + r, x = x0 - 2 + 2 * cp;
    uint32_t p[8];
    const bool in = y >= 0 && y < H && x >= 0 && x < Wd;   // pairs lie inside or outside as a whole
    const bf16* s = src + (size_t)(c0 + 8 * ch) * plane + (in ? (size_t)y * Wd + x : 0);
#pragma unroll
    for (int k = 0; k < 8; ++k) p[k] = (in && c0 + 8 * ch + k < C) ? ld_pair(s + k * plane, wide) : 0u;
#pragma unroll
    for (int k = 0; k < 8; ++k) bad |= nonfinite_pair(p[k]);
    uint4 a, b;
    a.x = __byte_perm(p[0], p[1], 0x5410), a.y = __byte_perm(p[2], p[3], 0x5410);
    a.z = __byte_perm(p[4], p[5], 0x5410), a.w = __byte_perm(p[6], p[7], 0x5410);
    b.x = __byte_perm(p[0], p[1], 0x7632), b.y = __byte_perm(p[2], p[3], 0x7632);
    b.z = __byte_perm(p[4], p[5], 0x7632), b.w = __byte_perm(p[6], p[7], 0x7632);
    if constexpr (COPIES == 0) {
      uint4* d = reinterpret_cast<uint4*>(dst) + (ch * ROWS + r) * PITCH + 2 * cp;
      d[0] = a;
      d[1] = b;
    } else {
#pragma unroll
      for (int dx = 0; dx < 3; ++dx) {
        uint4* d = reinterpret_cast<uint4*>(dst) + ((dx * CH + ch) * ROWS + r) * COPIES;
        const int c = 2 * cp - 1 - dx;   // the first pixel's place in this copy
        if (c >= 0 && c < COPIES) d[c] = a;
        if (c + 1 >= 0 && c + 1 < COPIES) d[c + 1] = b;
      }
    }
  }
  return bad;
}

// ------------------------------------------------------------------ forward and data gradient
// A CTA computes a 16 x 16 pixel tile for 32 output channels: two MMA row blocks of 8 x 16 pixels
// (a group of 8 rows is 8 pixels of an image row, groups one halo row apart), N = 3 x 32 columns
// (the three weight terms), input channels in stages of 32.
struct ConvCfg {
  static constexpr int THREADS = 256, T = 16, CO = 32, CI = 32;
  static constexpr int PITCH = T + 4, ROWS = T + 2, PX = PITCH * ROWS;
  static constexpr int N = 3 * CO;
  static constexpr uint32_t X_CHUNK = PX * 16;                 // bytes between chunks of 8 channels
  static constexpr uint32_t X_BYTES = (CI / 8) * X_CHUNK;
  static constexpr uint32_t W_BLOCK = 2 * N * 16;              // one tap, 16 input channels
  static constexpr uint32_t W_BYTES = (CI / 16) * 9 * W_BLOCK;
  static constexpr uint32_t SMEM = X_BYTES + W_BYTES;
  static_assert(CO * T * T * 2 <= (int)X_BYTES, "the output tile reuses the input's buffer");
};

// TRANS = 0: out[n][o][p] = act(b[o] + sum_i sum_t w[o][i][t] x[n][i][p + off(t)])   (forward)
// TRANS = 1: out[n][o][p] =          sum_i sum_t w[i][o][8 - t] x[n][i][p + off(t)]    (data gradient)
template <int TRANS, int RELU>
__global__ void __launch_bounds__(ConvCfg::THREADS, 2)
    conv3x3_mma_kernel(const bf16* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias,
                       bf16* __restrict__ out, int Ci, int Co, int H, int Wd, int wide, int wide4) {
  using C = ConvCfg;
  extern __shared__ __align__(128) unsigned char sm[];
  unsigned char *sx = sm, *sw = sm + C::X_BYTES;
  __shared__ uint64_t bar;
  __shared__ uint32_t tmem_s;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tiles_x = Wd / C::T;
  const int y0 = (blockIdx.x / tiles_x) * C::T, x0 = (blockIdx.x % tiles_x) * C::T;
  const int o0 = blockIdx.y * C::CO, n = blockIdx.z;
  const size_t plane = (size_t)H * Wd;
  const bf16* xn = x + (size_t)n * Ci * plane;
  if (tid == 0) {
    mbar_init(&bar, 1);
    fence_async_shared();
  }
  if (warp == 0) umma::tmem_alloc(&tmem_s, 256);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = tmem_s;
  uint32_t par = 0;
  int err = 0;
  bool bad = false;
  const int stages = (Ci + C::CI - 1) / C::CI;
  for (int s = 0; s < stages; ++s) {
    const int c0 = s * C::CI;
    if (s > 0) mbar_wait(&bar, par, &err);   // the previous stage's MMAs have read the buffers
    bad |= stage_tile<C::CI / 8, C::PITCH, C::ROWS>(sx, xn, c0, Ci, H, Wd, y0, x0, wide != 0, C::THREADS);
    // weights: a task is one output channel and four input channels with their nine taps; the
    // forward's 36 floats are neighbours in w, the data gradient's lanes are neighbours
    static_assert(C::CO * C::CI / 4 == C::THREADS, "one task per thread");
    {
      const int o = tid % C::CO, k4 = tid / C::CO, go = o0 + o, gi = c0 + 4 * k4;
      float v[4][9];
      if (!TRANS && wide4 && go < Co && gi < Ci) {
        const float4* wp = reinterpret_cast<const float4*>(w + ((size_t)go * Ci + gi) * 9);
        float f[36];
#pragma unroll
        for (int u = 0; u < 9; ++u) {
          const float4 q = wp[u];
          f[4 * u] = q.x, f[4 * u + 1] = q.y, f[4 * u + 2] = q.z, f[4 * u + 3] = q.w;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
          for (int u = 0; u < 9; ++u) v[k][u] = f[9 * k + u];
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const bool in = go < Co && gi + k < Ci;
          const float* wp = w + (TRANS ? (size_t)(gi + k) * Co + go : (size_t)go * Ci + gi + k) * 9;
#pragma unroll
          for (int u = 0; u < 9; ++u) v[k][u] = in ? wp[TRANS ? 8 - u : u] : 0.0f;
        }
      }
      unsigned char* d = sw + (k4 >> 2) * 9 * C::W_BLOCK + ((k4 >> 1) & 1) * (C::N * 16) + o * 16 + (k4 & 1) * 8;
#pragma unroll
      for (int u = 0; u < 9; ++u)
#pragma unroll
        for (int term = 0; term < 3; ++term) {
          uint16_t h[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            h[k] = umma::bf16_bits(v[k][u]);
            const float t = umma::bf16_value(h[k]);
            if (term == 0) bad |= !(fabsf(t) < INFINITY);
            v[k][u] -= t;
          }
          *reinterpret_cast<uint2*>(d + u * C::W_BLOCK + term * (C::CO * 16)) =
              make_uint2(h[0] | ((uint32_t)h[1] << 16), h[2] | ((uint32_t)h[3] << 16));
        }
    }
    fence_async_shared();
    __syncthreads();
    if (tid == 0) {
      umma::fence_after_sync();
      constexpr uint32_t idesc = umma::idesc_bf16_f32(128, C::N);
      const uint32_t ax = smem_u32(sx), bw = smem_u32(sw);
      const int ks = min(C::CI / 16, (Ci - c0 + 15) / 16);
      for (int k = 0; k < ks; ++k)
        for (int tap = 0; tap < 9; ++tap) {
          const uint64_t bd = desc_plain(bw + (uint32_t)(k * 9 + tap) * C::W_BLOCK, C::N * 16, 128);
          const uint32_t a0 = ax + 2 * k * C::X_CHUNK + (uint32_t)((tap / 3) * C::PITCH + tap % 3 + 1) * 16;
#pragma unroll
          for (int mb = 0; mb < 2; ++mb)
            umma::mma_bf16(tmem + mb * 128, desc_plain(a0 + mb * 128, C::X_CHUNK, C::PITCH * 16), bd, idesc,
                           (s | k | tap) != 0 ? 1u : 0u);
        }
      umma::mma_commit(&bar);
    }
  }
  umma::wait_mma(&bar, par, &err);
  const bool slow = __syncthreads_or(bad || err);   // also: every MMA has read the tile
  bf16* so = reinterpret_cast<bf16*>(sm);           // [32 channels][16][16]
  {
    const int q = warp & 3, mb = warp >> 2, m = 32 * q + lane;
    const int px = (m >> 3) * C::T + (m & 7) + 8 * mb;
    float a[32], b[32];
    const uint32_t t0 = tmem + ((uint32_t)(32 * q) << 16) + mb * 128;
    umma::tmem_ld32(t0 + 64, a);
    umma::tmem_ld32(t0 + 32, b);
#pragma unroll
    for (int j = 0; j < 32; ++j) a[j] += b[j];
    umma::tmem_ld32(t0, b);
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const int o = o0 + j;
      float v = b[j] + a[j] + ((!TRANS && bias && o < Co) ? bias[o] : 0.f);
      if (RELU) v = fmaxf(v, 0.f);
      so[j * (C::T * C::T) + px] = __float2bfloat16_rn(v);
    }
  }
  if (slow) {
    // an infinity or a NaN among the inputs: the terms of a split would turn it into others (inf
    // times a zero term), so the tile is summed as written above
    __syncthreads();
    for (int e = tid; e < C::CO * C::T * C::T; e += C::THREADS) {
      const int o = o0 + e / (C::T * C::T), py = y0 + (e / C::T) % C::T, pxx = x0 + e % C::T;
      if (o >= Co) break;
      float v = 0.f;
      for (int i = 0; i < Ci; ++i)
        for (int tap = 0; tap < 9; ++tap) {
          const int yy = py + tap / 3 - 1, xx = pxx + tap % 3 - 1;
          const float wv = TRANS ? w[((size_t)i * Co + o) * 9 + (8 - tap)] : w[((size_t)o * Ci + i) * 9 + tap];
          const float xv = (yy >= 0 && yy < H && xx >= 0 && xx < Wd)
                               ? __bfloat162float(xn[(size_t)i * plane + (size_t)yy * Wd + xx]) : 0.f;
          v = fmaf(wv, xv, v);
        }
      if (!TRANS && bias) v += bias[o];
      if (RELU) v = fmaxf(v, 0.f);
      so[e] = __float2bfloat16_rn(v);
    }
  }
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tmem, 256);
  // rows of 16 pixels: two 16-byte words
  for (int e = tid; e < C::CO * C::T * 2; e += C::THREADS) {
    const int j = e / (C::T * 2), r = (e / 2) % C::T, h = e & 1;
    if (o0 + j >= Co) break;
    bf16* d = out + ((size_t)n * Co + o0 + j) * plane + (size_t)(y0 + r) * Wd + x0 + 8 * h;
    const uint4 v = *reinterpret_cast<const uint4*>(so + j * (C::T * C::T) + r * C::T + 8 * h);
    if (wide) {
      uint32_t* d2 = reinterpret_cast<uint32_t*>(d);
      d2[0] = v.x, d2[1] = v.y, d2[2] = v.z, d2[3] = v.w;
    } else {
      uint16_t* d1 = reinterpret_cast<uint16_t*>(d);
      const uint32_t p[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) d1[2 * k] = (uint16_t)p[k], d1[2 * k + 1] = (uint16_t)(p[k] >> 16);
    }
  }
}

// ------------------------------------------------------------------ weight gradient
// A CTA sums dw[o][i][t] = sum_p dy[o][p] x[i][p + off(t)] over its share of the pixel tiles (32 x 8
// pixels) for 128 output and 16 input channels: per row of taps one MMA with M = 128 (dy, zero rows
// beyond Co), N = 3 x 16 (the taps dx from three shifted copies of x), K = 16 pixels of a row; nine
// accumulators of 16 columns, drained every 128 pixels.
// part[blk][t][i][o], pbias[blk][o].
struct WgradCfg {
  static constexpr int THREADS = 256, TW = 32, TH = 8, CO = 128, CI = 16;
  static constexpr int GROUP = 4;   // rows between drains of the accumulators
  static constexpr int PITCH = TW + 4, ROWS = TH + 2;
  static constexpr uint32_t D_CHUNK = TW * TH * 16, D_BYTES = (CO / 8) * D_CHUNK;
  static constexpr uint32_t X_CHUNK = TW * ROWS * 16, X_BYTES = 3 * (CI / 8) * X_CHUNK;   // [dx][chunk]
  static constexpr uint32_t SMEM = D_BYTES + X_BYTES;
  static constexpr int N = 3 * CI, COLS = 3 * N, SHARE = COLS / (THREADS / 128);   // columns that a warp drains
};

__global__ void __launch_bounds__(WgradCfg::THREADS, 2)
    conv3x3_wgrad_mma_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ x, float* __restrict__ part,
                             float* __restrict__ pbias, int Ci, int Co, int H, int Wd, int N, int wide) {
  using C = WgradCfg;
  extern __shared__ __align__(128) unsigned char sm[];
  unsigned char *sd = sm, *sx = sm + C::D_BYTES;
  __shared__ uint64_t bar;
  __shared__ uint32_t tmem_s;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int o0 = blockIdx.y * C::CO, i0 = blockIdx.z * C::CI, blk = blockIdx.x, nblk = gridDim.x;
  const size_t plane = (size_t)H * Wd;
  if (tid == 0) {
    mbar_init(&bar, 1);
    fence_async_shared();
  }
  if (warp == 0) umma::tmem_alloc(&tmem_s, 256);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = tmem_s;
  uint32_t par = 0;
  int err = 0;
  const int q = warp & 3, share = warp >> 2;
  float acc[C::SHARE];
#pragma unroll
  for (int k = 0; k < C::SHARE; ++k) acc[k] = 0.f;
  float bs[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) bs[k] = 0.f;
  const int tiles_x = Wd / C::TW, tiles = (H / C::TH) * tiles_x;
  const long long total = (long long)tiles * N, per = (total + nblk - 1) / nblk;
  const int chunks = min(C::CO, Co - o0 + 7) / 8;   // the others stay zero
  for (uint32_t e = chunks * C::D_CHUNK / 16 + tid; e < C::D_BYTES / 16; e += C::THREADS)
    reinterpret_cast<uint4*>(sd)[e] = make_uint4(0u, 0u, 0u, 0u);
  const long long b0 = blk * per, b1 = b0 + per < total ? b0 + per : total;
  bool failed = false;   // a wait ran out in some thread: the whole share becomes NaN
  for (long long b = b0; b < b1 && !failed; ++b) {
    const int n = (int)(b / tiles), tile = (int)(b % tiles);
    const int y0 = (tile / tiles_x) * C::TH, x0 = (tile % tiles_x) * C::TW;
    // dy: 16 chunks of 8 channels x 256 pixels, a task is 8 channels x 2 pixels
    const bf16* dn = dy + (size_t)n * Co * plane + (size_t)y0 * Wd + x0;
    for (int e = tid; e < chunks * (C::TW * C::TH / 2); e += C::THREADS) {
      const int ch = e / (C::TW * C::TH / 2), pp = e % (C::TW * C::TH / 2);
      const int r = pp / (C::TW / 2), cp = pp % (C::TW / 2);
      uint32_t p[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int o = o0 + 8 * ch + k;
        p[k] = o < Co ? ld_pair(dn + (size_t)o * plane + (size_t)r * Wd + 2 * cp, wide != 0) : 0u;
      }
      uint4* d = reinterpret_cast<uint4*>(sd) + ch * (C::TW * C::TH) + r * C::TW + 2 * cp;
      d[0] = make_uint4(__byte_perm(p[0], p[1], 0x5410), __byte_perm(p[2], p[3], 0x5410),
                        __byte_perm(p[4], p[5], 0x5410), __byte_perm(p[6], p[7], 0x5410));
      d[1] = make_uint4(__byte_perm(p[0], p[1], 0x7632), __byte_perm(p[2], p[3], 0x7632),
                        __byte_perm(p[4], p[5], 0x7632), __byte_perm(p[6], p[7], 0x7632));
    }
    stage_tile<C::CI / 8, C::PITCH, C::ROWS, C::TW>(sx, x + (size_t)n * Ci * plane, i0, Ci, H, Wd, y0, x0, wide != 0,
                                                   C::THREADS);
    fence_async_shared();
    __syncthreads();
    if (i0 == 0) {   // bias: 16 threads per chunk, 16 pixels each
      const uint4* d = reinterpret_cast<const uint4*>(sd) + (tid >> 4) * (C::TW * C::TH) + (tid & 15);
      float t[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) t[k] = 0.f;
#pragma unroll 4
      for (int r = 0; r < 16; ++r) {
        const uint4 v = d[16 * r];
        const uint32_t p[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          t[2 * k] += umma::bf16_value((uint16_t)p[k]);
          t[2 * k + 1] += umma::bf16_value((uint16_t)(p[k] >> 16));
        }
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) bs[k] += t[k];
    }
    for (int g = 0; g < C::TH / C::GROUP && !failed; ++g) {
      if (tid == 0) {
        umma::fence_after_sync();
        constexpr uint32_t idesc = umma::idesc_bf16_f32(128, C::N) | (1u << 15) | (1u << 16);   // A, B MN-major
        const uint32_t da = smem_u32(sd), xa = smem_u32(sx);
        for (int k = 0; k < 2 * C::GROUP; ++k) {
          const int r = C::GROUP * g + (k >> 1), c = 16 * (k & 1);
          const uint64_t ad = desc_plain(da + (uint32_t)(r * C::TW + c) * 16, 128, C::D_CHUNK);
#pragma unroll
          for (int ty = 0; ty < 3; ++ty)
            umma::mma_bf16(tmem + ty * C::N, ad,
                           desc_plain(xa + (uint32_t)((r + ty) * C::TW + c) * 16, 128, C::X_CHUNK), idesc,
                           k > 0 ? 1u : 0u);
        }
        umma::mma_commit(&bar);
      }
      umma::wait_mma(&bar, par, &err);
      const uint32_t t0 = tmem + ((uint32_t)(32 * q) << 16) + share * C::SHARE;
      static_assert(C::SHARE == 72, "32 + 32 + 8 columns");
      float v[32], u[8];
#pragma unroll
      for (int c = 0; c < 64; c += 32) {
        umma::tmem_ld32(t0 + c, v);
#pragma unroll
        for (int k = 0; k < 32; ++k) acc[c + k] += v[k];
      }
      umma::tmem_ld8(t0 + 64, u);
#pragma unroll
      for (int k = 0; k < 8; ++k) acc[64 + k] += u[k];
      umma::fence_before_sync();
      // the accumulators are read (and, after the last group, the tile is)
      failed = __syncthreads_or(err);
      umma::fence_after_sync();
    }
  }
  if (failed) {   // once more, bounded, before TMEM goes
    uint32_t last = par ^ 1u;
    mbar_wait(&bar, last, nullptr);
  }
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tmem, 256);
  const int o = o0 + 32 * q + lane;
  if (o < Co) {
    float* pw = part + (size_t)blk * 9 * Ci * Co;
#pragma unroll
    for (int k = 0; k < C::SHARE; ++k) {
      const int col = share * C::SHARE + k, tap = col / C::CI, i = i0 + col % C::CI;
      if (i < Ci) pw[((size_t)tap * Ci + i) * Co + o] = failed ? NAN : acc[k];
    }
  }
  if (i0 == 0) {
    const int ch = tid >> 4;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
#pragma unroll
      for (int s = 8; s > 0; s >>= 1) bs[k] += __shfl_down_sync(0xffffffffu, bs[k], s, 16);
      if ((tid & 15) == 0 && o0 + 8 * ch + k < Co) pbias[(size_t)blk * Co + o0 + 8 * ch + k] = failed ? NAN : bs[k];
    }
  }
}

// sum of n values `stride` apart in a fixed order: eight running sums (loads in flight together,
// shorter chains of roundings), then pairwise
__device__ __forceinline__ float strided_sum(const float* __restrict__ p, int n, size_t stride) {
  float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  int b = 0;
  for (; b + 8 <= n; b += 8)
#pragma unroll
    for (int k = 0; k < 8; ++k) s[k] += p[(size_t)(b + k) * stride];
  for (; b < n; ++b) s[b & 7] += p[(size_t)b * stride];
  return ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7]));
}

// dw[o][i][t] = sum over blocks of part[blk][t][i][o], db[o] = sum of pbias[blk][o]
__global__ void wgrad_reduce_kernel(const float* __restrict__ part, const float* __restrict__ pbias,
                                    float* __restrict__ dw, float* __restrict__ db, int nblk, int Ci, int Co) {
  const int n = 9 * Ci * Co, e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n + Co) return;
  if (e < n) {
    const int o = e % Co, i = (e / Co) % Ci, t = e / (Co * Ci);
    dw[((size_t)o * Ci + i) * 9 + t] = strided_sum(part + e, nblk, n);
  } else {
    db[e - n] = strided_sum(pbias + e - n, nblk, Co);
  }
}

}  // namespace nn
}  // namespace pty
