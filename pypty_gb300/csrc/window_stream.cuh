// One-transform and band-limit passes over many 128-px windows with the next window's load under
// the current window's transform.
//
// A 128-px window fills an SM's registers, so a block per window loads, transforms and stores one
// after the other (object windows: 15 us each, 7.7 of them FFT arithmetic). Here a block walks a
// run of windows. While a window is transformed, asynchronous copies bring most of the next one
// (SE of a thread's 32 elements) into a side buffer; the rest follows into the warp's own part of
// the exchange buffer as soon as its last round has read it, under the register-only tail and the
// stores. All copies are a warp's own, 8 or 16 bytes per lane, so that no alignment beyond the
// element's is asked for and no barrier is added between warps. 64-px windows have four blocks on
// an SM, which overlap by themselves.
// 1536 windows, one transform: 99 -> 85 us (4.7 TB/s); 720 windows band-limited, object windows 74 ->
// 62 us, gradient windows of two contributions 92 -> 77 us. What is left is the FFT (7.7 of 12.4 us
// a window), the eight rows that a store in (y, x) order touches, and the copies' issue.
#pragma once
#include "ptycho_kernels.cuh"

namespace pty {

struct Stream128 {
  using G = Geo<128>;
  static constexpr int SE = 20;                 // elements of a thread in the side buffer
  static constexpr int SROW = 4 * SE + 4;       // float2 from row to row of a warp's side part, and
  static constexpr int TROW = 4 * (32 - SE) + 4;   // of its tail: 32 bytes off a multiple of 128, no bank conflicts
  static constexpr int SPART = 8 * SROW;        // float2 of a warp's side part
  static constexpr int NW = G::T / 32;
  static constexpr size_t side_off = Smem<128>::bytes;
  static constexpr size_t bytes = side_off + sizeof(float2) * SPART * NW;
  static_assert(8 * TROW <= WinFFT<128>::WPART && SE * 32 <= SPART && (SE / 2) * 64 <= SPART && SE % 4 == 0, "");

  float2 *xbuf, *tw1, *tw2;
  float2 *side, *tail;   // this warp's side part, and its part of the exchange buffer

  __device__ Stream128(unsigned char* smem, const float2* g_tw) {
    double* red;
    carve<128>(smem, xbuf, tw1, tw2, red);
    load_twiddles<128>(tw1, tw2, g_tw);
    const int w = threadIdx.x >> 5;
    side = reinterpret_cast<float2*>(smem + side_off) + w * SPART;
    tail = xbuf + w * WinFFT<128>::WPART;
  }

  static __device__ __forceinline__ void copy8(float2* dst, const float2* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
  }
  static __device__ __forceinline__ void copy16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
  }
  // this warp's copies have landed
  static __device__ __forceinline__ void wait() {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
  }

  // ---- windows in natural (y, x) order, rows `pitch` apart: the warp's rows are 16 g + warp, g < 8;
  // an access is 8 bytes of 16 lanes in two rows or, WIDE and where the rows start on 16 bytes, 16
  // bytes of 8 lanes in four (FFTs: 119 -> 91 us a call; object windows, half of which start between,
  // lose 12 %)
  template <int I0, int I1, bool WIDE>
  __device__ __forceinline__ void rows_issue(const float2* src, size_t pitch) const {
    const int lane = threadIdx.x & 31;
    constexpr int P = I0 == 0 ? SROW : TROW;
    float2* d = I0 == 0 ? side : tail;
    const float2* s = src + (size_t)(threadIdx.x >> 5) * pitch + 4 * I0;
    if (WIDE && ((reinterpret_cast<uintptr_t>(src) | (pitch * sizeof(float2))) & 15) == 0) {
      d += (lane >> 3) * P + 2 * (lane & 7);
      s += (size_t)(16 * (lane >> 3)) * pitch + 2 * (lane & 7);
#pragma unroll
      for (int g = 0; g < 8; g += 4)
#pragma unroll
        for (int c = 0; c < 4 * (I1 - I0); c += 16) copy16(d + g * P + c, s + (size_t)(16 * g) * pitch + c);
    } else {
      d += (lane >> 4) * P + (lane & 15);
      s += (size_t)(16 * (lane >> 4)) * pitch + (lane & 15);
#pragma unroll
      for (int g = 0; g < 8; g += 2)
#pragma unroll
        for (int c = 0; c < 4 * (I1 - I0); c += 16) copy8(d + g * P + c, s + (size_t)(16 * g) * pitch + c);
    }
  }
  template <bool WIDE>
  __device__ __forceinline__ void rows_side(const float2* src, size_t pitch) const {
    rows_issue<0, SE, WIDE>(src, pitch);
  }
  template <bool WIDE>
  __device__ __forceinline__ void rows_tail(const float2* src, size_t pitch) const {
    rows_issue<SE, 32, WIDE>(src, pitch);
  }
  __device__ __forceinline__ void rows_read(Win& v) const {
    const int lane = threadIdx.x & 31;
    const float2* s = side + (lane >> 2) * SROW + (lane & 3);
    const float2* u = tail + (lane >> 2) * TROW + (lane & 3);
#pragma unroll
    for (int i = 0; i < 32; ++i) wset(v, i, i < SE ? s[4 * i] : u[4 * (i - SE)]);
  }

  // ---- natural (ky, kx) order or, with H = 64, detector order (ky and kx offset by H): element i of
  // a warp is 32 neighbouring kx; an access is two elements, or 8 bytes per lane of one
  template <int H>
  static __device__ __forceinline__ int freq_at(int i) {   // of lane 0
    const int w = threadIdx.x >> 5;
    return (w >> 1) * 128 + (w & 1) * 32 + (((8 * ((i >> 1) & 15)) ^ H) * 128 + ((64 * (i & 1)) ^ H));
  }
  template <int I0, int I1, int H>
  __device__ __forceinline__ void freq_issue(const float2* src) const {
    const int lane = threadIdx.x & 31;
    float2* d = I0 == 0 ? side : tail;
    if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
      // element i, the even lanes' pairs below 16 and element i + 1 above
      const int odd = lane >> 4;
      d += 2 * lane;
#pragma unroll
      for (int i = I0; i < I1; i += 2)
        copy16(d + (i - I0) * 32, src + freq_at<H>(i) + (odd ? freq_at<H>(1) - freq_at<H>(0) : 0) + 2 * (lane & 15));
    } else {
      d += lane;
#pragma unroll
      for (int i = I0; i < I1; ++i) copy8(d + (i - I0) * 32, src + freq_at<H>(i) + lane);
    }
  }
  __device__ __forceinline__ void freq_read(Win& v, float scale) const {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < 32; ++i) wset(v, i, cscale(i < SE ? side[i * 32 + lane] : tail[(i - SE) * 32 + lane], scale));
  }

  // ---- native windows
  template <int J0, int J1>
  __device__ __forceinline__ void native_issue(const float2* src) const {
    const float4* s = reinterpret_cast<const float4*>(src) + nword(0, threadIdx.x);
    float4* d = reinterpret_cast<float4*>(J0 == 0 ? side : tail) + (threadIdx.x & 31);
#pragma unroll
    for (int j = J0; j < J1; ++j) copy16(d + (j - J0) * 32, s + j * 32);
  }
  __device__ __forceinline__ void native_read(Win& v) const {
    const float4* s = reinterpret_cast<const float4*>(side) + (threadIdx.x & 31);
    const float4* u = reinterpret_cast<const float4*>(tail) + (threadIdx.x & 31);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const float4 q = j < SE / 2 ? s[j * 32] : u[(j - SE / 2) * 32];
      v.re[j] = make_float2(q.x, q.y);
      v.im[j] = make_float2(q.z, q.w);
    }
  }
};

// fft2 / ifft2 / shift_fft2 / ifft2_ishift (fft2_batch_kernel): windows [blockIdx * run, ...) of n
template <int INV, int H>
__global__ void __launch_bounds__(512) fft2_stream_kernel(const float2* in, float2* out, int n, int run,
                                                          const float2* __restrict__ g_tw) {
  using G = Geo<128>;
  extern __shared__ __align__(16) unsigned char smem[];
  const Stream128 s(smem, g_tw);
  const int t = threadIdx.x;
  const int w0 = blockIdx.x * run, w1 = min(w0 + run, n);
  constexpr size_t WW = 128 * 128;
  const float2* src = in + (size_t)w0 * WW;
  float2* dst = out + (size_t)w0 * WW + (INV ? G::ry(t) * 128 + G::rx(t, 0) : t & 31);
  auto side = [&]() {
    if constexpr (INV) s.freq_issue<0, Stream128::SE, H>(src);
    else s.rows_side<true>(src, 128);
  };
  auto tail = [&]() {
    if constexpr (INV) s.freq_issue<Stream128::SE, 32, H>(src);
    else s.rows_tail<true>(src, 128);
  };
  side();
  tail();
  for (int w = w0; w < w1; ++w, dst += WW) {
    const bool more = w + 1 < w1;
    src += WW;
    Win v;
    Stream128::wait();
    if constexpr (INV) s.freq_read(v, 1.0f / (float)WW);
    else s.rows_read(v);
    // the first window: the twiddles; inverse: every warp has read its part of the exchange buffer
    if (INV || w == w0) __syncthreads();
    else __syncwarp();
    if (more) side();
    if constexpr (INV) {
      WinFFT<128>::inverse_head(v, s.xbuf, s.tw1, s.tw2);
      __syncwarp();
      if (more) tail();
      WinFFT<128>::inverse_tail(v);
#pragma unroll
      for (int i = 0; i < 32; ++i) dst[4 * i] = wget(v, i);
    } else {
      WinFFT<128>::forward(v, s.xbuf, s.tw1, s.tw2);
      __syncthreads();   // the exchange buffer has been read
      if (more) tail();
#pragma unroll
      for (int i = 0; i < 32; ++i) dst[Stream128::freq_at<H>(i)] = wget(v, i);
    }
  }
}

// object_windows_kernel for windows [blockIdx * run, ...) of n
static __global__ void __launch_bounds__(512) object_windows_stream_kernel(WindowArgs a, int n, int run) {
  extern __shared__ __align__(16) unsigned char smem[];
  const Stream128 s(smem, a.tw);
  const int w0 = blockIdx.x * run, w1 = min(w0 + run, n);
  auto source = [&](int win) {
    const int b = win / a.zm, k = win % a.zm;
    const int gi = a.seq[b];
    return a.obj + ((size_t)k * a.Ny + a.pos[2 * gi]) * a.Nx + a.pos[2 * gi + 1];
  };
  {
    const float2* src = source(w0);
    s.rows_side<false>(src, a.Nx);
    s.rows_tail<false>(src, a.Nx);
  }
  for (int w = w0; w < w1; ++w) {
    const bool more = w + 1 < w1;
    const float2* next = source(more ? w + 1 : w);
    Win v;
    Stream128::wait();
    s.rows_read(v);
    if (w == w0) __syncthreads();
    else __syncwarp();
    if (more) s.rows_side<false>(next, a.Nx);
    WinFFT<128>::forward(v, s.xbuf, s.tw1, s.tw2);
    mul_real_table<128>(v, a.mask_sc);
    WinFFT<128>::inverse_head(v, s.xbuf, s.tw1, s.tw2);
    __syncwarp();
    if (more) s.rows_tail<false>(next, a.Nx);
    WinFFT<128>::inverse_tail(v);
    st_native(a.out + (size_t)w * 128 * 128, v);
  }
}

// grad_windows_kernel for windows [blockIdx * run, ...) of n. The first contribution comes through the
// copies, the others from L2, where one lane of each warp asked for them during the last transform.
static __global__ void __launch_bounds__(512) grad_windows_stream_kernel(float2* buf, const float* __restrict__ mask_sc,
                                                                         const float2* __restrict__ g_tw, int nsum,
                                                                         int n, int run) {
  using G = Geo<128>;
  extern __shared__ __align__(16) unsigned char smem[];
  const Stream128 s(smem, g_tw);
  const int t = threadIdx.x;
  constexpr size_t WW = 128 * 128;
  const int w0 = blockIdx.x * run, w1 = min(w0 + run, n);
  float2* win = buf + (size_t)w0 * nsum * WW;
  s.native_issue<0, Stream128::SE / 2>(win);
  s.native_issue<Stream128::SE / 2, 16>(win);
  for (int w = w0; w < w1; ++w, win += nsum * WW) {
    const bool more = w + 1 < w1;
    const float2* next = win + nsum * WW;
    Win v;
    Stream128::wait();
    s.native_read(v);
    for (int p = 1; p < nsum; ++p) {
      const float4* src = reinterpret_cast<const float4*>(win + p * WW) + nword(0, t);
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float4 q = src[j * 32];
        v.re[j] = padd(v.re[j], make_float2(q.x, q.y));
        v.im[j] = padd(v.im[j], make_float2(q.z, q.w));
      }
    }
    if (w == w0) __syncthreads();
    else __syncwarp();
    if (more) {
      s.native_issue<0, Stream128::SE / 2>(next);
      if ((t & 31) < nsum - 1) {
        const float2* q = next + (size_t)(1 + (t & 31)) * WW + (t >> 5) * 1024;   // this warp's share, 8 KB
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(q), "r"(8192) : "memory");
      }
    }
    WinFFT<128>::forward(v, s.xbuf, s.tw1, s.tw2);
    mul_real_table<128>(v, mask_sc);
    WinFFT<128>::inverse_head(v, s.xbuf, s.tw1, s.tw2);
    __syncwarp();
    if (more) s.native_issue<Stream128::SE / 2, 16>(next);
    WinFFT<128>::inverse_tail(v);
    // every read of this window's first contribution finished before forward()'s barrier
#pragma unroll
    for (int i = 0; i < 32; ++i) win[G::ry(t) * 128 + G::rx(t, i)] = wget(v, i);
  }
}

}  // namespace pty
