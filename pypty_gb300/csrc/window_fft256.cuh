// 256 x 256 window FFT over a thread-block cluster of 4 blocks (512 threads each).
//
// Block c = (cy, cx) = (c >> 1, c & 1) owns, in real space, the polyphase component
// x[2y' + cy, 2x' + cx] (y', x' < 128) and, in frequency, the quadrant
// X[ky' + 128 cy, kx' + 128 cx]. A forward transform is
//   1. the register-resident 128 x 128 FFT of the block's component (WinFFT<128>),
//   2. the twiddle w_256^(ky' cy + kx' cx),
//   3. a radix-2 x 2 butterfly across the four blocks through distributed shared memory:
//      X_q = sum_r (-1)^(qy ry + qx rx) T_r  (block q keeps quadrant q), one exchange in
//      which every block publishes its values and forms a quarter of everyone's results;
// the inverse runs the same steps backwards with conjugate twiddles (unnormalised).
// Each block's part of a window is stored in the 128 native order (window_fft.cuh) at
// offset c * 128^2 of the window.
#pragma once
#include <cooperative_groups.h>

#include "window_fft.cuh"

namespace pty {

namespace cg256 = cooperative_groups;

struct Geo256 {
  using G = Geo<128>;
  static constexpr int W = 256;
  static constexpr int H = 128;
  static constexpr int T = G::T;                  // 512 threads per block
  static constexpr size_t PART = (size_t)H * H;    // elements per block
  static __device__ __forceinline__ int ry(int c, int t) { return 2 * G::ry(t) + (c >> 1); }
  static __device__ __forceinline__ int rx(int c, int t, int i) { return 2 * G::rx(t, i) + (c & 1); }
  static __device__ __forceinline__ int fky(int c, int t, int i) { return G::fky(t, i) + H * (c >> 1); }
  static __device__ __forceinline__ int fkx(int c, int t, int i) { return G::fkx(t, i) + H * (c & 1); }
};

// tw256[k] = exp(-2 pi i k / 256) into shared memory (256 entries)
__device__ __forceinline__ void load_tw256(float2* tw256) {
  for (int k = threadIdx.x; k < 256; k += blockDim.x) {
    float s, c;
    sincospif((float)k / 128.0f, &s, &c);   // exact argument: k/128 is dyadic
    tw256[k] = make_float2(c, -s);
  }
}

// shared::cluster address of `p` (this block's shared memory) in block `rank` of the cluster
__device__ __forceinline__ uint32_t cluster_map(const void* p, int rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
  return r;
}

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}

__device__ __forceinline__ void st_cluster_f4(uint32_t addr, float4 v) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
               : "memory");
}

struct WinFFT256 {
  using G = Geo<128>;
  static constexpr int T = G::T;

  // One exchange across the cluster: every block stores its 16 packs (16-byte words) into its own
  // exchange buffer; block `me` takes the packs 4 me .. 4 me + 3 of all four, op(j, re, im) turns the
  // four blocks' values of pack j into the four blocks' results, and these go back to where the values
  // were. Bound by distributed shared memory: 96 KB read and 96 KB written per block, where pulling the
  // partners' whole buffers (and every block forming its own results from them) moves 384 KB: 30.8k of a
  // propagation step's 69.5k cycles, now 18.5k of 56.0k (280 positions, 5 modes, 24 slices, every 8th wave
  // kept: 99.3 -> 81.6 ms; 384 transforms 992 -> 878 us).
  template <typename Op>
  static __device__ __forceinline__ void exchange(Win& v, float2* xbuf, cg256::cluster_group& cl, int me, Op&& op) {
    const int t = threadIdx.x;
    __syncthreads();   // this block's own transform has finished reading xbuf
    float4* p = reinterpret_cast<float4*>(xbuf);
#pragma unroll
    for (int j = 0; j < 16; ++j) p[j * T + t] = pack4(v.re[j], v.im[j]);
    cl.sync();   // every block's values are published
    uint32_t a[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) a[r] = cluster_map(p + 4 * me * T + t, r);
    float4 q[4][4];   // all loads before the first store
#pragma unroll
    for (int jj = 0; jj < 4; ++jj)
#pragma unroll
      for (int r = 0; r < 4; ++r) q[jj][r] = ld_cluster_f4(a[r] + jj * T * 16);
#pragma unroll
    for (int jj = 0; jj < 4; ++jj) {
      float2 re[4], im[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        re[r] = make_float2(q[jj][r].x, q[jj][r].y);
        im[r] = make_float2(q[jj][r].z, q[jj][r].w);
      }
      op(4 * me + jj, re, im);
#pragma unroll
      for (int r = 0; r < 4; ++r) st_cluster_f4(a[r] + jj * T * 16, pack4(re[r], im[r]));
    }
    cl.sync();   // every block's results are in place
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const float4 r = p[j * T + t];
      v.re[j] = make_float2(r.x, r.y);
      v.im[j] = make_float2(r.z, r.w);
    }
    __syncthreads();   // xbuf may be reused
  }

  // z_q = sum_r (-1)^(q_y r_y + q_x r_x) z_r
  static __device__ __forceinline__ void butterfly4(float2 (&z)[4]) {
    const float2 e0 = padd(z[0], z[1]), e1 = psub(z[0], z[1]), e2 = padd(z[2], z[3]), e3 = psub(z[2], z[3]);
    z[0] = padd(e0, e2);
    z[1] = padd(e1, e3);
    z[2] = psub(e0, e2);
    z[3] = psub(e1, e3);
  }

  // Radix-2 x 2 butterfly across the four blocks, block `me` keeping output quadrant `me`.
  static __device__ __forceinline__ void cross(Win& v, float2* xbuf, cg256::cluster_group& cl, int me) {
    exchange(v, xbuf, cl, me, [&](int, float2 (&re)[4], float2 (&im)[4]) {
      butterfly4(re);
      butterfly4(im);
    });
  }

  // v *= w_256^(ky cy + kx cx), or its conjugate; the second element of a pack is 64 further in
  // kx, where w_256^(64 cx) = (-i)^cx
  static __device__ __forceinline__ void twiddle(Win& v, const float2* tw256, int c, bool conj) {
    if (c == 0) return;
    const int t = threadIdx.x;
    const int cy = c >> 1, cx = c & 1;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const float2 w = tw256[G::fky(t, 2 * j) * cy + G::fkx(t, 2 * j) * cx];
      const float2 wx = make_float2(w.x, cx ? w.y : w.x);
      const float2 wy = make_float2(w.y, cx ? -w.x : w.y), ny = pneg(wy);
      pcmul(v.re[j], v.im[j], wx, conj ? ny : wy, conj ? wy : ny);
    }
  }

  static __device__ __forceinline__ void forward(Win& v, float2* xbuf, const float2* tw1, const float2* tw2,
                                                 const float2* tw256, cg256::cluster_group& cl) {
    const int c = (int)cl.block_rank();
    WinFFT<128>::forward(v, xbuf, tw1, tw2);
    twiddle(v, tw256, c, false);
    cross(v, xbuf, cl, c);
  }

  static __device__ __forceinline__ void inverse(Win& v, float2* xbuf, const float2* tw1, const float2* tw2,
                                                 const float2* tw256, cg256::cluster_group& cl) {
    const int c = (int)cl.block_rank();
    cross(v, xbuf, cl, c);
    twiddle(v, tw256, c, true);
    WinFFT<128>::inverse(v, xbuf, tw1, tw2);
  }

  // The middle of one propagation step x -> IFFT(FFT(x) * P) (conj(P) in the adjoint): the
  // forward cross butterfly, the multiply and the inverse cross butterfly in one exchange, between
  // the twiddled forward sub-transform and the conjugate twiddle of the inverse. mul(j, zr, zi)
  // multiplies pack j's four quadrants by the propagator at (ky + 128 q_y, kx + 128 q_x).
  template <typename Mul>
  static __device__ __forceinline__ void cross_propagate(Win& v, float2* xbuf, cg256::cluster_group& cl, int me,
                                                         Mul&& mul) {
    exchange(v, xbuf, cl, me, [&](int j, float2 (&zr)[4], float2 (&zi)[4]) {
      butterfly4(zr);
      butterfly4(zi);
      mul(j, zr, zi);
      butterfly4(zr);
      butterfly4(zi);
    });
  }

  // z_q *= P_q (conj: conj(P_q)) for the propagator table P (256 x 256, natural order)
  static __device__ __forceinline__ void mul_quadrants(int t, int j, float2 (&zr)[4], float2 (&zi)[4],
                                                       const float2* __restrict__ P, bool conj) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float2* m = P + (G::fky(t, 2 * j) + 128 * (q >> 1)) * 256 + G::fkx(t, 2 * j) + 128 * (q & 1);
      const float2 a = m[0], b = m[64];
      const float2 py = conj ? make_float2(-a.y, -b.y) : make_float2(a.y, b.y);
      pcmul(zr[q], zi[q], make_float2(a.x, b.x), py, pneg(py));
    }
  }

  // x -> IFFT(FFT(x) * m) for a real multiplier m (256 x 256, unshifted frequency order)
  static __device__ __forceinline__ void band_limit(Win& v, float2* xbuf, const float2* tw1, const float2* tw2,
                                                    const float2* tw256, cg256::cluster_group& cl,
                                                    const float* __restrict__ m) {
    const int c = (int)cl.block_rank();
    const int t = threadIdx.x;
    WinFFT<128>::forward(v, xbuf, tw1, tw2);
    twiddle(v, tw256, c, false);
    cross_propagate(v, xbuf, cl, c, [&](int j, float2 (&zr)[4], float2 (&zi)[4]) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float* w = m + (G::fky(t, 2 * j) + 128 * (q >> 1)) * 256 + G::fkx(t, 2 * j) + 128 * (q & 1);
        const float2 mk = make_float2(w[0], w[64]);
        zr[q] = pmul(zr[q], mk);
        zi[q] = pmul(zi[q], mk);
      }
    });
    twiddle(v, tw256, c, true);
    WinFFT<128>::inverse(v, xbuf, tw1, tw2);
  }

  // x <- IFFT(FFT(x) * P * scale) (conj: conj(P)) for a (256, 256) table P in natural (ky, kx)
  // order, in the same single folded exchange
  static __device__ __forceinline__ void propagate(Win& v, float2* xbuf, const float2* tw1, const float2* tw2,
                                                   const float2* tw256, cg256::cluster_group& cl,
                                                   const float2* __restrict__ P, bool conj, float scale) {
    const int c = (int)cl.block_rank();
    const int t = threadIdx.x;
    WinFFT<128>::forward(v, xbuf, tw1, tw2);
    twiddle(v, tw256, c, false);
    cross_propagate(v, xbuf, cl, c, [&](int j, float2 (&zr)[4], float2 (&zi)[4]) {
      mul_quadrants(t, j, zr, zi, P, conj);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        zr[q] = pmul(zr[q], pdup(scale));
        zi[q] = pmul(zi[q], pdup(scale));
      }
    });
    twiddle(v, tw256, c, true);
    WinFFT<128>::inverse(v, xbuf, tw1, tw2);
  }
};

}  // namespace pty
