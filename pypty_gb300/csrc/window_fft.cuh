// Register-resident 2D FFT of one W x W probe window per thread block (W = 64 or 128).
//
// Every thread owns 32 complex values. A 2D transform is three register rounds separated
// by two exchanges through shared memory:
//
//   round 1  lane (m1, n2) of warp m2, n2 < A=W/32: 32-point DFT along x over x = A*n1 + n2
//            of row y = Bq*m1 + m2
//   round 2  lane k1 of warp m2 < Bq : twiddle w_W^(k1*n2), A-point DFT over n2 (finishes
//            kx = k1 + 32*k2), C-point DFT along y over y = Bq*m1 + m2, twiddle w_W^(j1*m2)
//   round 3  thread (j1, g), g < S3  : Bq-point DFT over m2 (finishes ky = j1 + C*j2),
//            the thread holds kx = g + S3*q
//
// with C = 32/A and Bq = W/C (the number of warps). The forward transform runs rounds 1-2-3 and
// leaves the spectrum in the "frequency layout"; the inverse runs 3-2-1 with conjugate twiddles
// and leaves the window in the "real layout" (round-1 ownership). Element-wise work (object
// slice, propagator, masks, loss) happens directly in those layouts, so a multislice step
// is FFT -> multiply -> IFFT without any extra data movement.
//
// Synchronisation. Warp m2 owns the rows y = m2 (mod Bq) in round 1 and the residue m2 in round
// 2, so the exchange between rounds 1 and 2 is a 32 x 32 transpose inside each warp, through the
// warp's own 8 KB part of the exchange buffer, ordered by __syncwarp alone. In the exchange
// between rounds 2 and 3 a warp stores only to its own part as well (rows m2*C + j1 of the
// buffer); what crosses warps are round 3's loads, and the inverse's round 3 stores to the very
// addresses that its thread loaded. So one FFT -> multiply -> IFFT step has two block barriers
// (before the forward's cross-warp loads and after the inverse's cross-warp stores); outside
// them each warp runs on its own, and its operand waits, stores and barriers of one warp overlap
// the arithmetic of the others. A thread's stores in the forward's first exchange go where only
// it has loaded since the last block barrier, so a transform may follow another without a
// barrier; code that uses the buffer otherwise in between puts a block barrier before the next
// transform.
//
// Packed arithmetic. The window is held as 16 packs of two values, real and imaginary parts
// apart (struct Win), and nearly all of the arithmetic is two-wide (add/mul/fma.f32x2): a packed
// instruction does two lanes' work in one issue slot. The two halves of a pack go through the same
// butterflies: round 1 packs the even and odd x of a 16-point DFT each (a scalar radix-2 stage
// joins them; the inverse the even and odd k), round 2 packs
// neighbouring n2, round 3 packs kx and kx + W/2. The exchanges store 16-byte words of real and
// imaginary packs, so that loads give packs without register moves.
//
// Shared-memory exchanges are free of bank conflicts for both W: the transpose inside a warp
// keeps real and imaginary parts in two planes of 32 rows (k1) x 8 words of 16 bytes, words
// XOR-swizzled by k1; the cross-warp exchange has rows of W/2 words read and written
// contiguously.
//
// What bounds it: the FP32 pipe and shared-memory bandwidth by turns (about 1300 FP32 lane
// operations per thread and 256 wavefronts per warp for a 128 x 128 transform, each close to half
// of the measured time, and with one window per SM the two overlap only where warps run apart).
// Against scalar arithmetic with four block barriers per transform: 1500 128-px windows,
// transform and store, 118 -> 105 us; a 256-px 24-slice call 120 -> 100 ms; the fused 128-px
// kernel executes 21 % fewer instructions (524 M -> 416 M per 192 blocks).
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <type_traits>

namespace pty {

// ------------------------------------------------------------------ complex helpers
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// a * conj(b)
__device__ __forceinline__ float2 cmulc(float2 a, float2 b) {
  return make_float2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
__device__ __forceinline__ float2 cconj(float2 a) { return make_float2(a.x, -a.y); }
__device__ __forceinline__ float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }
__device__ __forceinline__ float cabs2(float2 a) { return a.x * a.x + a.y * a.y; }

// compile-time loop
template <int I, int N, typename F>
__device__ __forceinline__ void static_for(F&& f) {
  if constexpr (I < N) {
    f(std::integral_constant<int, I>{});
    static_for<I + 1, N>(f);
  }
}

// cos / sin of 2*pi*m/32, m in [0, 32)
__host__ __device__ constexpr float kcos32(int m) {
  constexpr float t[32] = {
      1.000000000e+00f, 9.807852507e-01f, 9.238795042e-01f, 8.314695954e-01f,
      7.071067691e-01f, 5.555702448e-01f, 3.826834261e-01f, 1.950903237e-01f,
      0.0f, -1.950903237e-01f, -3.826834261e-01f, -5.555702448e-01f,
      -7.071067691e-01f, -8.314695954e-01f, -9.238795042e-01f, -9.807852507e-01f,
      -1.000000000e+00f, -9.807852507e-01f, -9.238795042e-01f, -8.314695954e-01f,
      -7.071067691e-01f, -5.555702448e-01f, -3.826834261e-01f, -1.950903237e-01f,
      0.0f, 1.950903237e-01f, 3.826834261e-01f, 5.555702448e-01f,
      7.071067691e-01f, 8.314695954e-01f, 9.238795042e-01f, 9.807852507e-01f};
  return t[m];
}
__host__ __device__ constexpr float ksin32(int m) { return kcos32((m + 24) & 31); }

// a * exp(SIGN * 2*pi*i * E / N) with E, N compile-time (N divides 32)
template <int N, int E, int SIGN>
__device__ __forceinline__ float2 tw(float2 a) {
  static_assert(32 % N == 0, "twiddle table covers N | 32");
  constexpr int m = ((E % N) * (32 / N)) & 31;
  if constexpr (m == 0) {
    return a;
  } else if constexpr (m == 16) {
    return make_float2(-a.x, -a.y);
  } else if constexpr (m == 8) {          // exp(SIGN * i*pi/2) = SIGN * i
    return SIGN > 0 ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
  } else if constexpr (m == 24) {         // exp(SIGN * i*3pi/2) = -SIGN * i
    return SIGN > 0 ? make_float2(a.y, -a.x) : make_float2(-a.y, a.x);
  } else if constexpr (m % 4 == 0) {      // odd multiples of pi/4
    constexpr float h = 7.071067691e-01f;
    constexpr float c = kcos32(m) > 0 ? h : -h;
    constexpr float s = (SIGN > 0 ? 1.0f : -1.0f) * (ksin32(m) > 0 ? h : -h);
    // (a.x + i a.y)(c + i s) with |c| = |s| = h
    constexpr float sc = (c > 0) == (s > 0) ? 1.0f : -1.0f;   // s = sc * c
    float u = a.x - sc * a.y;   // a.x - a.y*s/c
    float w = a.y + sc * a.x;   // a.y + a.x*s/c
    return make_float2(u * c, w * c);
  } else {
    constexpr float c = kcos32(m);
    constexpr float s = (SIGN > 0 ? 1.0f : -1.0f) * ksin32(m);
    return make_float2(a.x * c - a.y * s, a.x * s + a.y * c);
  }
}

// 4-point DFT butterfly: (t0..t3) -> X_q = sum_r t_r * exp(SIGN*2*pi*i*r*q/4)
template <int SIGN>
__device__ __forceinline__ void bfly4(float2& t0, float2& t1, float2& t2, float2& t3) {
  float2 u0 = cadd(t0, t2), u1 = csub(t0, t2), u2 = cadd(t1, t3), d = csub(t1, t3);
  // u3 = d * (SIGN * i)
  float2 u3 = SIGN > 0 ? make_float2(-d.y, d.x) : make_float2(d.y, -d.x);
  t0 = cadd(u0, u2);
  t2 = csub(u0, u2);
  t1 = cadd(u1, u3);
  t3 = csub(u1, u3);
}

// In-register DFT of the N values v[OFF + STRIDE*i], i < N, written back in natural order.
// Radix-4 decimation in time, radix-2 for the last factor of 2.
template <int N, int SIGN>
struct DFT {
  template <int LEN, int STRIDE, int OFF>
  static __device__ __forceinline__ void run(float2 (&v)[LEN]) {
    if constexpr (N == 1) {
    } else if constexpr (N == 2) {
      float2 a = v[OFF], b = v[OFF + STRIDE];
      v[OFF] = cadd(a, b);
      v[OFF + STRIDE] = csub(a, b);
    } else if constexpr (N == 4) {
      bfly4<SIGN>(v[OFF], v[OFF + STRIDE], v[OFF + 2 * STRIDE], v[OFF + 3 * STRIDE]);
    } else {
      constexpr int M = N / 4;
      DFT<M, SIGN>::template run<LEN, 4 * STRIDE, OFF>(v);
      DFT<M, SIGN>::template run<LEN, 4 * STRIDE, OFF + STRIDE>(v);
      DFT<M, SIGN>::template run<LEN, 4 * STRIDE, OFF + 2 * STRIDE>(v);
      DFT<M, SIGN>::template run<LEN, 4 * STRIDE, OFF + 3 * STRIDE>(v);
      float2 out[N];
      static_for<0, M>([&](auto KK) {
        constexpr int k = decltype(KK)::value;
        float2 t0 = v[OFF + STRIDE * (4 * k)];
        float2 t1 = tw<N, 1 * k, SIGN>(v[OFF + STRIDE * (4 * k + 1)]);
        float2 t2 = tw<N, 2 * k, SIGN>(v[OFF + STRIDE * (4 * k + 2)]);
        float2 t3 = tw<N, 3 * k, SIGN>(v[OFF + STRIDE * (4 * k + 3)]);
        bfly4<SIGN>(t0, t1, t2, t3);
        out[k] = t0;
        out[k + M] = t1;
        out[k + 2 * M] = t2;
        out[k + 3 * M] = t3;
      });
#pragma unroll
      for (int i = 0; i < N; ++i) v[OFF + STRIDE * i] = out[i];
    }
  }
};

// ------------------------------------------------------------------ window geometry
template <int W>
struct Geo {
  static_assert(W == 64 || W == 128, "window FFT supports W = 64 and 128");
  static constexpr int E = 32;             // complex values per thread
  static constexpr int T = W * W / E;      // threads per window
  static constexpr int A = W / 32;         // x sub-factor owned by round-1 threads
  static constexpr int C = 32 / A;         // y factor done in round 2
  static constexpr int Bq = W / C;         // y factor done in round 3
  static constexpr int Q = 32 / Bq;        // kx values per round-3 thread
  static constexpr int S3 = W / Q;         // kx stride in round 3
  static constexpr int TW1 = A * 32;       // round-1 twiddle table size
  static constexpr int TW2 = W;            // round-2 twiddle table size
  static constexpr int XBUF = W * W;       // exchange buffer (float2)
  // minimum blocks per SM of the kernels' launch bounds: at 64 px a cap of 128 registers a thread (four
  // blocks of the FFT passes fit; the fused kernel's shared memory lets three in)
  static constexpr int MINB = W == 64 ? 4 : 1;

  // real layout: element i of thread t is pixel (y, x)
  static __device__ __forceinline__ int ry(int t) { return Bq * ((t % 32) / A) + t / 32; }
  static __device__ __forceinline__ int rx(int t, int i) { return A * i + (t % A); }
  // frequency layout: element i of thread t is frequency (ky, kx) (unshifted FFT index); the
  // elements 2p and 2p + 1 of a pack are W/2 apart in kx
  static __device__ __forceinline__ int fky(int t, int i) { return (t / S3) + C * ((i >> 1) % Bq); }
  static __device__ __forceinline__ int fkx(int t, int i) {
    return (t % S3) + S3 * ((i >> 1) / Bq) + (W / 2) * (i & 1);
  }
};

// ------------------------------------------------------------------ packed pairs
// Two-wide FP32 arithmetic on the halves of a float2 (one issue slot per instruction).
__device__ __forceinline__ float2 padd(float2 a, float2 b) {
  float2 d;
  asm("{.reg .b64 ra, rb, rd; mov.b64 ra, {%2, %3}; mov.b64 rb, {%4, %5}; add.rn.f32x2 rd, ra, rb; mov.b64 {%0, %1}, rd;}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 psub(float2 a, float2 b) {
  float2 d;
  asm("{.reg .b64 ra, rb, rd; mov.b64 ra, {%2, %3}; mov.b64 rb, {%4, %5}; sub.rn.f32x2 rd, ra, rb; mov.b64 {%0, %1}, rd;}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 pmul(float2 a, float2 b) {
  float2 d;
  asm("{.reg .b64 ra, rb, rd; mov.b64 ra, {%2, %3}; mov.b64 rb, {%4, %5}; mul.rn.f32x2 rd, ra, rb; mov.b64 {%0, %1}, rd;}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 pfma(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{.reg .b64 ra, rb, rc, rd; mov.b64 ra, {%2, %3}; mov.b64 rb, {%4, %5}; mov.b64 rc, {%6, %7}; "
      "fma.rn.f32x2 rd, ra, rb, rc; mov.b64 {%0, %1}, rd;}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 pneg(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 pdup(float a) { return make_float2(a, a); }

// (re, im) *= w for packs; nwy = -w_y, so that both products fuse
__device__ __forceinline__ void pcmul(float2& re, float2& im, float2 wx, float2 wy, float2 nwy) {
  const float2 r = pfma(im, nwy, pmul(re, wx));
  im = pfma(re, wy, pmul(im, wx));
  re = r;
}

// A window's 32 values of one thread: pack p holds elements 2p and 2p + 1, real parts and
// imaginary parts apart.
struct Win {
  float2 re[16], im[16];
};
__device__ __forceinline__ float2 wget(const Win& v, int i) {
  return (i & 1) ? make_float2(v.re[i >> 1].y, v.im[i >> 1].y) : make_float2(v.re[i >> 1].x, v.im[i >> 1].x);
}
__device__ __forceinline__ void wset(Win& v, int i, float2 a) {
  if (i & 1) {
    v.re[i >> 1].y = a.x;
    v.im[i >> 1].y = a.y;
  } else {
    v.re[i >> 1].x = a.x;
    v.im[i >> 1].x = a.y;
  }
}

// In-register DFTs of packs: both halves transform alike. Radix 4 as DFT<N, SIGN> above, with
// the values re/im[OFF + STRIDE*i], i < N, written back in natural order.
template <int N, int E, int SIGN>
__device__ __forceinline__ void ptw(float2& re, float2& im) {
  static_assert(32 % N == 0, "twiddle table covers N | 32");
  constexpr int m = ((E % N) * (32 / N)) & 31;
  if constexpr (m == 0) {
  } else if constexpr (m == 8 || m == 24) {   // +-i
    constexpr bool plus = (m == 8) == (SIGN > 0);
    const float2 r = re;
    re = plus ? pneg(im) : im;
    im = plus ? r : pneg(r);
  } else if constexpr (m == 16) {
    re = pneg(re);
    im = pneg(im);
  } else if constexpr (m % 4 == 0) {          // odd multiples of pi/4
    constexpr float h = 7.071067691e-01f;
    constexpr float c = kcos32(m) > 0 ? h : -h;
    constexpr float s = (SIGN > 0 ? 1.0f : -1.0f) * (ksin32(m) > 0 ? h : -h);
    constexpr bool same = (c > 0) == (s > 0);
    const float2 u = same ? psub(re, im) : padd(re, im);
    const float2 w = same ? padd(im, re) : psub(im, re);
    re = pmul(u, pdup(c));
    im = pmul(w, pdup(c));
  } else {
    constexpr float c = kcos32(m);
    constexpr float s = (SIGN > 0 ? 1.0f : -1.0f) * ksin32(m);
    pcmul(re, im, pdup(c), pdup(s), pdup(-s));
  }
}

// one and two-wide FP32 under the same names
__device__ __forceinline__ float vadd(float a, float b) { return a + b; }
__device__ __forceinline__ float vsub(float a, float b) { return a - b; }
__device__ __forceinline__ float vfma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ float2 vadd(float2 a, float2 b) { return padd(a, b); }
__device__ __forceinline__ float2 vsub(float2 a, float2 b) { return psub(a, b); }
__device__ __forceinline__ float2 vfma(float2 a, float b, float2 c) { return pfma(a, pdup(b), c); }

// (s, d) = (a + w b, a - w b), w = exp(SIGN * 2 pi i E / N): the twiddle's products fuse with the
// butterfly's adds, one rounding less than multiplying first, for the same number of instructions
// (two fewer at odd multiples of pi/4)
template <int N, int E, int SIGN, typename V>
__device__ __forceinline__ void add_sub_tw(V ar, V ai, V br, V bi, V& sr, V& si, V& dr, V& di) {
  constexpr int m = ((E % N) * (32 / N)) & 31;
  if constexpr (m % 8 == 0) {                 // w = 1, +-i, -1
    constexpr bool swap = m % 16 == 8;
    constexpr bool neg_r = swap ? ((m == 8) == (SIGN > 0)) : m == 16;      // w b = (-+bi, +-br) or -b
    constexpr bool neg_i = swap ? !neg_r : m == 16;
    const V wr = swap ? bi : br, wi = swap ? br : bi;
    sr = neg_r ? vsub(ar, wr) : vadd(ar, wr);
    si = neg_i ? vsub(ai, wi) : vadd(ai, wi);
    dr = neg_r ? vadd(ar, wr) : vsub(ar, wr);
    di = neg_i ? vadd(ai, wi) : vsub(ai, wi);
  } else if constexpr (m % 4 == 0) {          // c (1 + i t), |c| = sqrt(1/2), t = +-1
    constexpr float h = 7.071067691e-01f;
    constexpr float c = kcos32(m) > 0 ? h : -h;
    constexpr float s = (SIGN > 0 ? 1.0f : -1.0f) * (ksin32(m) > 0 ? h : -h);
    constexpr bool same = (c > 0) == (s > 0);
    const V u = same ? vsub(br, bi) : vadd(br, bi);
    const V w = same ? vadd(bi, br) : vsub(bi, br);
    sr = vfma(u, c, ar);
    si = vfma(w, c, ai);
    dr = vfma(u, -c, ar);
    di = vfma(w, -c, ai);
  } else {
    constexpr float c = kcos32(m);
    constexpr float s = (SIGN > 0 ? 1.0f : -1.0f) * ksin32(m);
    sr = vfma(br, c, vfma(bi, -s, ar));
    si = vfma(bi, c, vfma(br, s, ai));
    dr = vfma(br, -c, vfma(bi, s, ar));
    di = vfma(bi, -c, vfma(br, -s, ai));
  }
}

// 4-point butterfly of (t0, w^e t1, w^2e t2, w^3e t3), w = exp(SIGN * 2 pi i / N)
template <int N, int E, int SIGN>
__device__ __forceinline__ void pbfly4_tw(float2& r0, float2& i0, float2& r1, float2& i1, float2& r2, float2& i2,
                                          float2& r3, float2& i3) {
  float2 ur0, ui0, ur1, ui1, ur2, ui2, dr, di;
  add_sub_tw<N, 2 * E, SIGN>(r0, i0, r2, i2, ur0, ui0, ur1, ui1);
  ptw<N, E, SIGN>(r1, i1);
  add_sub_tw<N, 3 * E, SIGN>(r1, i1, r3, i3, ur2, ui2, dr, di);
  r0 = padd(ur0, ur2);
  i0 = padd(ui0, ui2);
  r2 = psub(ur0, ur2);
  i2 = psub(ui0, ui2);
  r1 = SIGN > 0 ? psub(ur1, di) : padd(ur1, di);
  i1 = SIGN > 0 ? padd(ui1, dr) : psub(ui1, dr);
  r3 = SIGN > 0 ? padd(ur1, di) : psub(ur1, di);
  i3 = SIGN > 0 ? psub(ui1, dr) : padd(ui1, dr);
}

template <int SIGN>
__device__ __forceinline__ void pbfly4(float2& r0, float2& i0, float2& r1, float2& i1, float2& r2, float2& i2,
                                       float2& r3, float2& i3) {
  const float2 ur0 = padd(r0, r2), ui0 = padd(i0, i2), ur1 = psub(r0, r2), ui1 = psub(i0, i2);
  const float2 ur2 = padd(r1, r3), ui2 = padd(i1, i3), dr = psub(r1, r3), di = psub(i1, i3);
  r0 = padd(ur0, ur2);
  i0 = padd(ui0, ui2);
  r2 = psub(ur0, ur2);
  i2 = psub(ui0, ui2);
  // u3 = d * (SIGN * i) = SIGN * (-di, dr)
  r1 = SIGN > 0 ? psub(ur1, di) : padd(ur1, di);
  i1 = SIGN > 0 ? padd(ui1, dr) : psub(ui1, dr);
  r3 = SIGN > 0 ? padd(ur1, di) : psub(ur1, di);
  i3 = SIGN > 0 ? psub(ui1, dr) : padd(ui1, dr);
}

template <int N, int SIGN>
struct PDFT {
  template <int STRIDE, int OFF>
  static __device__ __forceinline__ void run(float2 (&re)[16], float2 (&im)[16]) {
    if constexpr (N == 1) {
    } else if constexpr (N == 2) {
      const float2 ar = re[OFF], ai = im[OFF], br = re[OFF + STRIDE], bi = im[OFF + STRIDE];
      re[OFF] = padd(ar, br);
      im[OFF] = padd(ai, bi);
      re[OFF + STRIDE] = psub(ar, br);
      im[OFF + STRIDE] = psub(ai, bi);
    } else if constexpr (N == 4) {
      pbfly4<SIGN>(re[OFF], im[OFF], re[OFF + STRIDE], im[OFF + STRIDE], re[OFF + 2 * STRIDE], im[OFF + 2 * STRIDE],
                   re[OFF + 3 * STRIDE], im[OFF + 3 * STRIDE]);
    } else {
      constexpr int M = N / 4;
      PDFT<M, SIGN>::template run<4 * STRIDE, OFF>(re, im);
      PDFT<M, SIGN>::template run<4 * STRIDE, OFF + STRIDE>(re, im);
      PDFT<M, SIGN>::template run<4 * STRIDE, OFF + 2 * STRIDE>(re, im);
      PDFT<M, SIGN>::template run<4 * STRIDE, OFF + 3 * STRIDE>(re, im);
      float2 outr[N], outi[N];
      static_for<0, M>([&](auto KK) {
        constexpr int k = decltype(KK)::value;
        float2 r0 = re[OFF + STRIDE * (4 * k)], i0 = im[OFF + STRIDE * (4 * k)];
        float2 r1 = re[OFF + STRIDE * (4 * k + 1)], i1 = im[OFF + STRIDE * (4 * k + 1)];
        float2 r2 = re[OFF + STRIDE * (4 * k + 2)], i2 = im[OFF + STRIDE * (4 * k + 2)];
        float2 r3 = re[OFF + STRIDE * (4 * k + 3)], i3 = im[OFF + STRIDE * (4 * k + 3)];
        pbfly4_tw<N, k, SIGN>(r0, i0, r1, i1, r2, i2, r3, i3);
        outr[k] = r0, outi[k] = i0;
        outr[k + M] = r1, outi[k + M] = i1;
        outr[k + 2 * M] = r2, outi[k + 2 * M] = i2;
        outr[k + 3 * M] = r3, outi[k + 3 * M] = i3;
      });
#pragma unroll
      for (int i = 0; i < N; ++i) {
        re[OFF + STRIDE * i] = outr[i];
        im[OFF + STRIDE * i] = outi[i];
      }
    }
  }
};

// Radii at which the table twiddles are rounded to float32. The DFTs' constants (kcos32) are pairs of
// rounded numbers whose magnitudes are 0.8e-8 to 2.9e-8 short of 1; a transform of them alone has a gain,
// which a multislice chain raises to the power of its 2 Z pairs, where errors of either sign average out.
// The tables are rounded at radii that make up for it. Mean gain of a forward and inverse pair, modelled in
// 64 bits: 64 px -8.8e-8 with every factor rounded at radius 1, here -1.7e-8; 128 px -9.0e-8, here -1.3e-8.
// Measured against 64 bits over 20 slices of 3 modes at 128 px: loss 4.5e-6 -> 0.5e-6, object gradient
// 1.1e-5 -> 1.5e-6, probe gradient 1.4e-5 -> 4.2e-6. Larger radii of the y twiddles, or the larger
// neighbours of the constants, also close the gain, but spread a point's error over others: the position
// gradients of near-field calls at 64 px, the outputs that gain least, went to 1.2 to 1.4 times the error
// (0.9 to 1.05 here).
constexpr double kRadiusX = 1.0 + 3e-8, kRadiusY = 1.0 + 1e-8;

// Twiddle tables, in global memory (twiddle_entry): w_W^(k1*n2) at n2*32 + k1, then w_W^(j1*m2)
// at m2*C + j1, w_W = exp(-2 pi i/W); in shared memory (load_twiddles) as the packed arithmetic
// reads them: tw1 the cosines [k1][n2] then the sines [k1][n2], tw2 (cos, cos, sin, sin) per
// entry. The x twiddle w_W^(k1*n2) between the 32-point and the A-point DFT along x is applied
// in round 2, where a thread holds one k1 and every n2.
template <int W>
__device__ __forceinline__ void load_twiddles(float2* s_tw1, float2* s_tw2, const float2* g_tw) {
  using G = Geo<W>;
  float* t1 = reinterpret_cast<float*>(s_tw1);
  float4* t2 = reinterpret_cast<float4*>(s_tw2);
  for (int i = threadIdx.x; i < G::TW1 + G::TW2; i += blockDim.x) {
    const float2 w = g_tw[i];
    if (i < G::TW1) {
      const int n2 = i / 32, k1 = i % 32;
      t1[k1 * G::A + n2] = w.x;
      t1[G::TW1 + k1 * G::A + n2] = w.y;
    } else {
      t2[i - G::TW1] = make_float4(w.x, w.x, w.y, w.y);
    }
  }
}

template <int W>
struct WinFFT {
  using G = Geo<W>;
  static constexpr int A = G::A, C = G::C, Bq = G::Bq, Q = G::Q, S3 = G::S3;
  static constexpr int WPART = 1024;   // float2 of the exchange buffer that a warp owns
  static constexpr int PLANE = 1024;   // floats of one plane (real or imaginary) of the warp's transpose
  static constexpr int H = W / 2;      // words of a row of the cross-warp exchange

  // the x twiddles of this lane's k1 as packs over n2: pack h of A/2 covers n2 = 2h, 2h + 1
  struct Tw1 {
    float2 x[A / 2], y[A / 2];
    __device__ __forceinline__ Tw1(const float2* tw1, int k1) {
      const float2* t = tw1 + k1 * (A / 2);
#pragma unroll
      for (int h = 0; h < A / 2; ++h) {
        x[h] = t[h];
        y[h] = t[G::TW1 / 2 + h];
      }
    }
  };

  // real layout -> frequency layout, unnormalised, exp(-2 pi i ...) kernel
  static __device__ __forceinline__ void forward(Win& v, float2* xbuf, const float2* tw1, const float2* tw2) {
    const int t = threadIdx.x, lane = t % 32, m2 = t / 32;   // lane: round 1's row, round 2's k1
    float* xw = reinterpret_cast<float*>(xbuf + m2 * WPART);
    float4* x4 = reinterpret_cast<float4*>(xbuf);
    // ---- round 1: 16-point DFTs of the even and odd x, then X_k, X_{k+16} = E_k +- w_32^k O_k
    PDFT<16, -1>::template run<1, 0>(v.re, v.im);
    static_for<0, 16>([&](auto KK) {
      constexpr int k = decltype(KK)::value;
      float2 a, b;
      add_sub_tw<32, k, -1>(v.re[k].x, v.im[k].x, v.re[k].y, v.im[k].y, a.x, a.y, b.x, b.y);
      // row k1, word (lane / 4) ^ (k1 & 7); rows k and k + 16 share the swizzle
      float* d = xw + k * 32 + ((((lane >> 2) ^ (k & 7)) << 2) | (lane & 3));
      d[0] = a.x;
      d[PLANE] = a.y;
      d[16 * 32] = b.x;
      d[16 * 32 + PLANE] = b.y;
    });
    __syncwarp();
    // ---- round 2: word c of row k1 = lane holds local rows 4c .. 4c + 3 (row m1*A + n2)
    {
      const float4* p4 = reinterpret_cast<const float4*>(xw) + lane * 8;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const float4 r = p4[c ^ (lane & 7)], i = p4[(c ^ (lane & 7)) + PLANE / 4];
        v.re[2 * c] = make_float2(r.x, r.y);
        v.re[2 * c + 1] = make_float2(r.z, r.w);
        v.im[2 * c] = make_float2(i.x, i.y);
        v.im[2 * c + 1] = make_float2(i.z, i.w);
      }
    }
    {   // x twiddle w_W^(k1*n2): this thread's k1 is fixed
      const Tw1 w(tw1, lane);
#pragma unroll
      for (int h = 0; h < A / 2; ++h) {
        const float2 ny = pneg(w.y[h]);
#pragma unroll
        for (int m1 = 0; m1 < C; ++m1) pcmul(v.re[m1 * (A / 2) + h], v.im[m1 * (A / 2) + h], w.x[h], w.y[h], ny);
      }
    }
    static_for<0, A / 2>([&](auto HH) { PDFT<C, -1>::template run<A / 2, decltype(HH)::value>(v.re, v.im); });
    if (m2 != 0) {
      const float4* t2 = reinterpret_cast<const float4*>(tw2) + m2 * C;
#pragma unroll
      for (int j1 = 1; j1 < C; ++j1) {
        const float4 w = t2[j1];
        const float2 ws = make_float2(w.z, w.w), ns = pneg(ws);
#pragma unroll
        for (int h = 0; h < A / 2; ++h)
          pcmul(v.re[j1 * (A / 2) + h], v.im[j1 * (A / 2) + h], make_float2(w.x, w.y), ws, ns);
      }
    }
    __syncwarp();   // the warp has read its transpose
    // A-point DFT over n2, joining the halves of the packs; kx and kx + W/2 leave as one word
    // (re, re', im, im')
#pragma unroll
    for (int j1 = 0; j1 < C; ++j1) {
      float4* row = x4 + (m2 * C + j1) * H + lane;
      if constexpr (A == 2) {
        const float2 r = v.re[j1], i = v.im[j1];
        row[0] = make_float4(r.x + r.y, r.x - r.y, i.x + i.y, i.x - i.y);
      } else {
        const float2 ur = padd(v.re[2 * j1], v.re[2 * j1 + 1]), ui = padd(v.im[2 * j1], v.im[2 * j1 + 1]);
        const float2 dr = psub(v.re[2 * j1], v.re[2 * j1 + 1]), di = psub(v.im[2 * j1], v.im[2 * j1 + 1]);
        row[0] = make_float4(ur.x + ur.y, ur.x - ur.y, ui.x + ui.y, ui.x - ui.y);         // k2 = 0, 2
        row[32] = make_float4(dr.x + di.y, dr.x - di.y, di.x - dr.y, di.x + dr.y);        // k2 = 1, 3
      }
    }
    __syncthreads();
    // ---- round 3
    {
      const int g = t % S3, j1 = t / S3;
      const float4* col = x4 + j1 * H + g;
#pragma unroll
      for (int q = 0; q < Q / 2; ++q)
#pragma unroll
        for (int r = 0; r < Bq; ++r) {
          const float4 w = col[r * C * H + S3 * q];
          v.re[q * Bq + r] = make_float2(w.x, w.y);
          v.im[q * Bq + r] = make_float2(w.z, w.w);
        }
      static_for<0, Q / 2>([&](auto QQ) { PDFT<Bq, -1>::template run<1, decltype(QQ)::value * Bq>(v.re, v.im); });
    }
  }

  // frequency layout -> real layout, unnormalised, exp(+2 pi i ...) kernel (no 1/W^2)
  static __device__ __forceinline__ void inverse(Win& v, float2* xbuf, const float2* tw1, const float2* tw2) {
    inverse_head(v, xbuf, tw1, tw2);
    inverse_tail(v);
  }

  // The register-only end of the inverse transform (round 1): callers that reuse xbuf may
  // run inverse_head (everything up to the last xbuf read), __syncwarp, refill the warp's part
  // of xbuf asynchronously, and then run inverse_tail while the copy is in flight.
  static __device__ __forceinline__ void inverse_tail(Win& v) {
    // 16-point DFTs of the even and odd k, then x_n, x_{n+16} = E_n +- w_32^-n O_n
    PDFT<16, +1>::template run<1, 0>(v.re, v.im);
    Win e = v;
    static_for<0, 16>([&](auto NN) {
      constexpr int n = decltype(NN)::value;
      float2 a, b;
      add_sub_tw<32, n, +1>(e.re[n].x, e.im[n].x, e.re[n].y, e.im[n].y, a.x, a.y, b.x, b.y);
      wset(v, n, a);
      wset(v, n + 16, b);
    });
  }

  // inverse() without its register-only tail
  static __device__ __forceinline__ void inverse_head(Win& v, float2* xbuf, const float2* tw1, const float2* tw2) {
    const int t = threadIdx.x, lane = t % 32, m2 = t / 32;
    float* xw = reinterpret_cast<float*>(xbuf + m2 * WPART);
    float4* x4 = reinterpret_cast<float4*>(xbuf);
    {
      const int g = t % S3, j1 = t / S3;
      static_for<0, Q / 2>([&](auto QQ) { PDFT<Bq, +1>::template run<1, decltype(QQ)::value * Bq>(v.re, v.im); });
      // the addresses that this thread loaded in the forward's round 3: no barrier between
      float4* col = x4 + j1 * H + g;
#pragma unroll
      for (int q = 0; q < Q / 2; ++q)
#pragma unroll
        for (int r = 0; r < Bq; ++r)
          col[r * C * H + S3 * q] =
              make_float4(v.re[q * Bq + r].x, v.re[q * Bq + r].y, v.im[q * Bq + r].x, v.im[q * Bq + r].y);
    }
    __syncthreads();
#pragma unroll
    for (int j1 = 0; j1 < C; ++j1) {
      const float4* row = x4 + (m2 * C + j1) * H + lane;
      if constexpr (A == 2) {
        const float4 a = row[0];
        v.re[j1] = make_float2(a.x + a.y, a.x - a.y);
        v.im[j1] = make_float2(a.z + a.w, a.z - a.w);
      } else {
        const float4 a = row[0], b = row[32];   // X0, X2 and X1, X3
        const float2 ur = make_float2(a.x + a.y, a.x - a.y), ui = make_float2(a.z + a.w, a.z - a.w);
        // (X1 + X3, i (X1 - X3))
        const float2 sr = make_float2(b.x + b.y, b.w - b.z), si = make_float2(b.z + b.w, b.x - b.y);
        v.re[2 * j1] = padd(ur, sr);
        v.im[2 * j1] = padd(ui, si);
        v.re[2 * j1 + 1] = psub(ur, sr);
        v.im[2 * j1 + 1] = psub(ui, si);
      }
    }
    if (m2 != 0) {
      const float4* t2 = reinterpret_cast<const float4*>(tw2) + m2 * C;
#pragma unroll
      for (int j1 = 1; j1 < C; ++j1) {
        const float4 w = t2[j1];
        const float2 ws = make_float2(w.z, w.w), ns = pneg(ws);
#pragma unroll
        for (int h = 0; h < A / 2; ++h)
          pcmul(v.re[j1 * (A / 2) + h], v.im[j1 * (A / 2) + h], make_float2(w.x, w.y), ns, ws);
      }
    }
    static_for<0, A / 2>([&](auto HH) { PDFT<C, +1>::template run<A / 2, decltype(HH)::value>(v.re, v.im); });
    {   // conjugate x twiddle w_W^(-k1*n2), this thread's k1 fixed
      const Tw1 w(tw1, lane);
#pragma unroll
      for (int h = 0; h < A / 2; ++h) {
        const float2 ny = pneg(w.y[h]);
#pragma unroll
        for (int m1 = 0; m1 < C; ++m1) pcmul(v.re[m1 * (A / 2) + h], v.im[m1 * (A / 2) + h], w.x[h], ny, w.y[h]);
      }
    }
    __syncwarp();   // the warp has read its part of the cross-warp exchange
    {
      float4* p4 = reinterpret_cast<float4*>(xw) + lane * 8;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        p4[c ^ (lane & 7)] = make_float4(v.re[2 * c].x, v.re[2 * c].y, v.re[2 * c + 1].x, v.re[2 * c + 1].y);
        p4[(c ^ (lane & 7)) + PLANE / 4] = make_float4(v.im[2 * c].x, v.im[2 * c].y, v.im[2 * c + 1].x, v.im[2 * c + 1].y);
      }
    }
    __syncwarp();
    // pack m: the elements k = 2m and 2m + 1 of this lane's row
    static_for<0, 16>([&](auto MM) {
      constexpr int m = decltype(MM)::value, k = 2 * m;
      const float* d0 = xw + k * 32 + ((((lane >> 2) ^ (k & 7)) << 2) | (lane & 3));
      const float* d1 = xw + (k + 1) * 32 + ((((lane >> 2) ^ ((k + 1) & 7)) << 2) | (lane & 3));
      v.re[m] = make_float2(d0[0], d1[0]);
      v.im[m] = make_float2(d0[PLANE], d1[PLANE]);
    });
  }
};

// ------------------------------------------------------------------ native window layout
// Windows that live only inside the library are stored in the order the FFT threads own
// them, warp by warp: pack p of lane l of warp w is the 16-byte word (re, re', im, im') at word
// w*512 + p*32 + l. A warp touches 512 contiguous bytes per access, and a warp's whole share is
// 8 KB in one piece (its first 512*p bytes the packs below p), so each warp's operands move by
// bulk copies of its own.
__device__ __forceinline__ int nword(int p, int t) { return (t >> 5) * 512 + p * 32 + (t & 31); }   // in float4

__device__ __forceinline__ float4 pack4(float2 re, float2 im) { return make_float4(re.x, re.y, im.x, im.y); }

__device__ __forceinline__ void ld_native(const float2* base, Win& v) {
  const float4* p = reinterpret_cast<const float4*>(base) + nword(0, threadIdx.x);
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const float4 q = p[j * 32];
    v.re[j] = make_float2(q.x, q.y);
    v.im[j] = make_float2(q.z, q.w);
  }
}

__device__ __forceinline__ void st_native(float2* base, const Win& v) {
  float4* p = reinterpret_cast<float4*>(base) + nword(0, threadIdx.x);
#pragma unroll
  for (int j = 0; j < 16; ++j) p[j * 32] = pack4(v.re[j], v.im[j]);
}

// element i of thread t of a native window
__device__ __forceinline__ float2 native_at(const float2* base, int i, int t) {
  const float* w = reinterpret_cast<const float*>(reinterpret_cast<const float4*>(base) + nword(i >> 1, t));
  return make_float2(w[i & 1], w[2 + (i & 1)]);
}

// ------------------------------------------------------------------ bulk async copies
// One-dimensional TMA bulk copies global -> shared completed on an mbarrier, with bounded
// waits: a wait that runs out sets *err and returns instead of spinning forever.
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

// orders this thread's earlier generic-proxy shared-memory accesses before later
// async-proxy (TMA) accesses
__device__ __forceinline__ void fence_async_shared() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// the same for global memory written with ordinary stores and read back by TMA
__device__ __forceinline__ void fence_async_global() {
  asm volatile("fence.proxy.async.global;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

// dst, src 16-byte aligned, bytes a multiple of 16
__device__ __forceinline__ void bulk_copy_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

constexpr int kMbarWaitLimit = 1 << 20;   // try_wait rounds before a wait is declared failed

__device__ __forceinline__ void mbar_wait(uint64_t* bar, uint32_t& parity, int* err) {
  for (int it = 0; !mbar_try_wait(bar, parity); ++it) {
    if (it >= kMbarWaitLimit) {
      if (err) *err = 1;
      break;
    }
  }
  parity ^= 1u;
}

// Asynchronous copies global -> shared through the load path (cp.async: any global address,
// device memory or mapped pinned host memory), 16 or 4 bytes per copy with both addresses
// aligned to the size; a thread's copies are complete after its cp_async_wait_all().
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// Issue (one thread) an L2 prefetch of `bytes` at `src` (16-byte aligned, a multiple of 16
// bytes) in chunks of at most 64 KiB; nothing waits on it.
__device__ __forceinline__ void prefetch_l2(const void* src, uint32_t bytes) {
  constexpr uint32_t kChunk = 64u * 1024u;
  for (uint32_t o = 0; o < bytes; o += kChunk) {
    const uint32_t n = bytes - o < kChunk ? bytes - o : kChunk;
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(static_cast<const char*>(src) + o), "r"(n)
                 : "memory");
  }
}

// Issue (one thread) a copy of `bytes` from global `src` into shared `dst` in chunks of at
// most 64 KiB, all completing on `bar`.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  mbar_expect_tx(bar, bytes);
  constexpr uint32_t kChunk = 64u * 1024u;
  for (uint32_t o = 0; o < bytes; o += kChunk) {
    const uint32_t n = bytes - o < kChunk ? bytes - o : kChunk;
    bulk_copy_g2s(static_cast<char*>(dst) + o, static_cast<const char*>(src) + o, n, bar);
  }
}

// Issue (one thread) a copy of `bytes` from shared `src` to global `dst` in chunks of at most
// 64 KiB as one bulk group. The writer threads of `src` have run fence_async_shared() and a
// block barrier before this; `src` may be overwritten after bulk_wait_read() in this thread.
__device__ __forceinline__ void bulk_store(void* dst, const void* src, uint32_t bytes) {
  constexpr uint32_t kChunk = 64u * 1024u;
  for (uint32_t o = 0; o < bytes; o += kChunk) {
    const uint32_t n = bytes - o < kChunk ? bytes - o : kChunk;
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(static_cast<char*>(dst) + o),
                 "r"(smem_u32(src) + o), "r"(n)
                 : "memory");
  }
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

// every bulk store of this thread has finished reading its shared-memory source
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }

// every bulk store of this thread has completed its writes to global memory
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// cos and sin of 2 pi k / 128 at a radius, rounded, formed by the compiler: the octant's Taylor series in
// 64 bits (x <= pi / 4: 14 terms are past 1e-16)
struct Roots128 {
  float c[128], s[128];
};
constexpr Roots128 make_roots128(double radius) {
  Roots128 r{};
  for (int k = 0; k < 128; ++k) {
    const int quadrant = k / 32, j = k % 32;              // angle (pi / 2) (quadrant + j / 32)
    const int o = j <= 16 ? j : 32 - j;                   // reflected at pi / 4
    const double x = 3.14159265358979323846 * o / 64;
    double term = 1, c = 0, s = 0;
    for (int n = 0; n < 14; ++n) {                        // term = x^n / n!
      const double signed_term = (n & 2) ? -term : term;
      if (n & 1) s += signed_term;
      else c += signed_term;
      term *= x / (n + 1);
    }
    double cq = j <= 16 ? c : s, sq = j <= 16 ? s : c;
    for (int q = 0; q < quadrant; ++q) {
      const double t = cq;
      cq = -sq;
      sq = t;
    }
    r.c[k] = (float)(cq * radius);
    r.s[k] = (float)(sq * radius);
  }
  return r;
}
__device__ constexpr Roots128 kRootsX = make_roots128(kRadiusX);
__device__ constexpr Roots128 kRootsY = make_roots128(kRadiusY);

// Entry i of the twiddle tables in global memory (see load_twiddles).
template <int W>
__device__ __forceinline__ float2 twiddle_entry(int i) {
  using G = Geo<W>;
  if (i < G::TW1) {
    const int n2 = i / 32, k1 = i % 32, e = (k1 * n2) % W * (128 / W);
    return make_float2(kRootsX.c[e], -kRootsX.s[e]);
  }
  const int j = i - G::TW1, m2 = j / G::C, j1 = j % G::C, e = (j1 * m2) % W * (128 / W);
  return make_float2(kRootsY.c[e], -kRootsY.s[e]);
}

// Builder of the twiddle tables in global memory.
template <int W>
__global__ void build_twiddles_kernel(float2* g_tw) {
  using G = Geo<W>;
  for (int i = threadIdx.x + blockIdx.x * blockDim.x; i < G::TW1 + G::TW2; i += blockDim.x * gridDim.x)
    g_tw[i] = twiddle_entry<W>(i);
}

}  // namespace pty
