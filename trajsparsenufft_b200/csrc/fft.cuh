// Line FFT of length G over C interleaved sequences, by the threads of one CTA in FP32.
//
// A line is [G][C] complex, coil fastest. Thread t works for coil t % C; a pass is a set of
// independent radix-R butterflies, taken TB at a time (TB = threads / C), so neighbouring
// threads touch neighbouring memory in global and in shared memory alike. G = R1 R2 R3:
//   1. radix R1 over n = b + S1 j (j < R1, S1 = G / R1), straight from the caller's load(n)
//      (global memory; zero padding costs no read), times W_G^(b k1), to shared row
//      b + S1 k1;
//   2. radix R2 inside each k1 block, in place, times W_S1^(b2 k2);
//   3. radix R3, straight to the caller's store(k): X[k1 + R1 k2 + R1 R2 k3].
// G = R1 R2 skips the middle pass. A butterfly of a pass reads and writes the same rows, so a
// pass needs no registers beyond one butterfly and one barrier separates two passes. Each k1
// block is followed by one pad row: the last pass reads rows S1 + 1 apart, an odd number of
// rows, which spreads them over the banks.
//
// What bounds it: shared-memory bandwidth and instruction issue, beside the line's own global
// traffic. The passes move each value through shared memory once (two radices) or twice
// (three). It replaces a warp-per-coil FFT that staged slabs, transposes and outputs through
// shared memory (four round trips per value, 1130 warp instructions per 512-point FFT).
// Launches before and after: 512 points, 8 coils, 512 columns forward / inverse 10.5 / 9.4 ->
// 7.2 / 7.0 us; 640 points, 12 coils 32.7 / 33.5 -> 17.8 / 16.8 us; 256^3 volume of 8 coils 461 /
// 466 -> 245 / 236 us (1.6 GB, 6.6 TB/s).
//
// Forward = exp(-2 pi i nk/G), inverse = exp(+2 pi i nk/G), both unnormalized. tw is the
// plan's table exp(-2 pi i e / G), FP64-computed and FP32-stored.
// The reference's FFT endpoints are SIMT FP32 shared-memory radix-8/16/32 kernels
// (nufft_custom_fft_forward_bench.cu:918-999, :1463-1552); this is an independent design.
#pragma once

#include "device.cuh"

namespace tsn {
namespace dev {

// multiply by exp(-i pi / 2) (forward) or exp(+i pi / 2) (inverse)
template <bool INV>
__host__ __device__ __forceinline__ float2 rot90(float2 a) {
  return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}
// multiply by (c, -s) (forward) or (c, +s) (inverse)
template <bool INV>
__host__ __device__ __forceinline__ float2 rot(float2 a, float c, float s) {
  return INV ? make_float2(a.x * c - a.y * s, a.y * c + a.x * s) : make_float2(a.x * c + a.y * s, a.y * c - a.x * s);
}

// In-register DFT of length R, natural order in and out.
template <int R, bool INV>
struct Dft;

template <bool INV>
struct Dft<2, INV> {
  static __host__ __device__ __forceinline__ void run(float2& a, float2& b) {
    const float2 t = a;
    a = cadd(t, b);
    b = csub(t, b);
  }
};

template <bool INV>
struct Dft<3, INV> {
  static __host__ __device__ __forceinline__ void run(float2& a, float2& b, float2& c) {
    const float h = 0.86602540378443864676f;  // sin(pi/3)
    const float2 s = cadd(b, c), d = cscale(rot90<INV>(csub(b, c)), h);
    const float2 m = make_float2(a.x - 0.5f * s.x, a.y - 0.5f * s.y);
    a = cadd(a, s);
    b = cadd(m, d);
    c = csub(m, d);
  }
};

template <bool INV>
struct Dft<4, INV> {
  static __host__ __device__ __forceinline__ void run(float2& a, float2& b, float2& c, float2& d) {
    const float2 s0 = cadd(a, c), d0 = csub(a, c), s1 = cadd(b, d), d1 = rot90<INV>(csub(b, d));
    a = cadd(s0, s1);
    b = cadd(d0, d1);
    c = csub(s0, s1);
    d = csub(d0, d1);
  }
};

template <bool INV>
struct Dft<5, INV> {
  static __host__ __device__ __forceinline__ void run(float2& a, float2& b, float2& c, float2& d, float2& e) {
    const float c1 = 0.30901699437494742410f, c2 = -0.80901699437494742410f;  // cos(2 pi/5), cos(4 pi/5)
    const float s1 = 0.95105651629515357212f, s2 = 0.58778525229247312917f;   // sin(2 pi/5), sin(4 pi/5)
    const float2 p1 = cadd(b, e), m1 = rot90<INV>(csub(b, e)), p2 = cadd(c, d), m2 = rot90<INV>(csub(c, d));
    const float2 u1 = make_float2(a.x + c1 * p1.x + c2 * p2.x, a.y + c1 * p1.y + c2 * p2.y);
    const float2 u2 = make_float2(a.x + c2 * p1.x + c1 * p2.x, a.y + c2 * p1.y + c1 * p2.y);
    const float2 v1 = make_float2(s1 * m1.x + s2 * m2.x, s1 * m1.y + s2 * m2.y);
    const float2 v2 = make_float2(s2 * m1.x - s1 * m2.x, s2 * m1.y - s1 * m2.y);
    a = make_float2(a.x + p1.x + p2.x, a.y + p1.y + p2.y);
    b = cadd(u1, v1);
    c = cadd(u2, v2);
    d = csub(u2, v2);
    e = csub(u1, v1);
  }
};

// Length 6 and 10 = 2 * odd, coprime factors (no twiddles): element n = (P n1 + 2 n2) mod R,
// output k = the index with k mod 2 = k1, k mod P = k2.
template <bool INV>
struct Dft<6, INV> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[6]) {
    float2 a[3] = {v[0], v[2], v[4]}, b[3] = {v[3], v[5], v[1]};
    Dft<3, INV>::run(a[0], a[1], a[2]);
    Dft<3, INV>::run(b[0], b[1], b[2]);
#pragma unroll
    for (int k = 0; k < 3; ++k) Dft<2, INV>::run(a[k], b[k]);
    // The length-3 output index is 2 k2 mod 3 of the decimated transform: k2 = 0, 1, 2 of a
    // belongs to k = 0, 4, 2 (even) and b to k = 3, 1, 5 (odd)
    v[0] = a[0]; v[4] = a[1]; v[2] = a[2];
    v[3] = b[0]; v[1] = b[1]; v[5] = b[2];
  }
};

template <bool INV>
struct Dft<10, INV> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[10]) {
    float2 a[5] = {v[0], v[2], v[4], v[6], v[8]}, b[5] = {v[5], v[7], v[9], v[1], v[3]};
    Dft<5, INV>::run(a[0], a[1], a[2], a[3], a[4]);
    Dft<5, INV>::run(b[0], b[1], b[2], b[3], b[4]);
#pragma unroll
    for (int k = 0; k < 5; ++k) Dft<2, INV>::run(a[k], b[k]);
    // even k = k2 mod 5: 0, 6, 2, 8, 4; odd k: 5, 1, 7, 3, 9
    v[0] = a[0]; v[6] = a[1]; v[2] = a[2]; v[8] = a[3]; v[4] = a[4];
    v[5] = b[0]; v[1] = b[1]; v[7] = b[2]; v[3] = b[3]; v[9] = b[4];
  }
};

template <bool INV>
struct Dft<8, INV> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[8]) {
    const float h = 0.70710678118654752440f;
    float2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    Dft<4, INV>::run(e[0], e[1], e[2], e[3]);
    Dft<4, INV>::run(o[0], o[1], o[2], o[3]);
    // o[k] *= W_8^k
    o[1] = cscale(INV ? make_float2(o[1].x - o[1].y, o[1].y + o[1].x) : make_float2(o[1].x + o[1].y, o[1].y - o[1].x), h);
    o[2] = rot90<INV>(o[2]);
    o[3] = cscale(INV ? make_float2(-o[3].x - o[3].y, o[3].x - o[3].y) : make_float2(o[3].y - o[3].x, -o[3].x - o[3].y), h);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[k] = cadd(e[k], o[k]);
      v[k + 4] = csub(e[k], o[k]);
    }
  }
};

template <bool INV>
struct Dft<16, INV> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[16]) {
    const float c1 = 0.92387953251128675613f, s1 = 0.38268343236508977173f;  // cos, sin of pi/8
    const float h = 0.70710678118654752440f;
#pragma unroll
    for (int i = 0; i < 4; ++i) Dft<4, INV>::run(v[i], v[i + 4], v[i + 8], v[i + 12]);
    // v[i + 4 k] *= W_16^(i k)
    v[5] = rot<INV>(v[5], c1, s1);
    v[6] = rot<INV>(v[6], h, h);
    v[7] = rot<INV>(v[7], s1, c1);
    v[9] = rot<INV>(v[9], h, h);
    v[10] = rot90<INV>(v[10]);
    v[11] = rot<INV>(v[11], -h, h);
    v[13] = rot<INV>(v[13], s1, c1);
    v[14] = rot<INV>(v[14], -h, h);
    v[15] = rot<INV>(v[15], -c1, -s1);
    float2 o[16];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      Dft<4, INV>::run(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
#pragma unroll
      for (int q = 0; q < 4; ++q) o[k + 4 * q] = v[4 * k + q];
    }
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = o[k];
  }
};

// Radices of each supported length.
template <int G>
struct FftRadix;
template <> struct FftRadix<128> { static constexpr int R1 = 8, R2 = 16, R3 = 1, TB = 16; };
template <> struct FftRadix<256> { static constexpr int R1 = 16, R2 = 16, R3 = 1, TB = 16; };
template <> struct FftRadix<384> { static constexpr int R1 = 8, R2 = 8, R3 = 6, TB = 16; };
template <> struct FftRadix<512> { static constexpr int R1 = 8, R2 = 8, R3 = 8, TB = 32; };
template <> struct FftRadix<640> { static constexpr int R1 = 8, R2 = 8, R3 = 10, TB = 40; };
template <> struct FftRadix<1024> { static constexpr int R1 = 16, R2 = 8, R3 = 8, TB = 64; };

// C: interleaved sequences in shared memory (coils of this CTA)
template <int G, int C, bool INV>
struct LineFft {
  using P = FftRadix<G>;
  static constexpr int R1 = P::R1, R2 = P::R2, R3 = P::R3, TB = P::TB;
  static constexpr int THREADS = C * TB;
  static constexpr int S1 = G / R1, S2 = S1 / R2;
  static constexpr int RL = R3 > 1 ? R3 : R2;     // radix of the last pass
  static constexpr int NL = G / RL;               // butterflies of the last pass
  static constexpr int ITL = (NL + TB - 1) / TB;  // its iterations per thread
  static constexpr int ROWS = G + R1;             // shared rows of C complex values
  static_assert(R1 * R2 * R3 == G, "radices");

  static __host__ __device__ __forceinline__ float2 twiddle(float2 v, const float2* tw, int e) {
    const float2 w = tw[e];
    return INV ? cmulc(v, w) : cmul(v, w);
  }

  // load(n): element n of the line, 0 <= n < G
  template <class Load>
  static __host__ __device__ __forceinline__ void first(float2* s, const float2* tw, int tid, Load load) {
    constexpr int IT = (S1 + TB - 1) / TB;
    constexpr int GROUP = R1 >= 16 ? 1 : 2;  // butterflies whose loads are in flight together
    const int c = tid % C, b0 = tid / C;
#pragma unroll
    for (int i0 = 0; i0 < IT; i0 += GROUP) {
      float2 v[GROUP][R1];
#pragma unroll
      for (int g = 0; g < GROUP; ++g) {
        const int b = b0 + (i0 + g) * TB;
        if (i0 + g < IT && (S1 % TB == 0 || b < S1)) {
#pragma unroll
          for (int j = 0; j < R1; ++j) v[g][j] = load(b + S1 * j);
        }
      }
#pragma unroll
      for (int g = 0; g < GROUP; ++g) {
        const int b = b0 + (i0 + g) * TB;
        if (i0 + g < IT && (S1 % TB == 0 || b < S1)) {
          Dft<R1, INV>::run(v[g]);
          s[b * C + c] = v[g][0];
#pragma unroll
          for (int k = 1; k < R1; ++k) s[(b + (S1 + 1) * k) * C + c] = twiddle(v[g][k], tw, b * k);
        }
      }
    }
  }

  // middle pass of a three-radix length
  static __host__ __device__ __forceinline__ void middle(float2* s, const float2* tw, int tid) {
    if constexpr (R3 > 1) {
      constexpr int NB = R1 * S2, IT = (NB + TB - 1) / TB;
      const int c = tid % C, b0 = tid / C;
#pragma unroll
      for (int i = 0; i < IT; ++i) {
        const int b = b0 + i * TB;
        if (NB % TB == 0 || b < NB) {
          const int b2 = b % S2, k1 = b / S2;
          float2* q = s + (b2 + (S1 + 1) * k1) * C + c;
          float2 v[R2];
#pragma unroll
          for (int j = 0; j < R2; ++j) v[j] = q[S2 * j * C];
          Dft<R2, INV>::run(v);
          q[0] = v[0];
#pragma unroll
          for (int k = 1; k < R2; ++k) q[S2 * k * C] = twiddle(v[k], tw, R1 * b2 * k);
        }
      }
    }
  }

  // store(i, j, k, value): output element k; i (iteration) and j are compile-time constants
  // after unrolling, for callers that keep the values in registers
  template <class Store>
  static __host__ __device__ __forceinline__ void last(const float2* s, int tid, Store store) {
    const int c = tid % C, b0 = tid / C;
#pragma unroll
    for (int i = 0; i < ITL; ++i) {
      const int b = b0 + i * TB;
      if (NL % TB == 0 || b < NL) {
        // b = k1 + R1 k2
        const float2* q = s + ((R3 > 1 ? RL * (b / R1) : 0) + (S1 + 1) * (b % R1)) * C + c;
        float2 v[RL];
#pragma unroll
        for (int j = 0; j < RL; ++j) v[j] = q[j * C];
        Dft<RL, INV>::run(v);
#pragma unroll
        for (int j = 0; j < RL; ++j) store(i, j, b + NL * j, v[j]);
      }
    }
  }
  // The last pass in place: output k is left in shared row out_row(k).
  static __host__ __device__ __forceinline__ void last_in_place(float2* s, int tid) {
    const int c = tid % C, b0 = tid / C;
#pragma unroll
    for (int i = 0; i < ITL; ++i) {
      const int b = b0 + i * TB;
      if (NL % TB == 0 || b < NL) {
        float2* q = s + ((R3 > 1 ? RL * (b / R1) : 0) + (S1 + 1) * (b % R1)) * C + c;
        float2 v[RL];
#pragma unroll
        for (int j = 0; j < RL; ++j) v[j] = q[j * C];
        Dft<RL, INV>::run(v);
#pragma unroll
        for (int j = 0; j < RL; ++j) q[j * C] = v[j];
      }
    }
  }
  static __host__ __device__ __forceinline__ int out_row(int k) {
    const int b = k % NL, j = k / NL;
    return (R3 > 1 ? RL * (b / R1) : 0) + (S1 + 1) * (b % R1) + j;
  }
  // last-pass butterfly of iteration i of thread tid (its outputs: b + NL j), or -1
  static __host__ __device__ __forceinline__ int last_base(int tid, int i) {
    const int b = tid / C + i * TB;
    return NL % TB == 0 || b < NL ? b : -1;
  }
};

}  // namespace dev
}  // namespace tsn
