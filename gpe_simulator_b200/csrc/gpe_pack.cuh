// gpe_pack.cuh -- complex64 line transforms of two lines at once with packed FP32 (sm_100a).
//
// sm_100a issues fma, add and mul on a pair of floats in one instruction
// (fma.rn.f32x2 and so on) at half the rate of the scalar ones: the same operations per
// clock for half the issue slots.  The fused complex64 sweeps are bound by issue, so
// they hold two lines per thread as pairs: F2 = (line a, line b), a complex value C2 =
// (re pair, im pair).  Multiplications by +-i and conjugations then only rename and change
// a sign, and one 16-byte access moves both lines' values.
//
// The operations, their fused multiply-adds and their order are those of gpe_fft.cuh;
// inverse transforms negate the sines instead of conjugating the data, which mirrors every
// rounding.
#pragma once
#include "gpe_fft.cuh"

namespace gpe {

struct F2 { unsigned long long v; };
struct C2 { F2 x, y; };

__device__ __forceinline__ F2 f2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ F2 f2(float a) { return f2(a, a); }
__device__ __forceinline__ float2 unpack(F2 a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.v));
  return r;
}
__device__ __forceinline__ F2 operator+(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 operator-(F2 a, F2 b) {
  F2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 operator*(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ F2 operator-(F2 a) {
  const float2 f = unpack(a);
  return f2(-f.x, -f.y);
}
__device__ __forceinline__ C2 c2(F2 x, F2 y) { C2 r; r.x = x; r.y = y; return r; }
__device__ __forceinline__ C2 operator+(C2 a, C2 b) { return c2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ C2 operator-(C2 a, C2 b) { return c2(a.x - b.x, a.y - b.y); }

// x * (hi + lo)
__device__ __forceinline__ F2 kmul2(F2 x, float hi, float lo) { return fma2(x, f2(hi), x * f2(lo)); }

// v * (c - i s), INV: v * (c + i s), for split constants
template <bool INV> __device__ __forceinline__ C2 rot2(C2 v, float ch, float cl, float sh, float sl) {
  if (INV) { sh = -sh; sl = -sl; }
  return c2(fma2(v.x, f2(ch), fma2(v.y, f2(sh), fma2(v.x, f2(cl), v.y * f2(sl)))),
            fma2(v.y, f2(ch), fma2(v.x, f2(-sh), fma2(v.y, f2(cl), v.x * f2(-sl)))));
}

// v * w (INV: v * conj(w)) for a twiddle {hi.x, hi.y, lo.x, lo.y}, the same for both lines.
// (Entries stored as pairs saved the copies into pairs but doubled the shared-memory reads,
// which bound the z sweeps.)
template <bool INV> __device__ __forceinline__ C2 tw2(C2 v, const float4& w) {
  const F2 wx = f2(w.x), wy = f2(w.y), lx = f2(w.z), ly = f2(w.w);
  if (INV) {
    const F2 nx = -v.x;
    return c2(fma2(v.x, wx, fma2(v.y, wy, fma2(v.x, lx, v.y * ly))),
              fma2(nx, wy, fma2(v.y, wx, fma2(nx, ly, v.y * lx))));
  }
  const F2 ny = -v.y;
  return c2(fma2(v.x, wx, fma2(ny, wy, fma2(v.x, lx, ny * ly))),
            fma2(v.x, wy, fma2(v.y, wx, fma2(v.x, ly, v.y * lx))));
}

// v * W_16^q, W_16 = exp(-+2 pi i / 16), q known at compile time
template <int Q, bool INV> __device__ __forceinline__ C2 mul_w16_2(C2 v) {
  using k = K<float>;
  constexpr int q = Q & 15;
  if constexpr (q == 0) return v;
  else if constexpr (q == 4) return INV ? c2(-v.y, v.x) : c2(v.y, -v.x);
  else if constexpr (q == 8) return c2(-v.x, -v.y);
  else if constexpr (q == 12) return INV ? c2(v.y, -v.x) : c2(-v.y, v.x);
  else if constexpr (q == 2)
    return INV ? c2(kmul2(v.x - v.y, k::R2, k::R2L), kmul2(v.y + v.x, k::R2, k::R2L))
               : c2(kmul2(v.x + v.y, k::R2, k::R2L), kmul2(v.y - v.x, k::R2, k::R2L));
  else if constexpr (q == 6)
    return INV ? c2(kmul2(v.x + v.y, -k::R2, -k::R2L), kmul2(v.x - v.y, k::R2, k::R2L))
               : c2(kmul2(v.y - v.x, k::R2, k::R2L), kmul2(v.y + v.x, -k::R2, -k::R2L));
  else if constexpr (q == 1) return rot2<INV>(v, k::C8, k::C8L, k::S8, k::S8L);
  else if constexpr (q == 3) return rot2<INV>(v, k::S8, k::S8L, k::C8, k::C8L);
  else {
    static_assert(q == 9, "W_16 powers of the radix-4 splits");
    return rot2<INV>(v, -k::C8, -k::C8L, -k::S8, -k::S8L);
  }
}

// DFTs of gpe_fft.cuh (INV: with the opposite sign of the exponent)
template <int R, bool INV> struct Dft2;

template <bool INV> struct Dft2<2, INV> {
  __device__ __forceinline__ static void run(C2* v) {
    const C2 a = v[0], b = v[1];
    v[0] = a + b;
    v[1] = a - b;
  }
};
template <bool INV> struct Dft2<4, INV> {
  __device__ __forceinline__ static void run(C2* v) {
    const C2 t0 = v[0] + v[2], t1 = v[0] - v[2], t2 = v[1] + v[3], d = v[1] - v[3];
    v[0] = t0 + t2;
    v[2] = t0 - t2;
    const C2 p = c2(t1.x + d.y, t1.y - d.x), m = c2(t1.x - d.y, t1.y + d.x);
    v[1] = INV ? m : p;
    v[3] = INV ? p : m;
  }
};
// R = R1*R2 in {8, 16} with W_16 twiddles
template <int R1, int R2, bool INV> struct DftSplit2 {
  static_assert(16 % (R1 * R2) == 0, "W_16 twiddles");
  __device__ __forceinline__ static void run(C2* v) {
    C2 y[R2][R1];
    SFor<0, R2>::run([&](auto n2c) {
      constexpr int n2 = decltype(n2c)::value;
#pragma unroll
      for (int n1 = 0; n1 < R1; ++n1) y[n2][n1] = v[R2 * n1 + n2];
      Dft2<R1, INV>::run(y[n2]);
      SFor<1, R1>::run([&](auto k1c) {
        if constexpr (n2 != 0) {
          constexpr int k1 = decltype(k1c)::value, RR = R1 * R2;
          y[n2][k1] = mul_w16_2<(16 / RR) * ((n2 * k1) % RR), INV>(y[n2][k1]);
        }
      });
    });
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1) {
      C2 z[R2];
#pragma unroll
      for (int n2 = 0; n2 < R2; ++n2) z[n2] = y[n2][k1];
      Dft2<R2, INV>::run(z);
#pragma unroll
      for (int k2 = 0; k2 < R2; ++k2) v[k1 + R1 * k2] = z[k2];
    }
  }
};
template <bool INV> struct Dft2<8, INV>  : DftSplit2<4, 2, INV> {};
template <bool INV> struct Dft2<16, INV> : DftSplit2<4, 4, INV> {};

}  // namespace gpe
