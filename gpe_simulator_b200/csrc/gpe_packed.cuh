// gpe_packed.cuh -- the register-resident complex64 sweeps with two lines per thread
// (packed FP32, gpe_pack.cuh), sm_100a.
//
// Same sweeps, splits, modes and operations as gpe_fast.cuh for n = 256 (16 x 16) and 512
// (8 x 8 x 8): a tile is 16 lines = 8 line pairs, a thread holds 16 values of one pair in one
// slot (n = 512: two).  Against one line per thread that halves the issue slots of the transforms' arithmetic, of the exchange
// (one 16-byte access moves (re a, re b, im a, im b)) and, in y/x tiles, of the loads and
// stores from HBM; twiddles and table values are read once for both lines.  The twiddles
// are copied into shared memory by cp.async (through L1 they missed: with most of it taken
// as shared memory, psi and its stores evict them).
#pragma once
#include "gpe_fast.cuh"
#include "gpe_pack.cuh"

namespace gpe {

template <int N> struct PackCfg {
  static_assert(N == 256 || N == 512, "sides whose twiddles d_twp holds");
  static constexpr bool THREE = N == 512;
  static constexpr int L = FastCfg<N, float>::L, LP = L / 2;
  static constexpr int LANES = Split<N>::N1, VALS = Split<N>::N2;   // of a pair, in every layout
  static constexpr int V = 16;                                      // values per line and thread
  static constexpr int T = LP * N / V, Q = LP * LANES / T;          // threads, slots
  static_assert(Q * T == LP * LANES && Q * VALS == V, "no partial slots");
  // exchange buffer (16-byte elements)
  static constexpr int EX = THREE ? LP * N : LP * (N + LANES);
  static constexpr size_t EXB = (size_t)EX * 16;
  // twiddles of the (first) split, n = 512: then the 64 second-phase ones
  static constexpr int TW = N + (THREE ? 64 : 0);
  // tables of a z sweep: reduction scratch, vz, c1, c2, c12; of an x sweep: kx, kyz, kx2, kyz2
  static constexpr size_t ZB = 32 * 16 + (size_t)(N + 3 * L) * 4, XB = (size_t)(N + L) * 24;
};
template <int N, int MODE> constexpr size_t pack_smem() {
  return PackCfg<N>::EXB + (size_t)PackCfg<N>::TW * 16 + (MODE == FM_PLAIN ? 0 : MODE == FM_XKIN ? PackCfg<N>::XB : PackCfg<N>::ZB);
}

// slot gs of a phase with `per` lanes per pair: pair lp and lane (as slot() in gpe_fast.cuh)
template <int N, int AX> __device__ __forceinline__ void pack_slot(int gs, int per, int& lp, int& lane) {
  constexpr int LP = PackCfg<N>::LP, T = PackCfg<N>::T;
  if (AX == FZ) {
    if (PackCfg<N>::THREE) { const int t = gs % T; lp = t >> 5; lane = (t & 31) + 32 * (gs / T); }
    else { lane = gs % per; lp = gs / per; }
  } else {
    lp = gs % LP;
    lane = gs / LP;
  }
}

// 16 bytes from global to shared memory, asynchronously
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ void ex_store(ulonglong2* p, C2 v) { *p = make_ulonglong2(v.x.v, v.y.v); }
__device__ __forceinline__ C2 ex_load(const ulonglong2* p) {
  const ulonglong2 q = *p;
  C2 v;
  v.x.v = q.x;
  v.y.v = q.y;
  return v;
}

// fft_2phase of gpe_fast.cuh on line pairs (n = 256); tw: the split's twiddles, [k2*16 + lane].
template <int N, int AX, bool INV, bool TAIL>
__device__ __forceinline__ void pack_2phase(C2 (&v)[PackCfg<N>::V], ulonglong2* ex, const float4* tw) {
  constexpr int LP = PackCfg<N>::LP, A = 16;
  static_assert(N == A * A && PackCfg<N>::Q == 1, "two-phase layout");
  constexpr bool WARP_LOCAL = AX == FZ && LP * A == PackCfg<N>::T;
  int lp, lane;
  pack_slot<N, AX>(threadIdx.x, A, lp, lane);
  Dft2<A, INV>::run(v);
#pragma unroll
  for (int k2 = 1; k2 < A; ++k2) v[k2] = tw2<INV>(v[k2], tw[k2 * A + lane]);
#pragma unroll
  for (int k2 = 0; k2 < A; ++k2)
    ex_store(ex + (AX == FZ ? (lp * A + k2) * (A + 1) + lane : (k2 * A + lane) * LP + lp), v[k2]);
  if (WARP_LOCAL) __syncwarp(); else __syncthreads();
  // (the slot's lane is the second phase's k2)
#pragma unroll
  for (int n1 = 0; n1 < A; ++n1)
    v[n1] = ex_load(ex + (AX == FZ ? (lp * A + lane) * (A + 1) + n1 : (lane * A + n1) * LP + lp));
  Dft2<A, INV>::run(v);
  if (TAIL) {
    if (WARP_LOCAL) __syncwarp(); else __syncthreads();
  }
}

// fft_3phase of gpe_fast.cuh on line pairs (n = 512).
template <int N, int AX, bool INV, bool TAIL>
__device__ __forceinline__ void pack_3phase(C2 (&v)[PackCfg<N>::V], ulonglong2* ex, const float4* twa, const float4* twb) {
  constexpr int LP = PackCfg<N>::LP, T = PackCfg<N>::T, Q = PackCfg<N>::Q;
  constexpr int RD = 8, A = 64;
  static_assert(N == RD * RD * RD, "three-phase layout");
  constexpr bool WARP_LOCAL = AX == FZ && T == 32 * LP;
  auto e1 = [](int lp, int k3, int p) { return AX == FZ ? (lp * RD + k3) * A + p : (k3 * A + p) * LP + lp; };
  auto e2 = [](int lp, int k3, int k1, int p1) {
    return AX == FZ ? (lp * RD + k1) * A + 8 * p1 + (k3 ^ p1) : ((k1 * RD + k3) * RD + p1) * LP + lp;
  };
  auto sync = [] { if (WARP_LOCAL) __syncwarp(); else __syncthreads(); };
#pragma unroll
  for (int s = 0; s < Q; ++s) {
    int lp, p;
    pack_slot<N, AX>(threadIdx.x + s * T, A, lp, p);
    C2* x = v + s * RD;
    Dft2<RD, INV>::run(x);
#pragma unroll
    for (int k3 = 1; k3 < RD; ++k3) x[k3] = tw2<INV>(x[k3], twa[k3 * A + p]);
#pragma unroll
    for (int k3 = 0; k3 < RD; ++k3) ex_store(ex + e1(lp, k3, p), x[k3]);
  }
  sync();
#pragma unroll
  for (int s = 0; s < Q; ++s) {
    int lp, q;
    pack_slot<N, AX>(threadIdx.x + s * T, A, lp, q);
    const int p1 = q & 7, k3 = q >> 3;
#pragma unroll
    for (int p2 = 0; p2 < RD; ++p2) v[s * RD + p2] = ex_load(ex + e1(lp, k3, p1 + RD * p2));
  }
  sync();
#pragma unroll
  for (int s = 0; s < Q; ++s) Dft2<RD, INV>::run(v + s * RD);
  {
    int lp0, q0;
    pack_slot<N, AX>(threadIdx.x, A, lp0, q0);
    const int p1 = q0 & 7;   // (the same in every slot of a thread: slots are 32 lanes apart)
#pragma unroll
    for (int k1 = 1; k1 < RD; ++k1) {
      const float4 w = twb[k1 * RD + p1];
#pragma unroll
      for (int s = 0; s < Q; ++s) v[s * RD + k1] = tw2<INV>(v[s * RD + k1], w);
    }
  }
#pragma unroll
  for (int s = 0; s < Q; ++s) {
    int lp, q;
    pack_slot<N, AX>(threadIdx.x + s * T, A, lp, q);
    const int p1 = q & 7, k3 = q >> 3;
#pragma unroll
    for (int k1 = 0; k1 < RD; ++k1) ex_store(ex + e2(lp, k3, k1, p1), v[s * RD + k1]);
  }
  sync();
#pragma unroll
  for (int s = 0; s < Q; ++s) {
    int lp, q;
    pack_slot<N, AX>(threadIdx.x + s * T, A, lp, q);
    const int k3 = q & 7, k1 = q >> 3;
#pragma unroll
    for (int p1 = 0; p1 < RD; ++p1) v[s * RD + p1] = ex_load(ex + e2(lp, k3, k1, p1));
    Dft2<RD, INV>::run(v + s * RD);
  }
  if (TAIL) sync();
}

// ---------------------------------------------------------------- pointwise on pairs
// One element's local factor with every range of the phase (half_all's two passes): the
// elements outside the packed short series, and array potentials.
template <bool REAL, bool ARR, bool TWO>
__device__ __forceinline__ float2 half_one(float2 x, float V, float g, float beta, float h) {
  const float p = local_phase<true, ARR, TWO>(x, V, g, beta, h);
  if (!REAL) {
    const float em = fabsf(p) <= 0.125f ? expm1_tiny(-p) : fabsf(p) <= 0.5f ? expm1_series(-p) : expm1f(-p);
    return make_float2(fmaf(x.x, em, x.x), fmaf(x.y, em, x.y));
  }
  float sn, cm1;
  if (fabsf(p) <= 0.125f) {
    sin_cosm1_tiny(p, sn, cm1);
  } else if (fabsf(p) <= 0.78539816f) {
    sin_cosm1_series(p, sn, cm1);
  } else {
    float sh, ch;
    sincosf(0.5f * p, &sh, &ch);
    cm1 = -2.0f * sh * sh;
    sn = 2.0f * sh * ch;
  }
  if (ARR) times_amplitude<true>(expm1f(TWO ? g + g : g), cm1, sn);
  return make_float2(fmaf(x.x, cm1, fmaf(x.y, sn, x.x)), fmaf(x.y, cm1, fmaf(-x.x, sn, x.y)));
}

// half_all of gpe_fast.cuh on pairs: layout LANES x VALS, element m = lane + LANES*a of
// lines 2 lp, 2 lp + 1.
template <int N, bool REAL, bool ARR, bool TWO>
__device__ __forceinline__ void pack_half(C2 (&v)[PackCfg<N>::V], const FastTile<N, FZ, float>& tl, const Phys& ph,
                                          const FastTables<float>& tb, const float* ctab, float beta, float h) {
  constexpr int T = PackCfg<N>::T, LANES = PackCfg<N>::LANES, VALS = PackCfg<N>::VALS, SLOTS = PackCfg<N>::Q;
  static_assert(SLOTS * VALS <= 32, "pending mask");
  unsigned pend = 0;
#pragma unroll
  for (int s = 0; s < SLOTS; ++s) {
    int lp, lane;
    pack_slot<N, FZ>(threadIdx.x + s * T, LANES, lp, lane);
    const float2 c = *(const float2*)(ctab + 2 * lp);
    if constexpr (ARR) {
      const long long row = tl.base + 2LL * lp * N;
#pragma unroll
      for (int a = 0; a < VALS; ++a) {
        const int m = lane + LANES * a;
        const float* re = (const float*)ph.vre;
        const float* im = (const float*)ph.vim;
        const float2 x = unpack(v[s * VALS + a].x), y = unpack(v[s * VALS + a].y);
        float2 r[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const float va = re ? re[row + q * N + m] : 0.0f, g = im ? im[row + q * N + m] * h : 0.0f;
          float Vq = tb.vz[m] + (q ? c.y : c.x);
          Vq = TWO ? fmaf(va, h + h, Vq) : Vq + va;
          r[q] = half_one<REAL, true, TWO>(q ? make_float2(x.y, y.y) : make_float2(x.x, y.x), Vq, g, beta, h);
        }
        v[s * VALS + a] = c2(f2(r[0].x, r[1].x), f2(r[0].y, r[1].y));
      }
    } else {
    const F2 cc = f2(c.x, c.y), bb = f2(beta);
#pragma unroll
    for (int a = 0; a < VALS; ++a) {
      const int e = s * VALS + a;
      const F2 Vp = f2(tb.vz[lane + LANES * a]) + cc;
      const C2 x = v[e];
      const F2 rho = fma2(x.x, x.x, x.y * x.y);
      F2 p = fma2(bb, rho, Vp);
      if (!TWO) p = p * f2(h);
      const float2 ps = unpack(p);
      if (fmaxf(fabsf(ps.x), fabsf(ps.y)) <= 0.125f && ps.x == ps.x && ps.y == ps.y) {
        if (!REAL) {
          const F2 n = -p;
          const F2 em = n * fma2(n, fma2(n, fma2(n, fma2(n, fma2(n, f2(1.3888888888888889e-03f),
                        f2(8.3333333333333333e-03f)), f2(4.1666666666666667e-02f)), f2(1.6666666666666667e-01f)),
                        f2(0.5f)), f2(1.0f));
          v[e] = c2(fma2(x.x, em, x.x), fma2(x.y, em, x.y));
        } else {
          const F2 z = p * p;
          const F2 sn = p * fma2(z, fma2(z, f2(8.3333333333333333e-03f), f2(-1.6666666666666667e-01f)), f2(1.0f));
          const F2 cm1 = z * fma2(z, fma2(z, f2(-1.3888888888888889e-03f), f2(4.1666666666666667e-02f)), f2(-0.5f));
          v[e] = c2(fma2(x.x, cm1, fma2(x.y, sn, x.x)), fma2(x.y, cm1, fma2(-x.x, sn, x.y)));
        }
      } else {
        pend |= 1u << e;
      }
    }
    }
  }
  if constexpr (!ARR) {
    if (!__any_sync(0xffffffffu, pend != 0)) return;
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
      int lp, lane;
      pack_slot<N, FZ>(threadIdx.x + s * T, LANES, lp, lane);
      const float2 c = *(const float2*)(ctab + 2 * lp);
#pragma unroll
      for (int a = 0; a < VALS; ++a) {
        const int e = s * VALS + a;
        if (!((pend >> e) & 1)) continue;
        const float2 x = unpack(v[e].x), y = unpack(v[e].y);
        const float vz = tb.vz[lane + LANES * a];
        const float2 r0 = half_one<REAL, false, TWO>(make_float2(x.x, y.x), vz + c.x, 0.0f, beta, h);
        const float2 r1 = half_one<REAL, false, TWO>(make_float2(x.y, y.y), vz + c.y, 0.0f, beta, h);
        v[e] = c2(f2(r0.x, r1.x), f2(r0.y, r1.y));
      }
    }
  }
}

template <int N>
__device__ __forceinline__ void pack_half_dispatch(C2 (&v)[PackCfg<N>::V], const FastTile<N, FZ, float>& tl, const Phys& ph,
                                                   const FastTables<float>& tb) {
  const float beta = (float)ph.beta, h = (float)(ph.dt * 0.5);
  const bool arr = ph.vre != nullptr || ph.vim != nullptr;
  if (ph.kind == 1) {
    if (arr) pack_half<N, true, true, false>(v, tl, ph, tb, tb.c1, beta, h);
    else pack_half<N, true, false, false>(v, tl, ph, tb, tb.c1, beta, h);
  } else {
    if (arr) pack_half<N, false, true, false>(v, tl, ph, tb, tb.c1, beta, h);
    else pack_half<N, false, false, false>(v, tl, ph, tb, tb.c1, beta, h);
  }
}

template <int N, bool REAL, bool CUT>
__device__ __forceinline__ void pack_kin(C2 (&v)[PackCfg<N>::V], const Phys& ph, const FastTables<float>& tb) {
  constexpr int T = PackCfg<N>::T, LANES = PackCfg<N>::LANES, VALS = PackCfg<N>::VALS, SLOTS = PackCfg<N>::Q;
#pragma unroll
  for (int s = 0; s < SLOTS; ++s) {
    int lp, lane;
    pack_slot<N, FX>(threadIdx.x + s * T, LANES, lp, lane);
#pragma unroll
    for (int a = 0; a < VALS; ++a) {
      const int e = s * VALS + a, i = lane + LANES * a;
      const float2 x = unpack(v[e].x), y = unpack(v[e].y);
      const float2 r0 = fast_kin<float, REAL, CUT>(ph, tb, make_float2(x.x, y.x), i, 2 * lp);
      const float2 r1 = fast_kin<float, REAL, CUT>(ph, tb, make_float2(x.y, y.y), i, 2 * lp + 1);
      v[e] = c2(f2(r0.x, r1.x), f2(r0.y, r1.y));
    }
  }
}

// ---------------------------------------------------------------- loads and stores
// (past L1, which holds the twiddles) vec: y/x rows by 16-byte accesses (psi aligned to 16 bytes), else one line at a time
template <int N, int AX>
__device__ __forceinline__ void pack_load(C2 (&v)[PackCfg<N>::V], const FastTile<N, AX, float>& tl,
                                          const float2* __restrict__ src, bool vec) {
  constexpr int T = PackCfg<N>::T, LANES = PackCfg<N>::LANES, VALS = PackCfg<N>::VALS, SLOTS = PackCfg<N>::Q;
#pragma unroll
  for (int s = 0; s < SLOTS; ++s) {
    int lp, lane;
    pack_slot<N, AX>(threadIdx.x + s * T, LANES, lp, lane);
    const float2* p = src + tl.gidx(2 * lp, lane);
    if (AX != FZ && vec) {
#pragma unroll
      for (int a = 0; a < VALS; ++a) {
        const float4 q = __ldcg((const float4*)(p + (long long)(LANES * a) * tl.nstride));
        v[s * VALS + a] = c2(f2(q.x, q.z), f2(q.y, q.w));
      }
    } else {
#pragma unroll
      for (int a = 0; a < VALS; ++a) {
        const float2 f = __ldcg(p + (long long)(LANES * a) * tl.nstride);
        const float2 g = __ldcg(p + (long long)(LANES * a) * tl.nstride + tl.lstride);
        v[s * VALS + a] = c2(f2(f.x, g.x), f2(f.y, g.y));
      }
    }
  }
}

template <int N, int AX>
__device__ __forceinline__ void pack_store(const C2 (&v)[PackCfg<N>::V], const FastTile<N, AX, float>& tl,
                                           float2* __restrict__ dst, bool vec) {
  constexpr int T = PackCfg<N>::T, LANES = PackCfg<N>::LANES, VALS = PackCfg<N>::VALS, SLOTS = PackCfg<N>::Q;
#pragma unroll
  for (int s = 0; s < SLOTS; ++s) {
    int lp, lane;
    pack_slot<N, AX>(threadIdx.x + s * T, LANES, lp, lane);
    float2* p = dst + tl.gidx(2 * lp, lane);
#pragma unroll
    for (int a = 0; a < VALS; ++a) {
      const float2 x = unpack(v[s * VALS + a].x), y = unpack(v[s * VALS + a].y);
      float2* q = p + (long long)(LANES * a) * tl.nstride;
      if (AX != FZ && vec) {
        *(float4*)q = make_float4(x.x, y.x, x.y, y.y);
      } else {
        q[0] = make_float2(x.x, y.x);
        q[tl.lstride] = make_float2(x.y, y.y);
      }
    }
  }
}

// ---------------------------------------------------------------- the sweep
template <int N, int AX, int MODE>
__device__ __forceinline__ void pack_body(const Phys& ph, const Sweep& sw, const FastOps& op, int tile, int ntiles) {
  constexpr int L = PackCfg<N>::L;
  constexpr bool ZM = MODE == FM_Z1 || MODE == FM_Z2 || MODE == FM_Z21;
  constexpr bool THREE = PackCfg<N>::THREE;
  constexpr bool TWO_FFT = MODE == FM_Z21 || MODE == FM_XKIN;
  griddep_launch_dependents();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ulonglong2* ex = (ulonglong2*)smem_raw;
  float4* tw = (float4*)(smem_raw + PackCfg<N>::EXB);
  unsigned char* tail = (unsigned char*)(tw + PackCfg<N>::TW);
  Acc* red = (Acc*)tail;
  FastTables<float> tb;
  tb.kx = (double2*)tail;
  tb.kyz = tb.kx + N;
  tb.kx2 = (double*)(tb.kyz + L);
  tb.kyz2 = tb.kx2 + N;
  tb.vz = (float*)(red + 32);
  tb.c1 = tb.vz + N;
  tb.c2 = tb.c1 + L;
  tb.c12 = tb.c2 + L;
  // (plan constants: copied past the registers, in flight with the tile's loads)
  for (int q = threadIdx.x; q < PackCfg<N>::TW; q += PackCfg<N>::T) cp_async16(tw + q, (const float4*)sw.twp + q);
  const FastTile<N, AX, float> tl(tile);
  griddep_wait();
  float sc_mul = 1.0f;
  if (MODE == FM_Z1 && op.scale) sc_mul = (float)__ldcg(sw.scale + 1);
  const bool vec = op.vec != 0;
  constexpr int V = PackCfg<N>::V;
  C2 v[V];
  pack_load<N, AX>(v, tl, (const float2*)sw.src, vec);
  if (op.pf > 0) {
    const int next = op.rev ? tile - op.pf : tile + op.pf;
    if (next >= 0 && next < ntiles) fast_prefetch_l2<N, AX, float, PackCfg<N>::T>(FastTile<N, AX, float>(next), sw.src);
  }
  if (ZM) z_tables<N, float, PackCfg<N>::T>(ph, sw, tl.a0, tb, MODE == FM_Z21);
  if (MODE == FM_XKIN) x_tables<N, float, PackCfg<N>::T>(ph, tl.a0, tl.b0, tb);
  cp_async_wait();
  __syncthreads();   // twiddles and tables visible
  if constexpr (MODE == FM_Z1) {
    if (op.scale) {
#pragma unroll
      for (int e = 0; e < V; ++e) v[e] = c2(v[e].x * f2(sc_mul), v[e].y * f2(sc_mul));
    }
    pack_half_dispatch<N>(v, tl, ph, tb);
  }
  auto first = [&](auto inv) {
    constexpr bool INV = decltype(inv)::value;
    if constexpr (THREE) pack_3phase<N, AX, INV, TWO_FFT>(v, ex, tw, tw + N);
    else pack_2phase<N, AX, INV, TWO_FFT>(v, ex, tw);
  };
  using std::integral_constant;
  if constexpr (MODE == FM_Z2 || MODE == FM_Z21) {
    first(integral_constant<bool, true>{});
  } else if constexpr (MODE == FM_PLAIN) {
    if (op.inv1) first(integral_constant<bool, true>{});
    else first(integral_constant<bool, false>{});
  } else {
    first(integral_constant<bool, false>{});
  }
  if constexpr (TWO_FFT) {
    if constexpr (MODE == FM_Z21) {
      const float h = (float)(ph.dt * 0.5), b2 = (float)(2.0 * ph.beta) * h;
      if (ph.vre == nullptr && ph.vim == nullptr)
        pack_half<N, true, false, true>(v, tl, ph, tb, tb.c12, b2, h);
      else
        pack_half<N, true, true, true>(v, tl, ph, tb, tb.c12, b2, h);
    } else if (ph.kind == 1) {
      if (ph.kcut) pack_kin<N, true, true>(v, ph, tb);
      else pack_kin<N, true, false>(v, ph, tb);
    } else {
      pack_kin<N, false, false>(v, ph, tb);
    }
    constexpr bool INV = MODE == FM_XKIN;
    if constexpr (THREE) pack_3phase<N, AX, INV, false>(v, ex, tw, tw + N);
    else pack_2phase<N, AX, INV, false>(v, ex, tw);
    pack_store<N, AX>(v, tl, (float2*)sw.dst, vec);
  } else {
    if constexpr (MODE == FM_Z2) pack_half_dispatch<N>(v, tl, ph, tb);
    pack_store<N, AX>(v, tl, (float2*)sw.dst, vec);
    if (MODE == FM_Z2 && op.norm) {
      // a thread's values of a line summed in plain FP64 (fixed order), then compensated
      Acc a[1];
#pragma unroll
      for (int s = 0; s < PackCfg<N>::Q; ++s) {
        double s0 = 0.0, s1 = 0.0;
#pragma unroll
        for (int e = s * PackCfg<N>::VALS; e < (s + 1) * PackCfg<N>::VALS; ++e) {
          const float2 x = unpack(v[e].x), y = unpack(v[e].y);
          s0 = fma((double)x.x, (double)x.x, fma((double)y.x, (double)y.x, s0));
          s1 = fma((double)x.y, (double)x.y, fma((double)y.y, (double)y.y, s1));
        }
        a[0].add(s0);
        a[0].add(s1);
      }
      block_merge<1>(a, red);
      norm_finish_n(ph, sw, a[0], red, tile, ntiles);
    }
  }
}

// Resident blocks per SM asked of the register allocation: 512 threads at 128 registers
// (two lines of 16 values take 64).  With 96 or 80 registers (640, 768 threads) the loads of
// a tile no longer fit in flight together: 512^3 2111 -> 2806 us per step at 768.  (2111 was with twiddle
// entries twice the size; 1944 now.)
template <int N, int MODE> struct PackBounds {
  static constexpr int value = 512 / PackCfg<N>::T;
};

template <int N, int AX, int MODE>
__global__ void __launch_bounds__(PackCfg<N>::T, PackBounds<N, MODE>::value ? PackBounds<N, MODE>::value : 1)
k_pack(Phys ph, Sweep sw, FastOps op) {
  pack_body<N, AX, MODE>(ph, sw, op, tile_of(op), gridDim.x);
}

// Batched launch: blockIdx.y selects the instance (structs staged in shared memory).
template <int N, int AX, int MODE>
__global__ void __launch_bounds__(PackCfg<N>::T, PackBounds<N, MODE>::value ? PackBounds<N, MODE>::value : 1)
k_pack_batch(const Phys* __restrict__ phs, const Sweep* __restrict__ sws, FastOps op) {
  __shared__ Phys ph;
  __shared__ Sweep sw;
  copy_words(&ph, phs + blockIdx.y);
  copy_words(&sw, sws + blockIdx.y);
  __syncthreads();
  if (batch_frozen(sw.live)) return;
  pack_body<N, AX, MODE>(ph, sw, op, tile_of(op), gridDim.x);
}

// Sweeps that take two lines per thread: the steps' at n = 512; at n = 256 the fused z sweep and
// the x sweep (transforms, reductions and the y sweeps at 256, which HBM bounds, keep one line
// per thread; so do Z1 and Z2 there, which run the arithmetic of the plane-fused launches to
// the last bit).  Per step, 512^3 stirred 2294 -> 1944 us (z 589 -> 501, y 427 -> 377, x 770 -> 696);
// 256^3 stirred 207.8 -> 199.9 (z 69.2 -> 62.7, x 70.0 -> 66.1).  At n = 128 there are too few
// warps for it: 31.9 -> 36.8.
constexpr bool pack_sweep(int n, int mode) {
  if (n == 256) return mode == FM_Z21 || mode == FM_XKIN;
  return n == 512 && (mode == FM_PLAIN || mode == FM_Z1 || mode == FM_Z2 || mode == FM_Z21 || mode == FM_XKIN);
}

}  // namespace gpe
