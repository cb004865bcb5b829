// gpe_line.cuh -- sweep kernels for any grid side n = r0 r1 .. rP-1 (two or more radices
// of at most 16, chosen on the host), sm_100a.
//
// The register-resident sweeps of gpe_fast.cuh fix the side at compile time.  These take
// it at run time and keep what makes those fast: values go from HBM into the registers
// of the first butterflies, cross shared memory once between two phases, and leave for
// HBM from the registers of the last ones, with the pointwise physics applied there.
//
// A transform runs in place: with the input index m = d0 nb0 + d1 (..) + .. + dP-1 as
// mixed-radix digits, phase p replaces digit dp by the output digit kp, and the frequency
// is k = k0 + r0 k1 + r0 r1 k2 + ..  The twiddles between two phases can multiply the
// outputs of the first (W^(kp (later digits)) of its sub-transform's length) or the inputs
// of the second (W^(dp (earlier output digits))).  Sweeps with two transforms take the
// first form: the transform back runs the same phases in reverse order with the same
// tables, so the sweep turns around in the registers of phase P-1 and needs no reordering
// pass.  Sweeps with one transform take the second form, which is the arithmetic of the
// Stockham passes of gpe_fft.cuh: with their radices every value is the same bit for bit
// (complex64 transforms and reductions run so).  Inverses are conj(FFT(conj(x))).  Each
// butterfly rewrites only the shared positions it read, so a phase costs one barrier.
//
// Tiles are L lines: z tiles L consecutive lines (lanes walk along the line; digit strides
// padded to odd numbers keep the accesses of the last phase, strided by S0, free of bank
// conflicts), y/x tiles L adjacent z's of one row (lanes walk across the lines).  The
// twiddles come from per-phase tables [k - 1][column] laid out by the host in the order
// the lanes read them, through L1.
//
// Against the Stockham sweeps these replace (run-time strides and divisions per element,
// every stage through shared memory, five sweeps per step instead of four): 200^3
// complex64, 6 imaginary-time steps 7343 -> 1448 us; 512^3 complex128, one stirred step
// 24.6 -> 5.6 ms; 294^3 complex64 with array potentials, 2 steps 14.0 -> 1.84 ms.  Bound
// by the latency of the loads and barriers at 16 (complex128, radices above 8) to 32 warps
// per SM and, in complex64, by issue.
//
// Sums over the state add every element to a compensated accumulator, as the Stockham
// sweeps do.  Error of five complex128 steps against 80-bit references, over 27 sides from 30
// to 125: 0.97 times the Stockham sweeps' (0.74 to 1.13).
#pragma once
#include "gpe_fast.cuh"
#include "gpe_line_plan.h"

namespace gpe {

constexpr int FM_LZ = 7;          // forward transform, angular-momentum sums, no store (y and x sweeps)

// b / d for b, d < 2^16 by the rounded-up reciprocal mg = ceil(2^32 / d)
__device__ __forceinline__ int div_mg(int b, unsigned mg) { return mg ? (int)__umulhi((unsigned)b, mg) : b; }

// RMAX: largest radix of the launch's geometry (8 or 16).  The radices up to 8 need half the
// registers of 16, so their own instantiations run twice the warps per SM.
template <int RMAX, typename F> __device__ __forceinline__ void by_radix(int r, F&& f) {
  switch (r) {
    case 2: f(std::integral_constant<int, 2>{}); return;
    case 3: f(std::integral_constant<int, 3>{}); return;
    case 4: f(std::integral_constant<int, 4>{}); return;
    case 5: f(std::integral_constant<int, 5>{}); return;
    case 6: f(std::integral_constant<int, 6>{}); return;
    case 7: f(std::integral_constant<int, 7>{}); return;
    case 8: f(std::integral_constant<int, 8>{}); return;
    default: break;
  }
  if constexpr (RMAX > 8) {
    switch (r) {
      case 9: f(std::integral_constant<int, 9>{}); return;
      case 10: f(std::integral_constant<int, 10>{}); return;
      case 11: f(std::integral_constant<int, 11>{}); return;
      case 12: f(std::integral_constant<int, 12>{}); return;
      case 13: f(std::integral_constant<int, 13>{}); return;
      case 14: f(std::integral_constant<int, 14>{}); return;
      case 15: f(std::integral_constant<int, 15>{}); return;
      default: f(std::integral_constant<int, 16>{}); return;
    }
  }
}

// DFT of a phase: the small DFTs of gpe_fft.cuh; prime radices by conjugate pairs, or
// (g.direct) by the direct sum of the Stockham passes.
template <int R> struct LineDft : Dft<R> {};
template <> struct LineDft<7>  : DftPrime<7> {};
template <> struct LineDft<11> : DftPrime<11> {};
template <> struct LineDft<13> : DftPrime<13> {};
template <> struct LineDft<14> : DftSplitG<7, 2, DftPrime<7>, Dft<2>> {};
template <int RAD, bool DIRECT, typename C> __device__ __forceinline__ void line_dft(const LineGeo& g, C* v) {
  if constexpr (DIRECT && (RAD == 7 || RAD == 11 || RAD == 13)) {
    if (g.direct) {
      DftDirect<RAD>::run(v, (const C*)g.w, (const C*)g.w + g.n, g.n / RAD);
      return;
    }
  }
  LineDft<RAD>::run(v, (const C*)nullptr, (const C*)nullptr, 0);
}

// ---------------------------------------------------------------- pointwise physics
// What the pointwise stages of one tile need besides Phys.
template <typename R>
struct LineCx {
  const R* vz;            // static potential along z (global, plan constant)
  const R* c1;            // [L] line part of the potential at t1 (shared)
  const R* c12;           // [L] (line parts at t1 and t2) dt/2 (shared; fused half-steps)
  const double2* kyz;     // [L] kinetic factor of the line, with 1/M (shared)
  const double* kyz2;     // [L] k_y^2 + k_z^2 of the line (shared)
  const R* vd1;           // dynamic potential with z terms at t1 (t2), per point (global, null: none)
  const R* vd2;
  long long row0;         // z tiles: global index of line 0
  int n;
};

// One local half-step of the RAD elements m = q + a*nb of line l (TWO: two consecutive
// real-time half-steps as one rotation, see half_all in gpe_fast.cuh for why that is
// exact), a few at a time with their potentials loaded together.
template <typename R, bool ARR, bool TWO, int RAD>
__device__ __forceinline__ void line_half_arr(const Phys& ph, const LineCx<R>& cx, typename Cx<R>::T (&v)[RAD], int l,
                                              int q, int nb) {
  constexpr int U = sizeof(R) == 8 || ARR ? local_unroll(RAD) : 1;
  const R h = (R)(ph.dt * 0.5), beta = TWO ? (R)(2.0 * ph.beta) * h : (R)ph.beta;
  const R c = TWO ? cx.c12[l] : cx.c1[l];
  const long long row = cx.row0 + (long long)l * cx.n + q;
#pragma unroll
  for (int a0 = 0; a0 < RAD; a0 += U) {
    R V[U], g[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const R vz = cx.vz[q + (a0 + u) * nb];
      V[u] = TWO ? fma(vz, h + h, c) : vz + c;
      g[u] = (R)0;
      if (ARR) {
        const long long e = row + (a0 + u) * nb;
        if (cx.vd1) V[u] = TWO ? fma(cx.vd1[e] + cx.vd2[e], h, V[u]) : V[u] + cx.vd1[e];
        if (ph.vre) V[u] = TWO ? fma(((const R*)ph.vre)[e], h + h, V[u]) : V[u] + ((const R*)ph.vre)[e];
        if (ph.vim) g[u] = ((const R*)ph.vim)[e] * h;
      }
    }
    local_block<R, ARR, TWO, U>(v + a0, V, g, TWO || ph.kind == 1, beta, h);
  }
}
template <typename R, bool TWO, int RAD>
__device__ __forceinline__ void line_half(const Phys& ph, const LineCx<R>& cx, typename Cx<R>::T (&v)[RAD], int l,
                                          int q, int nb) {
  if (ph.vre || cx.vd1) line_half_arr<R, true, TWO, RAD>(ph, cx, v, l, q, nb);
  else line_half_arr<R, false, TWO, RAD>(ph, cx, v, l, q, nb);
}

// ---------------------------------------------------------------- the sweep
template <typename R, bool ZT, int MODE, int RMAX>
__device__ __forceinline__ void line_body(const Phys& ph, const Sweep& sw, const FastOps& op, const LineGeo& g,
                                          const LineShape& sh, int ax, int tile, int ntiles) {
  using C = typename Cx<R>::T;
  using TW = typename TwE<R>::T;
  constexpr bool TWO_FFT = MODE == FM_Z21 || MODE == FM_XKIN;
  constexpr bool ZM = MODE == FM_Z1 || MODE == FM_Z2 || MODE == FM_Z21 || MODE == FM_DIAGR;
  // one transform: twiddles before the phases; direct prime sums only exist in complex64
  constexpr bool DIT = !TWO_FFT;
  constexpr bool DIRECT = sizeof(R) == 4 && DIT && MODE != FM_Z1 && MODE != FM_Z2;
  constexpr bool SUMS = MODE == FM_DIAGR || MODE == FM_DIAGK || MODE == FM_LZ;
  griddep_launch_dependents();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n = g.n, L = sh.L, P = g.P, tid = threadIdx.x, T = blockDim.x;
  C* s = (C*)smem_raw;
  unsigned char* tail = smem_raw + (size_t)(ZT ? L * sh.pitch : g.span * L) * sizeof(C);
  LineCx<R> lc;
  R* c1 = (R*)tail;
  R* c12 = c1 + L;
  double2* kyz = (double2*)tail;
  double* kyz2 = (double*)(kyz + L);
  Acc* red = (Acc*)(tail + ((size_t)L * 24 + 15) / 16 * 16);
  double* hist = (double*)(red + 32 * 4);
  lc.vz = (const R*)ph.vax + 2 * n;
  lc.c1 = c1;
  lc.c12 = c12;
  lc.vd1 = (const R*)sw.vd1;
  lc.vd2 = (const R*)sw.vd2;
  lc.kyz = kyz;
  lc.kyz2 = kyz2;
  lc.n = n;

  // the tile's lines
  int nlines, a0;                 // z: first line; y/x: the row (x of a y tile, y of an x tile)
  int z0 = 0;
  long long base, lstride, nstride;
  if (ZT) {
    a0 = tile * L;
    nlines = min(L, n * n - a0);
    base = (long long)a0 * n; lstride = n; nstride = 1;
  } else {
    a0 = tile / sh.tpr;
    z0 = (tile - a0 * sh.tpr) * L;
    nlines = min(L, n - z0);
    lstride = 1;
    if (ax == FY) { base = (long long)a0 * n * n + z0; nstride = n; }
    else { base = (long long)a0 * n + z0; nstride = (long long)n * n; }
  }
  lc.row0 = base;
  // psi, the renormalisation scale and the line table come from earlier launches
  griddep_wait();
  PwCtx<R> cx;
  if (MODE == FM_Z1 && op.scale) {
    cx.sc_div = __ldcg(sw.scale);
    cx.sc_rcp = __ldcg(sw.scale + 1);
    cx.sc_mul = (R)cx.sc_rcp;
  }
  // per-line tables
  if (ZM) {
    for (int l = tid; l < nlines; l += T) {
      const int gl = a0 + l, i = gl / n, j = gl - i * n;
      const R* vax = (const R*)ph.vax;
      const R stat = vax[i] + vax[n + j];
      R b1 = (R)0, b2 = (R)0;
      if (MODE == FM_DIAGR) {
        // (the beam's exponential apart: potential() adds it after the arrays)
        if (ph.kind == 1 && ph.beam) {
          const R dx = (R)(ph.x[i] - sw.bc1x), dy = (R)(ph.x[j] - sw.bc1y);
          c12[l] = rexp(-(dx * dx + dy * dy) * (R)ph.beam_inv_w2);
        }
      } else if (ph.kind == 1 && ph.beam) {
        const R dx = (R)(ph.x[i] - sw.bc1x), dy = (R)(ph.x[j] - sw.bc1y), iw = (R)ph.beam_inv_w2;
        b1 = (R)ph.beam_amp * rexp(-dx * dx * iw) * rexp(-dy * dy * iw);
        if (MODE == FM_Z21) {
          const R ex = (R)(ph.x[i] - sw.bc2x), ey = (R)(ph.x[j] - sw.bc2y);
          b2 = (R)ph.beam_amp * rexp(-ex * ex * iw) * rexp(-ey * ey * iw);
        }
      }
      if (ph.ltab) {
        const R* lt = (const R*)ph.ltab;
        b1 += lt[gl];
        if (MODE == FM_Z21) b2 += lt[(long long)n * n + gl];
      }
      c1[l] = stat + b1;
      if (MODE == FM_Z21) c12[l] = ((stat + b1) + (stat + b2)) * (R)(ph.dt * 0.5);
    }
  }
  if (MODE == FM_XKIN) {
    for (int l = tid; l < nlines; l += T) {
      const double2 a = ph.kin[a0], b = ph.kin[z0 + l];
      const double2 f = ph.kind == 0 ? make_double2(a.x * b.x, 0.0) : cmul(a, b);
      kyz[l] = make_double2(f.x * ph.inv_m, f.y * ph.inv_m);
      kyz2[l] = fma(ph.k[a0], ph.k[a0], __dmul_rn(ph.k[z0 + l], ph.k[z0 + l]));
    }
  }
  const int copies = MODE == FM_DIAGK && sw.hist ? hist_copies(sw.nbins, LINE_HIST) : 0;
  if (MODE == FM_DIAGK)
    for (int b = tid; b < copies * sw.nbins; b += T) hist[b] = 0.0;
  if (MODE == FM_Z1 || MODE == FM_DIAGR) __syncthreads();   // (other modes read the tables after a phase's barrier)

  const bool conj_in = MODE == FM_Z2 || MODE == FM_Z21 || (MODE == FM_PLAIN && op.inv1);
  auto at = [&](int l, int pos) { return ZT ? l * sh.pitch + pos : pos * L + l; };
  // butterfly b of phase p: line l and index q within the line; false past the tile's lines
  auto split = [&](int b, int p, int& l, int& q) {
    if (ZT) { l = div_mg(b, g.mg_nb[p]); q = b - l * g.nb[p]; return true; }
    q = div_mg(b, sh.mg_L);
    l = b - q * L;
    return l < nlines;
  };
  auto count = [&](int p) { return g.nb[p] * (ZT ? nlines : L); };
  const C* __restrict__ src = (const C*)sw.src;
  C* __restrict__ dst = (C*)sw.dst;

  // phase 0: HBM -> registers -> shared memory
  by_radix<RMAX>(g.r[0], [&](auto rc) {
    constexpr int RAD = decltype(rc)::value;
    const int nb = g.nb[0], total = count(0), S0 = g.S[0];
    const TW* tw = (const TW*)g.tw[0];
    const long long st = (long long)nb * nstride;
    for (int b = tid; b < total; b += T) {
      int l, q;
      if (!split(b, 0, l, q)) continue;
      const C* p = src + base + (long long)l * lstride + (long long)q * nstride;
      C v[RAD];
#pragma unroll
      for (int a = 0; a < RAD; ++a) v[a] = __ldcg(p + a * st);   // (past L1, which holds the tables)
      if (conj_in) {
#pragma unroll
        for (int a = 0; a < RAD; ++a) v[a].y = -v[a].y;
      }
      if (MODE == FM_Z1) {
        if (op.scale) {
#pragma unroll
          for (int a = 0; a < RAD; ++a) {
            if (sizeof(R) == 8) {
              v[a].x = (R)div_by((double)v[a].x, cx.sc_div, cx.sc_rcp);
              v[a].y = (R)div_by((double)v[a].y, cx.sc_div, cx.sc_rcp);
            } else {
              v[a].x *= cx.sc_mul;
              v[a].y *= cx.sc_mul;
            }
          }
        }
        line_half<R, false, RAD>(ph, lc, v, l, q, nb);
      }
      if (MODE == FM_DIAGR) {
#pragma unroll
        for (int a = 0; a < RAD; ++a) {
          const int m = q + a * nb;
          const double rho = (double)v[a].x * v[a].x + (double)v[a].y * v[a].y;
          R V = lc.vz[m] + c1[l];
          if (ph.vre) V += ((const R*)ph.vre)[lc.row0 + (long long)l * n + m];
          if (ph.kind == 1 && ph.beam) V += (R)ph.beam_amp * c12[l];
          if (lc.vd1) V += lc.vd1[lc.row0 + (long long)l * n + m];
          cx.acc[0].add(rho);
          cx.acc[1].add((double)V * rho);
          cx.acc[2].add(rho * rho);
        }
      }
      line_dft<RAD, DIRECT>(g, v);
      if (!DIT) {
#pragma unroll
        for (int k = 1; k < RAD; ++k) v[k] = tw_apply(v[k], tw[(k - 1) * nb + q]);
      }
#pragma unroll
      for (int k = 0; k < RAD; ++k) s[at(l, q + k * S0)] = v[k];
    }
  });
  __syncthreads();
  // middle phases, in place
  for (int p = 1; p < P - 1; ++p) {
    by_radix<RMAX>(g.r[p], [&](auto rc) {
      constexpr int RAD = decltype(rc)::value;
      // (twiddle row length and this butterfly's place in it)
      const int total = count(p), S = g.S[p], row = DIT ? g.np[p] : g.nl[p];
      const TW* tw = (const TW*)(DIT ? g.twi[p] : g.tw[p]);
      for (int b = tid; b < total; b += T) {
        int l, q;
        if (!split(b, p, l, q)) continue;
        const int2 f = ((const int2*)g.bf[p])[q];
        const int at_row = DIT ? f.y >> 16 : f.y & 0xffff;
        C v[RAD];
#pragma unroll
        for (int a = 0; a < RAD; ++a) v[a] = s[at(l, f.x + a * S)];
        if (DIT) {
#pragma unroll
          for (int a = 1; a < RAD; ++a) v[a] = tw_apply(v[a], tw[(a - 1) * row + at_row]);
        }
        line_dft<RAD, DIRECT>(g, v);
        if (!DIT) {
#pragma unroll
          for (int k = 1; k < RAD; ++k) v[k] = tw_apply(v[k], tw[(k - 1) * row + at_row]);
        }
#pragma unroll
        for (int k = 0; k < RAD; ++k) s[at(l, f.x + k * S)] = v[k];
      }
    });
    __syncthreads();
  }
  // last phase: shared memory -> registers, pointwise, then HBM or the transform back
  by_radix<RMAX>(g.r[P - 1], [&](auto rc) {
    constexpr int RAD = decltype(rc)::value;
    const int nb = g.nb[P - 1], total = count(P - 1);
    const int2* bf = (const int2*)g.bf[P - 1];
    const TW* twi = (const TW*)g.twi[P - 1];
    for (int b = tid; b < total; b += T) {
      int l, q;
      if (!split(b, P - 1, l, q)) continue;
      const int f = bf[q].x;
      C v[RAD];
#pragma unroll
      for (int a = 0; a < RAD; ++a) v[a] = s[at(l, f + a)];
      if (DIT) {
#pragma unroll
        for (int a = 1; a < RAD; ++a) v[a] = tw_apply(v[a], twi[(a - 1) * nb + q]);
      }
      line_dft<RAD, DIRECT>(g, v);
      if (TWO_FFT) {
        if (MODE == FM_Z21) {
#pragma unroll
          for (int a = 0; a < RAD; ++a) v[a].y = -v[a].y;
          line_half<R, true, RAD>(ph, lc, v, l, q, nb);
        } else {
          const double2 fl = kyz[l];
#pragma unroll
          for (int a = 0; a < RAD; ++a) {
            const int i = q + a * nb;
            const double2 fx = ph.kin[i];
            const double vx = v[a].x, vy = v[a].y;
            if (ph.kind == 0) {
              const double w = fx.x * fl.x;
              v[a] = mk((R)(vx * w), -(R)(vy * w));     // (conjugated: the inverse starts here)
            } else {
              const double wx = fx.x * fl.x - fx.y * fl.y, wy = fx.x * fl.y + fx.y * fl.x;
              v[a] = mk((R)(vx * wx - vy * wy), -(R)(vx * wy + vy * wx));
              // (fused operations named: the rounding of this sum decides which modes of exactly
              // the cutoff's length stay, and must not depend on the compiler)
              if (ph.kcut && fma(ph.k[i], ph.k[i], kyz2[l]) > ph.kcut2) v[a] = mk((R)0, (R)0);
            }
          }
        }
        line_dft<RAD, DIRECT>(g, v);
#pragma unroll
        for (int a = 0; a < RAD; ++a) s[at(l, f + a)] = v[a];
      } else {
        if (conj_in) {
#pragma unroll
          for (int a = 0; a < RAD; ++a) v[a].y = -v[a].y;
        }
        if (MODE == FM_PLAIN && op.invm) {
#pragma unroll
          for (int a = 0; a < RAD; ++a) { v[a].x *= (R)ph.inv_m; v[a].y *= (R)ph.inv_m; }
        }
        if (MODE == FM_Z2) {
          line_half<R, false, RAD>(ph, lc, v, l, q, nb);
          if (op.norm) {
#pragma unroll
            for (int a = 0; a < RAD; ++a) cx.acc[0].add((double)v[a].x * v[a].x + (double)v[a].y * v[a].y);
          }
        }
        if (MODE == FM_DIAGK) {
#pragma unroll
          for (int a = 0; a < RAD; ++a) {
            const double kk = kk_ref(ph.k[q + a * nb], ph.k[a0], ph.k[z0 + l]);
            const double w = (double)v[a].x * v[a].x + (double)v[a].y * v[a].y;
            cx.acc[3].add(kk * w);
            if (sw.hist)
              atomicAdd(hist + (l & (copies - 1)) * sw.nbins + shell_of(kk, sw.shell_t, sw.inv_shell, sw.nbins), w);
          }
        } else if (MODE == FM_LZ) {
          // y sweep: sum x k_y |v|^2; x sweep: sum y k_x |v|^2 (a0 is the other axis' index)
#pragma unroll
          for (int a = 0; a < RAD; ++a)
            cx.acc[3].add(ph.x[a0] * ph.k[q + a * nb] * ((double)v[a].x * v[a].x + (double)v[a].y * v[a].y));
        } else {
          C* p = dst + base + (long long)l * lstride + (long long)q * nstride;
          const long long st = (long long)nb * nstride;
#pragma unroll
          for (int a = 0; a < RAD; ++a) p[a * st] = v[a];
        }
      }
    }
  });
  if (TWO_FFT) {
    __syncthreads();
    for (int p = P - 2; p > 0; --p) {
      by_radix<RMAX>(g.r[p], [&](auto rc) {
        constexpr int RAD = decltype(rc)::value;
        const int total = count(p), S = g.S[p], nl = g.nl[p];
        const TW* tw = (const TW*)g.tw[p];
        for (int b = tid; b < total; b += T) {
          int l, q;
          if (!split(b, p, l, q)) continue;
          const int2 f = ((const int2*)g.bf[p])[q];
          C v[RAD];
#pragma unroll
          for (int k = 0; k < RAD; ++k) v[k] = s[at(l, f.x + k * S)];
#pragma unroll
          for (int k = 1; k < RAD; ++k) v[k] = tw_apply(v[k], tw[(k - 1) * nl + (f.y & 0xffff)]);
          line_dft<RAD, DIRECT>(g, v);
#pragma unroll
          for (int a = 0; a < RAD; ++a) s[at(l, f.x + a * S)] = v[a];
        }
      });
      __syncthreads();
    }
    by_radix<RMAX>(g.r[0], [&](auto rc) {
      constexpr int RAD = decltype(rc)::value;
      const int nb = g.nb[0], total = count(0), S0 = g.S[0];
      const TW* tw = (const TW*)g.tw[0];
      const long long st = (long long)nb * nstride;
      for (int b = tid; b < total; b += T) {
        int l, q;
        if (!split(b, 0, l, q)) continue;
        C v[RAD];
#pragma unroll
        for (int k = 0; k < RAD; ++k) v[k] = s[at(l, q + k * S0)];
#pragma unroll
        for (int k = 1; k < RAD; ++k) v[k] = tw_apply(v[k], tw[(k - 1) * nb + q]);
        line_dft<RAD, DIRECT>(g, v);
        C* p = dst + base + (long long)l * lstride + (long long)q * nstride;
#pragma unroll
        for (int a = 0; a < RAD; ++a) p[a * st] = MODE == FM_XKIN ? conj_<R>(v[a]) : v[a];
      }
    });
  }
  if (MODE == FM_Z2 && op.norm) {
    Acc a[1] = {cx.acc[0]};
    block_merge<1>(a, red);
    norm_finish_n(ph, sw, a[0], red, tile, ntiles);
  }
  if (SUMS) {
    // per-tile partials [tile][N, E_pot, E_int, E_kin or Lz]
    Acc a[4] = {cx.acc[0], cx.acc[1], cx.acc[2], cx.acc[3]};
    block_merge<4>(a, red);
    if (tid == 0)
      for (int q = 0; q < 4; ++q) sw.partial[(long long)tile * 4 + q] = a[q].value();
    if (MODE == FM_DIAGK && sw.hist) {
      __syncthreads();
      for (int b = tid; b < sw.nbins; b += T) {
        double h = hist[b];
        for (int c = 1; c < copies; ++c) h += hist[c * sw.nbins + b];
        sw.hist[(long long)tile * sw.nbins + b] = h;
      }
    }
  }
}

// Resident blocks.  Radices to 16: 64 registers in complex64 (80 measured slower: 200^3
// 236 -> 261 us per step), 128 in complex128.  Radices to 8: 64 registers, the complex128 x
// sweep with its FP64 factors 80 (per step, complex128: 200^3 450 -> 349 us at 4 blocks, 385
// at 3, 422 at 2; 512^3 x sweep 1.84 ms at 4 blocks, 1.49 at 3, where its 68 KB tiles allow
// no more; complex64 at 48 registers: 125^3 82 -> 90 us, 384^3 1.55 -> 1.48 ms).
template <typename R, int MODE, int RMAX> struct LineBounds {
  static constexpr int blocks = sizeof(R) == 4 ? 4 : RMAX > 8 ? 2 : MODE == FM_XKIN ? 3 : 4;
};

template <typename R, bool ZT, int MODE, int RMAX>
__global__ void __launch_bounds__(LINE_T, LineBounds<R, MODE, RMAX>::blocks) k_line(Phys ph, Sweep sw, FastOps op, LineGeo g,
                                                                      LineShape sh, int ax) {
  line_body<R, ZT, MODE, RMAX>(ph, sw, op, g, sh, ax, sh.tile0 + tile_of(op), gridDim.x);
}

// Batched launch: blockIdx.y selects the instance (structs staged in shared memory).
template <typename R, bool ZT, int MODE, int RMAX>
__global__ void __launch_bounds__(LINE_T, LineBounds<R, MODE, RMAX>::blocks) k_line_batch(const Phys* __restrict__ phs,
                                                                            const Sweep* __restrict__ sws,
                                                                            FastOps op, LineGeo g, LineShape sh,
                                                                            int ax) {
  __shared__ Phys ph;
  __shared__ Sweep sw;
  copy_words(&ph, phs + blockIdx.y);
  copy_words(&sw, sws + blockIdx.y);
  __syncthreads();
  if (batch_frozen(sw.live)) return;
  line_body<R, ZT, MODE, RMAX>(ph, sw, op, g, sh, ax, tile_of(op), gridDim.x);
}

// host: launch one sweep (one translation unit per precision and group of modes)
template <typename R>
cudaError_t launch_line(int ax, const Phys& ph, const Sweep& sw, const FastOps& op, const LineGeo& g,
                        const LineShape& sh, size_t smem, cudaStream_t st);
template <typename R>
cudaError_t launch_line_batch(int ax, const Phys* phs, const Sweep* sws, int count, const FastOps& op,
                              const LineGeo& g, const LineShape& sh, size_t smem, cudaStream_t st);

}  // namespace gpe
