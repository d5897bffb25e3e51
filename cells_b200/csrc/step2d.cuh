// Device code shared by the D2Q9 step kernels (one step per launch and the persistent kernel: step2d.cu;
// several steps per launch on tiles in shared memory: block2d.cu): parameters, the boundary rules, the
// collision. Compiled into cells::fast (contraction allowed) and, with -fmad=false -DCELLS_EXACT_ARITH,
// into cells::exact.
#pragma once

#include "kernels2d.h"

#ifdef CELLS_EXACT_ARITH
#define CELLS_NS exact
constexpr bool kExact2 = true;
#else
#define CELLS_NS fast
constexpr bool kExact2 = false;
#endif

namespace cells {
namespace CELLS_NS {

// Storage type S, arithmetic type R, and how populations are loaded: through the read-only path
// when a launch never writes what it reads (one step per launch), through L2 when it does (the
// persistent kernel rewrites the buffer it read two steps earlier, which a stale read-only line
// would miss).
template <class S_, class R_, bool COHERENT>
struct Store2 {
  using S = S_;
  using R = R_;
  __device__ __forceinline__ static S ld(const S* p) { return COHERENT ? __ldcg(p) : __ldg(p); }
};
using Store2F32 = Store2<float, float, false>;
using Store2F64 = Store2<double, double, false>;
using Store2F32P = Store2<float, float, true>;
using Store2F64P = Store2<double, double, true>;

template <class R>
__device__ __forceinline__ R prm(const Tunnel2& T, int k);
template <>
__device__ __forceinline__ float prm<float>(const Tunnel2& T, int k) {
  return __ldg(&T.pf[k]);
}
template <>
__device__ __forceinline__ double prm<double>(const Tunnel2& T, int k) {
  return __ldg(&T.pd[k]);
}

template <class R>
__device__ __forceinline__ R clampR(R v, R lo, R hi) {
  return v < lo ? lo : (hi < v ? hi : v);
}
// 1 / v: IEEE in the exact build and for f64; the hardware reciprocal (within 2 ulp, no branch)
// for f32 in the fast build
template <class R>
__device__ __forceinline__ R recip2(R v) {
  if constexpr (!kExact2 && sizeof(R) == 4)
    return __fdividef(R(1), v);
  else
    return R(1) / v;
}
template <class R>
struct XTab2;
template <>
struct XTab2<float> {
  using T = float4;
};
template <>
struct XTab2<double> {
  using T = double4;
};

struct Geo2 {
  int W, H;
  int left, right, bottom, top;
};

// wrapPeriodic, src/shaders/common.ts:48-57
__device__ __forceinline__ void wrap2(const Geo2& g, int& x, int& y) {
  if (x < 0 && g.left == X2_PERIODIC) x += g.W;
  if (x >= g.W && g.right == X2_PERIODIC) x -= g.W;
  if (y < 0 && g.bottom == Y2_PERIODIC) y += g.H;
  if (y >= g.H && g.top == Y2_PERIODIC) y -= g.H;
}

// inletVelocity, src/shaders/common.ts:39-45
template <class R>
__device__ __forceinline__ R inlet_velocity2(int parabolic, R uIn, int H, int y) {
  if (parabolic == 0) return uIn;
  const R h = R(H);
  const R s = R(y) + R(0.5);
  return R(4) * uIn * s * (h - s) / (h * h);
}

// The source populations of a cell as one step of a global buffer sees them: element pop of a node of the grid, given
// as its index and as (sx, sy). at() also gets the node's offset (dx, dy) from the cell, before wrapping. f32 takes
// the index, f64 forms it again, each as the one-step kernel measured faster (4000x1000, us per step, index /
// formed again: f32 68.0 / 68.8, f64 184 / 156).
template <class C>
struct GridSource2 {
  const typename C::S* __restrict__ src;
  long long N;
  int W;
  __device__ __forceinline__ typename C::R at(int pop, long long node, int sx, int sy, int, int) const {
    return (typename C::R)C::ld(&src[pop * N + (sizeof(typename C::R) == 4 ? node : (long long)sy * W + sx)]);
  }
};

// pullSlow, src/shaders/step.ts:119-175, for a flagged direction i of the cell (x, y)
template <class C, class Source>
__device__ __forceinline__ typename C::R pull_slow2(int i, const Geo2& g, const Source& src,
                                                    const uint32_t* __restrict__ flags, const float* __restrict__ sdf,
                                                    int x, int y, long long idx, typename C::R uLid,
                                                    typename C::R force[2]) {
  using R = typename C::R;
  const int j = opp2(i);
  int sx = x - cx2(i);
  int sy = y - cy2(i);
  wrap2(g, sx, sy);
  const bool inX = sx >= 0 && sx < g.W;
  const bool inY = sy >= 0 && sy < g.H;
  if (inX && inY) {
    const long long s = (long long)sy * g.W + sx;
    if ((__ldg(&flags[s]) & FLAG2_SOLID) == 0u) return src.at(i, s, sx, sy, -cx2(i), -cy2(i));
    // Bouzidi linear interpolated bounce-back with q from the SDF
    const R fj = src.at(j, idx, x, y, 0, 0);
    const R dF = (R)__ldg(&sdf[idx]);
    const R dS = (R)__ldg(&sdf[s]);
    const R den = (dF - dS) < (R)1e-6 ? (R)1e-6 : (dF - dS);
    const R q = clampR<R>(dF / den, (R)1e-3, R(1));
    R fi = fj;
    if (q < R(0.5)) {
      int nx = x + cx2(i), ny = y + cy2(i);
      wrap2(g, nx, ny);
      if (nx >= 0 && nx < g.W && ny >= 0 && ny < g.H) {
        const long long n = (long long)ny * g.W + nx;
        if ((__ldg(&flags[n]) & FLAG2_SOLID) == 0u)
          fi = R(2) * q * fj + (R(1) - R(2) * q) * src.at(j, n, nx, ny, cx2(i), cy2(i));
      }
    } else {
      fi = fj / (R(2) * q) + (R(2) * q - R(1)) / (R(2) * q) * src.at(i, idx, x, y, 0, 0);
    }
    const R t = fj + fi;
    force[0] += R(cx2(j)) * t;
    force[1] += R(cy2(j)) * t;
    return fi;
  }
  if (!inY) {
    const int mode = sy < 0 ? g.bottom : g.top;
    if (mode == Y2_SLIP) {
      const int rx = sx < 0 ? 0 : (sx > g.W - 1 ? g.W - 1 : sx);
      return src.at(mirror_y2(i), (long long)y * g.W + rx, rx, y, inX ? -cx2(i) : 0, 0);
    }
    if (mode == Y2_MOVING) return src.at(j, idx, x, y, 0, 0) + R(6) * w2<R>(i) * R(cx2(i)) * uLid;
    return src.at(j, idx, x, y, 0, 0);
  }
  // walls, and placeholders that the open-boundary fix-up overwrites
  return src.at(j, idx, x, y, 0, 0);
}

// Zou-He inlet and outlet (populations stored shifted by w_i)
template <class C>
__device__ __forceinline__ void zou_he2(int parabolic, int H, bool inlet, typename C::R uIn, int y,
                                        typename C::R (&f)[Q2]) {
  using R = typename C::R;
  if (inlet) {
    const R u = inlet_velocity2<R>(parabolic, uIn, H, y);
    const R r = (R(1) + f[0] + f[2] + f[4] + R(2) * (f[3] + f[6] + f[7])) / (R(1) - u);
    f[1] = f[3] + (R)(2.0 / 3.0) * r * u;
    f[5] = f[7] - R(0.5) * (f[2] - f[4]) + (R)(1.0 / 6.0) * r * u;
    f[8] = f[6] + R(0.5) * (f[2] - f[4]) + (R)(1.0 / 6.0) * r * u;
  } else {
    const R u = f[0] + f[2] + f[4] + R(2) * (f[1] + f[5] + f[8]);
    f[3] = f[1] - (R)(2.0 / 3.0) * u;
    f[7] = f[5] + R(0.5) * (f[2] - f[4]) - (R)(1.0 / 6.0) * u;
    f[6] = f[8] - R(0.5) * (f[2] - f[4]) - (R)(1.0 / 6.0) * u;
  }
}

// The pulled populations of a flagged fluid cell (x, y) whose plain pulls are in f. pullSlow's first
// rule: a direction without its flag bit is the plain pull (the same element), so the general rules
// run for the flagged directions only. An inlet (outlet) cell whose only flagged directions are the
// three entering from outside the grid skips them altogether: Zou-He replaces those three pulls. Returns
// whether the cell has a force slot (its force is then in force[0..1]).
template <class C, class Source>
__device__ __forceinline__ bool boundary2(const Tunnel2& T, const Geo2& g, const Source& src,
                                          const uint32_t* __restrict__ flags, typename C::R uIn, int x, int y,
                                          long long idx, uint32_t fl, typename C::R (&f)[Q2],
                                          typename C::R force[2]) {
  using R = typename C::R;
  bool slot = false;
  constexpr uint32_t kInletPlain = FLAG2_INLET | (1u << 1) | (1u << 5) | (1u << 8);
  constexpr uint32_t kOutletPlain = FLAG2_OUTLET | (1u << 3) | (1u << 6) | (1u << 7);
  if (fl != kInletPlain && fl != kOutletPlain) {
    const R uLid = prm<R>(T, P2_ULID);
#pragma unroll
    for (int i = 1; i < Q2; i++)
      if (fl & (1u << i)) f[i] = pull_slow2<C>(i, g, src, flags, T.sdf, x, y, idx, uLid, force);
    slot = (fl >> BIDX2_SHIFT) != 0u;
  }
  if (fl & (FLAG2_INLET | FLAG2_OUTLET)) zou_he2<C>(T.parabolic, g.H, (fl & FLAG2_INLET) != 0u, uIn, y, f);
  return slot;
}

// The same update as collide2 in the block kernel's fast build, with about half the operations (that
// kernel is bound by issue, the one-step kernel by latency): pair sums s = f_a + f_b and differences
// d = f_a - f_b feed the moments and the update o_a, o_b = (S +- D) / 2 with
//   S = s - omega+ (s - 2 w (rho cu^2 / 2 + K0)),  D = d - omega- (d - 2 w rho cu),
//   K0 = drho - rho u.u 3/2, cu = 3 c_a . u.
// The relaxed differences are formed as written: in (1 - omega) s + omega w (..) the rounding of the two
// factors is the same in every cell of a column and step, a drift of mass and momentum that put the drag of
// a 400x100 cylinder after 400 steps off by 1.7e-6 of its value instead of 0.8e-6.
// xt: the column's x table entry. Both cells of a thread in the packed f32x2 instructions would halve the
// issue slots again, but the two sets of 18 populations do not fit beside the loop's state: 64 tunnels of
// the NACA section take 102 us per step like this and 163 to 190 us packed (spills at 64 and 128 registers).
template <class R>
__device__ __forceinline__ void collide2_lean(const Tunnel2& T, const typename XTab2<R>::T& xt, int forcing, R smagC2,
                                              R lambda, int H, int parabolic, R uIn, int y, const R (&f)[Q2], R (&o)[Q2]) {
  constexpr int A[4] = {1, 2, 5, 6}, B[4] = {3, 4, 7, 8};
  R s[4], d[4];
#pragma unroll
  for (int p = 0; p < 4; p++) {
    s[p] = f[A[p]] + f[B[p]];
    d[p] = f[A[p]] - f[B[p]];
  }
  const R drho = f[0] + ((s[0] + s[1]) + (s[2] + s[3]));
  const R rho = R(1) + drho;
  const R invRho = recip2<R>(rho);
  R ux = (d[0] + (d[2] - d[3])) * invRho;
  R uy = (d[1] + (d[2] + d[3])) * invRho;
  R bfx = R(0), bfy = R(0);
  if (forcing != 0) {
    bfx = prm<R>(T, P2_FX);
    bfy = prm<R>(T, P2_FY);
    ux += R(0.5) * bfx * invRho;
    uy += R(0.5) * bfy * invRho;
  }
  const R uu = ux * ux + uy * uy;
  const R K0 = drho - R(1.5) * rho * uu;
  const R hr = R(0.5) * rho;
  const R x3 = R(3) * ux, y3 = R(3) * uy;
  const R cu[4] = {x3, y3, x3 + y3, y3 - x3};
  R e[4];  // rho cu^2 / 2 + K0
#pragma unroll
  for (int p = 0; p < 4; p++) e[p] = hr * cu[p] * cu[p] + K0;
  R ns[4];  // non-equilibrium part of the pair sums
#pragma unroll
  for (int p = 0; p < 4; p++) ns[p] = s[p] - R(2) * w2<R>(A[p]) * e[p];
  R omP = xt.x, omM = xt.y;
  if (smagC2 > R(0)) {
    const R diag = ns[2] + ns[3], pxy = ns[2] - ns[3];
    const R pxx = ns[0] + diag, pyy = ns[1] + diag;
    const R pi = sqrt(pxx * pxx + R(2) * pxy * pxy + pyy * pyy);
    const R t0 = xt.w;  // 1 / omegaBase
    const R tEff = R(0.5) * (t0 + sqrt(t0 * t0 + (R)25.45584412271571 * smagC2 * pi * invRho));
    // omega- = 1 / (1/2 + Lambda / (tEff - 1/2)) with one quotient
    const R h = tEff - R(0.5);
    omP = recip2<R>(tEff);
    if constexpr (sizeof(R) == 4)
      omM = __fdividef(h, R(0.5) * h + lambda);
    else
      omM = h / (R(0.5) * h + lambda);
  }
  const R r2 = R(2) * rho;
  R S[4], D[4];
  R o0 = f[0] - omP * (f[0] - w2<R>(0) * K0);
#pragma unroll
  for (int p = 0; p < 4; p++) {
    S[p] = s[p] - omP * ns[p];
    D[p] = d[p] - omM * (d[p] - w2<R>(A[p]) * r2 * cu[p]);
  }
  // absorbing-layer and Guo body-force sources (src/shaders/step.ts:65-91)
  const R sig = xt.z;
  if (sig > R(0)) {
    const R ut = inlet_velocity2<R>(parabolic, uIn, H, y);
    const R dq = R(1.5) * rho * (ut * ut - uu);
    o0 -= sig * w2<R>(0) * dq;
#pragma unroll
    for (int p = 0; p < 4; p++) {
      const R cut = R(3) * R(cx2(A[p])) * ut, sw = R(2) * sig * w2<R>(A[p]);
      S[p] += sw * (hr * (cut * cut - cu[p] * cu[p]) - dq);
      D[p] += sw * rho * (cut - cu[p]);
    }
  }
  if (forcing != 0) {
    const R uF = ux * bfx + uy * bfy;
    const R gP = R(1) - R(0.5) * omP, gM = R(1) - R(0.5) * omM;
    o0 -= gP * w2<R>(0) * R(3) * uF;
#pragma unroll
    for (int p = 0; p < 4; p++) {
      const R cF = R(cx2(A[p])) * bfx + R(cy2(A[p])) * bfy;
      S[p] += gP * (R(2) * w2<R>(A[p])) * (R(3) * cF * cu[p] - R(3) * uF);
      D[p] += gM * (R(6) * w2<R>(A[p])) * cF;
    }
  }
  o[0] = o0;
#pragma unroll
  for (int p = 0; p < 4; p++) {
    const R h = R(0.5) * S[p];
    o[A[p]] = h + R(0.5) * D[p];
    o[B[p]] = h - R(0.5) * D[p];
  }
}

// Moments, Smagorinsky, the absorbing-layer and Guo sources and the TRT update of one cell of row y
// (src/shaders/step.ts:177-227), each population to store(i, value) as it is known; xt: the x table's entry of its
// column. The exact build evaluates every other expression in the reference's order.
template <class C, class Store>
__device__ __forceinline__ void collide2(const Tunnel2& T, const typename XTab2<typename C::R>::T& xt, int forcing,
                                         typename C::R smagC2, int H, typename C::R uIn, int y,
                                         const typename C::R (&f)[Q2], const Store& store) {
  using R = typename C::R;
  // moments (src/shaders/step.ts:22-32)
  const R drho = f[0] + f[1] + f[2] + f[3] + f[4] + f[5] + f[6] + f[7] + f[8];
  const R rho = R(1) + drho;
  const R invRho = recip2<R>(rho);
  R ux = (f[1] - f[3] + f[5] - f[6] - f[7] + f[8]) * invRho;
  R uy = (f[2] - f[4] + f[5] + f[6] - f[7] - f[8]) * invRho;
  R bfx = R(0), bfy = R(0);
  if (forcing != 0) {
    bfx = prm<R>(T, P2_FX);
    bfy = prm<R>(T, P2_FY);
    ux += R(0.5) * bfx * invRho;
    uy += R(0.5) * bfy * invRho;
  }
  const R usq = R(1.5) * (ux * ux + uy * uy);
  R cu[Q2];
  cu[1] = R(3) * (ux);
  cu[2] = R(3) * (uy);
  cu[5] = R(3) * (ux + uy);
  cu[6] = R(3) * (-ux + uy);
  R eqS[Q2], eqA[Q2];
#pragma unroll
  for (int a : {1, 2, 5, 6}) {
    eqS[a] = w2<R>(a) * (drho + rho * (R(0.5) * cu[a] * cu[a] - usq));
    eqA[a] = w2<R>(a) * rho * cu[a];
  }
  // sponge and absorbing layers (src/shaders/step.ts:215-223), from the x table
  const R omegaBase = xt.x;
  const R sigma = xt.z;
  // Smagorinsky (src/shaders/step.ts:48-63)
  R omP = omegaBase, omM = xt.y;
  if (smagC2 > R(0)) {
    R n[Q2];
#pragma unroll
    for (int a : {1, 2, 5, 6}) {
      const int b = opp2(a);
      n[a] = f[a] - (eqS[a] + eqA[a]);
      n[b] = f[b] - (eqS[a] - eqA[a]);
    }
    const R pxx = n[1] + n[3] + n[5] + n[6] + n[7] + n[8];
    const R pyy = n[2] + n[4] + n[5] + n[6] + n[7] + n[8];
    const R pxy = n[5] - n[6] + n[7] - n[8];
    const R pi = sqrt(pxx * pxx + pyy * pyy + R(2) * pxy * pxy);
    const R t0 = xt.w;  // 1 / omegaBase
    const R tEff = R(0.5) * (t0 + sqrt(t0 * t0 + (R)25.45584412271571 * smagC2 * pi * invRho));
    omP = recip2<R>(tEff);
    // the exact build divides 1 by omega+ again, as the reference does; the fast build uses tEff
    const R tP = kExact2 ? R(1) / omP : tEff;
    omM = recip2<R>(R(0.5) + prm<R>(T, P2_LAMBDA) / (tP - R(0.5)));
  }
  // absorbing-layer and Guo body-force sources (src/shaders/step.ts:65-91)
  R s0 = R(0);
  R sS[Q2], sA[Q2];
#pragma unroll
  for (int a : {1, 2, 5, 6}) {
    sS[a] = R(0);
    sA[a] = R(0);
  }
  if (sigma > R(0)) {
    const R ut = inlet_velocity2<R>(T.parabolic, uIn, H, y);
    const R dq = R(1.5) * rho * (ut * ut - ux * ux - uy * uy);
    s0 += sigma * w2<R>(0) * -dq;
#pragma unroll
    for (int a : {1, 2, 5, 6}) {
      const R cut = R(3) * R(cx2(a)) * ut;
      sS[a] += sigma * w2<R>(a) * (R(0.5) * rho * (cut * cut - cu[a] * cu[a]) - dq);
      sA[a] += sigma * w2<R>(a) * rho * (cut - cu[a]);
    }
  }
  if (forcing != 0) {
    const R uF = ux * bfx + uy * bfy;
    s0 += (R(1) - R(0.5) * omP) * w2<R>(0) * (R(-3) * uF);
#pragma unroll
    for (int a : {1, 2, 5, 6}) {
      const R cF = (R(cx2(a)) * bfx + R(cy2(a)) * bfy);
      sS[a] += (R(1) - R(0.5) * omP) * w2<R>(a) * (R(-3) * uF + R(9) * (cu[a] / R(3)) * cF);
      sA[a] += (R(1) - R(0.5) * omM) * w2<R>(a) * R(3) * cF;
    }
  }
  // TRT collide (src/shaders/step.ts:93-103)
  store(0, f[0] - omP * (f[0] - w2<R>(0) * (drho - rho * usq)) + s0);
#pragma unroll
  for (int a : {1, 2, 5, 6}) {
    const int b = opp2(a);
    const R sym = omP * (R(0.5) * (f[a] + f[b]) - eqS[a]);
    const R asym = omM * (R(0.5) * (f[a] - f[b]) - eqA[a]);
    store(a, f[a] - sym - asym + sS[a] + sA[a]);
    store(b, f[b] - sym + asym + sS[a] - sA[a]);
  }
}

__device__ __forceinline__ double ramp_speed2(int kind, double target, double rampSteps, int every, unsigned step) {
  const double sq = (double)((step / (unsigned)every) * (unsigned)every);
  const double t = fmin(1.0, sq / rampSteps);
  return kind == 1 ? target * t : target * (t * t * (3.0 - 2.0 * t));
}

}  // namespace CELLS_NS
}  // namespace cells
