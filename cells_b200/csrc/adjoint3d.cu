// Discrete adjoint of the D3Q19 step: the adjoint step kernels, the recorded forward run with
// checkpoints, the backward sweep with recomputation, and their C ABI (include/cells.h). No
// counterpart in the reference.
//
// Adjoint step n (from lambda^{n+1} to lambda^n over the recomputed state f^n), per cell x:
//   g = P(f^n)(x): the 19 pulled values (plain pulls, or the cell's link records at boundaries);
//   lambda_g = (dC/dg)^T lambda^{n+1}(x): the transposed Jacobian of the TRT collision (or of the
//     outlet's feq(1, u), or zero at the inlet, whose output does not depend on g);
//   the streaming transpose: a plain pull of direction i from x - c_i is the only regular reader of
//     that element, so lambda^n_i(x - c_i) = lambda_g,i is a plain store; a link's adjoint goes to
//     lamG and a second kernel adds it, with the objective's direct force terms, to the link's
//     source elements (a fixed-order sum per element: deterministic).
// Shape: dJ/dq per Bouzidi link accumulates (lambda_g + w cF) dg/dq; dq/dsdf then gives dJ/dsdf.
// Inflow: dJ/du_n from the inlet's feq(1, u_n) and the absorbing layer's target u_n, summed per
// step in f64 with a fixed order.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "adjoint3d.h"
#include "solver3d_state.h"

using namespace cells;

namespace {

__host__ __device__ __forceinline__ long long off3(int i, int W, int H) {
  return (long long)cx3(i) + (long long)W * ((long long)cy3(i) + (long long)H * cz3(i));
}

// Arithmetic on one cell's values (float, double) or on those of two x-neighbours (float2: the packed
// f32x2 instructions of sm_100, each component rounding as the scalar instruction would).
template <class V>
struct Lane {
  using R = V;
  __device__ __forceinline__ static V bc(R v) { return v; }
  __device__ __forceinline__ static V add(V a, V b) { return a + b; }
  __device__ __forceinline__ static V sub(V a, V b) { return a - b; }
  __device__ __forceinline__ static V mul(V a, V b) { return a * b; }
  __device__ __forceinline__ static V fma(V a, V b, V c) { return ::fma(a, b, c); }
  // f32: the hardware reciprocal (branch-free, within 2 ulp)
  __device__ __forceinline__ static V recip(V a) {
    if constexpr (sizeof(V) == 4)
      return __fdividef(V(1), a);
    else
      return V(1) / a;
  }
  __device__ __forceinline__ static bool positive(V a) { return a > V(0); }
};
template <>
struct Lane<float2> {
  using R = float;
  __device__ __forceinline__ static float2 bc(float v) { return make_float2(v, v); }
  __device__ __forceinline__ static float2 add(float2 a, float2 b) { return __fadd2_rn(a, b); }
  __device__ __forceinline__ static float2 sub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }
  __device__ __forceinline__ static float2 mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
  __device__ __forceinline__ static float2 fma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
  __device__ __forceinline__ static float2 recip(float2 a) {
    return make_float2(__fdividef(1.0f, a.x), __fdividef(1.0f, a.y));
  }
  __device__ __forceinline__ static bool positive(float2 a) { return a.x > 0.0f || a.y > 0.0f; }
};

// c_p . v for direction p
template <class V>
__device__ __forceinline__ V dot_c3(int p, const V (&v)[3]) {
  using L = Lane<V>;
  V r = L::bc(0);
  bool any = false;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const int c = k == 0 ? cx3(p) : (k == 1 ? cy3(p) : cz3(p));
    if (c == 0) continue;
    if (!any)
      r = v[k];  // the first component of a pair's lower member is +1
    else
      r = c > 0 ? L::add(r, v[k]) : L::sub(r, v[k]);
    any = true;
  }
  return r;
}

// (dC/dg)^T lp for the TRT collision with sponge rate omP/omM and absorbing strength sigma toward
// the inflow speed ut (src/shaders/step3d.ts:38-102, Smagorinsky off). Also returns dJ/dut.
// ABS = false: a cell known to lie outside the absorbing layer, compiled without its terms.
//
// With S, D = lp_a +- lp_b of each pair (a, b), s = omega+ w S, d = omega- w D and cu = 3 c_a . u:
//   d/drho:  (1 - 3u^2/2) sum s + sum cu (s cu / 2 + d)      (s of the rest direction included)
//   d/du:    3 rho sum c_a (s cu + d) - 3 u rho sum s
//   lg_a, lg_b = (1 - omega+)/2 S + rhoB +- ((1 - omega-)/2 D + c_a . jB)
// so a pair costs about 16 operations; written per direction with the pair's sums formed twice, the
// kernel issued 850 thread instructions per cell and was bound by them.
template <class V, bool ABS = true>
__device__ __forceinline__ void collide_adjoint3(const V g[Q3], const V lp[Q3], V omP, V omM, V sigma,
                                                 typename Lane<V>::R utS, V lg[Q3], V& dut) {
  using L = Lane<V>;
  using R = typename L::R;
  const R w0 = w3<R>(0), w1 = w3<R>(1), w7 = w3<R>(7);
  V u[3], rho, inv;
  {
    V sum = g[0];
    V j[3] = {L::bc(0), L::bc(0), L::bc(0)};
#pragma unroll
    for (int p = 1; p < Q3; p += 2) {
      sum = L::add(sum, L::add(g[p], g[p + 1]));
      const V d = L::sub(g[p], g[p + 1]);
      if (cx3(p) != 0) j[0] = cx3(p) > 0 ? L::add(j[0], d) : L::sub(j[0], d);
      if (cy3(p) != 0) j[1] = cy3(p) > 0 ? L::add(j[1], d) : L::sub(j[1], d);
      if (cz3(p) != 0) j[2] = cz3(p) > 0 ? L::add(j[2], d) : L::sub(j[2], d);
    }
    rho = L::add(L::bc(1), sum);
    inv = L::recip(rho);
#pragma unroll
    for (int k = 0; k < 3; k++) u[k] = L::mul(j[k], inv);
  }
  const V uu = L::fma(u[2], u[2], L::fma(u[1], u[1], L::mul(u[0], u[0])));
  const V u3[3] = {L::mul(L::bc(3), u[0]), L::mul(L::bc(3), u[1]), L::mul(L::bc(3), u[2])};
  const V sP[2] = {L::mul(omP, L::bc(w1)), L::mul(omP, L::bc(w7))};
  const V sM[2] = {L::mul(omM, L::bc(w1)), L::mul(omM, L::bc(w7))};
  const bool absorb = ABS && L::positive(sigma);
  const V ut = L::bc(utS);
  V S[Q3], D[Q3];  // entries p = 1, 3, .., 17
  V sumS = L::mul(L::mul(omP, L::bc(w0)), lp[0]);
  V rB = L::bc(0);
  V T[3] = {L::bc(0), L::bc(0), L::bc(0)};
  V dqB = L::bc(0), utA = L::bc(0);
  if (absorb) dqB = L::mul(L::mul(L::bc(-w0), sigma), lp[0]);
#pragma unroll
  for (int p = 1; p < Q3; p += 2) {
    const int k = p <= 5 ? 0 : 1;
    S[p] = L::add(lp[p], lp[p + 1]);
    D[p] = L::sub(lp[p], lp[p + 1]);
    const V cu = dot_c3<V>(p, u3);
    const V s = L::mul(sP[k], S[p]), d = L::mul(sM[k], D[p]);
    sumS = L::add(sumS, s);
    rB = L::fma(cu, L::fma(L::mul(L::bc(R(0.5)), s), cu, d), rB);
    V t = L::fma(s, cu, d);
    if (absorb) {
      const V sw = L::mul(sigma, L::bc(k == 0 ? w1 : w7));
      const V as = L::mul(sw, S[p]), ad = L::mul(sw, D[p]);
      const V cut = L::mul(L::bc(R(3) * R(cx3(p))), ut);
      const V dc = L::sub(cut, cu);
      // as (cut^2 - cu^2) / 2 + ad (cut - cu)
      rB = L::fma(dc, L::fma(L::mul(L::bc(R(0.5)), as), L::add(cut, cu), ad), rB);
      t = L::sub(t, L::fma(as, cu, ad));
      dqB = L::sub(dqB, as);
      if (cx3(p) != 0) utA = L::fma(L::bc(R(cx3(p))), L::fma(as, cut, ad), utA);
    }
    if (cx3(p) != 0) T[0] = cx3(p) > 0 ? L::add(T[0], t) : L::sub(T[0], t);
    if (cy3(p) != 0) T[1] = cy3(p) > 0 ? L::add(T[1], t) : L::sub(T[1], t);
    if (cz3(p) != 0) T[2] = cz3(p) > 0 ? L::add(T[2], t) : L::sub(T[2], t);
  }
  const V rho3 = L::mul(L::bc(3), rho);
  V rhoB = L::fma(L::fma(L::bc(R(-1.5)), uu, L::bc(1)), sumS, rB);
  V uB[3];
  // 3 rho (T - u sum s), and the absorbing layer's dq = 1.5 rho (ut^2 - |u|^2)
  const V usq = absorb ? L::add(sumS, dqB) : sumS;
#pragma unroll
  for (int k = 0; k < 3; k++) uB[k] = L::mul(rho3, L::sub(T[k], L::mul(u[k], usq)));
  dut = L::bc(0);
  if (absorb) {
    rhoB = L::fma(L::mul(L::bc(R(1.5)), dqB), L::sub(L::mul(ut, ut), uu), rhoB);
    dut = L::mul(rho3, L::fma(dqB, ut, utA));
  }
  const V jB[3] = {L::mul(uB[0], inv), L::mul(uB[1], inv), L::mul(uB[2], inv)};
  rhoB = L::sub(rhoB, L::fma(u[2], jB[2], L::fma(u[1], jB[1], L::mul(u[0], jB[0]))));
  lg[0] = L::fma(L::sub(L::bc(1), omP), lp[0], rhoB);
  const V hP = L::fma(L::bc(R(-0.5)), omP, L::bc(R(0.5))), hM = L::fma(L::bc(R(-0.5)), omM, L::bc(R(0.5)));
#pragma unroll
  for (int p = 1; p < Q3; p += 2) {
    const V a = L::fma(hP, S[p], rhoB), b = L::fma(hM, D[p], dot_c3<V>(p, jB));
    lg[p] = L::add(a, b);
    lg[p + 1] = L::sub(a, b);
  }
}

// (d feq(1, u(g)) / dg)^T lp: the outlet stores feq(1, u) with u the velocity of the pulled values.
template <class R>
__device__ __forceinline__ void outlet_adjoint3(const R g[Q3], const R lp[Q3], R lg[Q3]) {
  R drho = R(0);
#pragma unroll
  for (int i = 0; i < Q3; i++) drho += g[i];
  const R rho = R(1) + drho;
  const R inv = R(1) / rho;
  R jx = R(0), jy = R(0), jz = R(0);
#pragma unroll
  for (int i = 1; i < Q3; i++) {
    jx += R(cx3(i)) * g[i];
    jy += R(cy3(i)) * g[i];
    jz += R(cz3(i)) * g[i];
  }
  const R ux = jx * inv, uy = jy * inv, uz = jz * inv;
  R uxB = R(0), uyB = R(0), uzB = R(0);
#pragma unroll
  for (int i = 0; i < Q3; i++) {
    const R cu = R(3) * (R(cx3(i)) * ux + R(cy3(i)) * uy + R(cz3(i)) * uz);
    const R k = lp[i] * w3<R>(i);
    uxB += k * (R(3) * R(cx3(i)) * (R(1) + cu) - R(3) * ux);
    uyB += k * (R(3) * R(cy3(i)) * (R(1) + cu) - R(3) * uy);
    uzB += k * (R(3) * R(cz3(i)) * (R(1) + cu) - R(3) * uz);
  }
  const R jxB = uxB * inv, jyB = uyB * inv, jzB = uzB * inv;
  const R rhoB = -(ux * uxB + uy * uyB + uz * uzB) * inv;
#pragma unroll
  for (int i = 0; i < Q3; i++) lg[i] = rhoB + R(cx3(i)) * jxB + R(cy3(i)) * jyB + R(cz3(i)) * jzB;
}

// The block's f64 sum of dJ/du_n into part[slot] (adj_du3_kernel sums the slots in order).
__device__ __forceinline__ void block_du_partial(double du, double* part, int slot, double* red, int tid) {
  for (int o = 16; o > 0; o >>= 1) du += __shfl_down_sync(0xffffffffu, du, o);
  if ((tid & 31) == 0) red[tid >> 5] = du;
  __syncthreads();
  if (tid == 0) {
    double s = 0.0;
    for (int k = 0; k < kAdjThreads / 32; k++) s += red[k];
    part[slot] = s;
  }
}

// One adjoint step, one launch: blocks of 128 threads in a grid of z slices. The first roleZ slices
// hold the listed flagged fluid cells (adj_slow_role) and, with x-pairs, the face rows
// (adj_face_pairs_role), the others the rows y = 1 .. H-2 of the planes z = 1 .. D-2 in tiles of 4 rows of
// 32 cells or pairs (every cell of the remaining rows is flagged). The roles write disjoint elements. The launch and the boundary-element kernel after it are programmatic
// dependents of their predecessors: their blocks take the slots a finishing grid frees.
//
// What bounds it: memory. An adjoint step moves 228 bytes per f32 cell and the recompute beside it 152;
// the adjoint states and the recomputed state together are larger than L2 at 128x64x64, where all of it
// at the copy bandwidth takes 31 us. Per adjoint step there, recompute included (6,000 steps, K = 100):
// 53 us with all 40k flagged cells in the list on a second stream, the per-direction collision and
// the sum of dJ/du_n in the boundary-element kernel; 49 us as one launch with loads batched; 44 us with
// the face rows as x-pairs, the packed collision, direct stores for links that are their source's only
// reader, and f^n asked for before the dependency wait.

// Programmatic dependent launch: waits for the boundary-element kernel of the step before to complete.
// f^n, the tables and the flags do not depend on it, so the roles ask for them first: a segment's first adjoint
// step is launched without the attribute (launch_adjoint_step3's `first`), after all work before it, the recompute
// that wrote the segment's states included. lambda^{n+1} comes through L2 (__ldcg): the launch before may still write it
// while these blocks are resident, which the read-only path does not allow for.
__device__ __forceinline__ void adj_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class R>
__device__ __forceinline__ double adj_cells_role(const AdjLaunch3& a, int tz) {
  // a tile of x-rows per block (no division per cell); 32-bit element indices (19 N < 2^31)
  const int W = a.W, H = a.H;
  const int N = (int)a.N;
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = 1 + blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= W || y >= H - 1) return 0.0;
  const R* __restrict__ f = (const R*)a.f;
  const R* __restrict__ lamNext = (const R*)a.lamNext;
  R* __restrict__ lamOut = (R*)a.lamOut;
  const int idx = x + W * (y + H * (1 + tz));
  // the plain pulls go out with the flag load rather than after it: the sources of an interior row
  // lie inside the 19 N arrays, and flagged cells discard the values
  R g[Q3], lp[Q3];
#pragma unroll
  for (int i = 0; i < Q3; i++) g[i] = __ldg(&f[i * N + idx - (int)off3(i, W, H)]);
  const uint32_t fl = __ldg(&a.flags[idx]);
  adj_wait();
#pragma unroll
  for (int i = 0; i < Q3; i++) lp[i] = __ldcg(&lamNext[i * N + idx]);
  if (fl != 0u) return 0.0;
  // interior cell: plain pulls, the collision's transposed Jacobian, plain pushes
  R lg[Q3];
  const R* xt = (const R*)a.xTab + 4 * x;
  R dut;
  // block-uniform: tiles that end before the absorbing layer take the code without it
  if ((int)((blockIdx.x + 1) * blockDim.x) > a.absorbX0)
    collide_adjoint3<R, true>(g, lp, xt[0], xt[1], xt[2], (R)a.u, lg, dut);
  else
    collide_adjoint3<R, false>(g, lp, xt[0], xt[1], xt[2], (R)a.u, lg, dut);
#pragma unroll
  for (int i = 0; i < Q3; i++) lamOut[i * N + idx - (int)off3(i, W, H)] = lg[i];
  return (double)dut;
}

// f32 and an even width: the x-pair (x0, x0 + 1), x0 even, per thread. lambda^{n+1} and the
// directions with c_x = 0 move as 8-byte words, and both cells go through one packed instruction stream.
__device__ __forceinline__ double adj_pairs_role(const AdjLaunch3& a, int tz) {
  const int W = a.W, H = a.H;
  const int N = (int)a.N;
  const int x0 = blockIdx.x * (2 * blockDim.x) + 2 * threadIdx.x;
  const int y = 1 + blockIdx.y * blockDim.y + threadIdx.y;
  if (x0 >= W || y >= H - 1) return 0.0;
  const float* __restrict__ f = (const float*)a.f;
  const float* __restrict__ lamNext = (const float*)a.lamNext;
  float* __restrict__ lamOut = (float*)a.lamOut;
  const int idx = x0 + W * (y + H * (1 + tz));
  float2 g[Q3], lp[Q3];
#pragma unroll
  for (int i = 0; i < Q3; i++) {
    const float* p = f + (i * N + idx - (int)off3(i, W, H));
    g[i] = cx3(i) == 0 ? __ldg(reinterpret_cast<const float2*>(p)) : make_float2(__ldg(p), __ldg(p + 1));
  }
  const uint2 fl = __ldg(reinterpret_cast<const uint2*>(a.flags + idx));
  adj_wait();
#pragma unroll
  for (int i = 0; i < Q3; i++) lp[i] = __ldcg(reinterpret_cast<const float2*>(lamNext + (i * N + idx)));
  if (fl.x != 0u && fl.y != 0u) return 0.0;
  const float4* xt = (const float4*)a.xTab + x0;
  const float4 t0 = __ldg(xt), t1 = __ldg(xt + 1);
  const float2 omP = make_float2(t0.x, t1.x), omM = make_float2(t0.y, t1.y), sigma = make_float2(t0.z, t1.z);
  float2 lg[Q3], dut;
  if ((int)((blockIdx.x + 1) * 2 * blockDim.x) > a.absorbX0)
    collide_adjoint3<float2, true>(g, lp, omP, omM, sigma, (float)a.u, lg, dut);
  else
    collide_adjoint3<float2, false>(g, lp, omP, omM, sigma, (float)a.u, lg, dut);
  if (fl.x == 0u && fl.y == 0u) {
#pragma unroll
    for (int i = 0; i < Q3; i++) {
      float* p = lamOut + (i * N + idx - (int)off3(i, W, H));
      if (cx3(i) == 0) {
        *reinterpret_cast<float2*>(p) = lg[i];
      } else {
        p[0] = lg[i].x;
        p[1] = lg[i].y;
      }
    }
    return (double)dut.x + (double)dut.y;
  }
  const int k = fl.x == 0u ? 0 : 1;  // the other cell is flagged
#pragma unroll
  for (int i = 0; i < Q3; i++) lamOut[i * N + idx + k - (int)off3(i, W, H)] = k ? lg[i].y : lg[i].x;
  return (double)(k ? dut.y : dut.x);
}

// The x-pairs of a face row with one outside side (rows y = 1 .. H-2 of the z = 0 / z = D-1 planes,
// sides 0 / 1; the y = 0 / y = H-1 rows of the planes between, sides 2 / 3) away from bodies: a
// direction that enters from outside pulls the mirrored population of the same plane or row
// (foff[side], as the forward step's face tiles). No other cell reads that element, so its adjoint is a
// plain store as well. The row's inlet and outlet cells, and all cells of rows that hold a body cell, are
// in the flagged-cell list.
__device__ __forceinline__ double adj_face_pairs_role(const AdjLaunch3& a, int fb) {
  const int W = a.W, H = a.H, D = a.D;
  const int tilesX = gridDim.x, perPlane = gridDim.x * gridDim.y;
  int side, tx, y, z;
  if (fb < 2 * perPlane) {
    side = fb >= perPlane ? 1 : 0;
    const int rem = fb - side * perPlane, ty = rem / tilesX;
    tx = rem - ty * tilesX;
    y = 1 + ty * blockDim.y + threadIdx.y;
    z = side ? D - 1 : 0;
    if (y >= H - 1) return 0.0;
  } else {
    fb -= 2 * perPlane;
    const int perSide = (D - 2 + (int)blockDim.y - 1) / (int)blockDim.y * tilesX;
    side = fb >= perSide ? 3 : 2;
    const int rem = fb - (side - 2) * perSide, gz = rem / tilesX;
    tx = rem - gz * tilesX;
    y = side == 3 ? H - 1 : 0;
    z = 1 + gz * blockDim.y + threadIdx.y;
    if (z >= D - 1) return 0.0;
  }
  const int x0 = tx * (2 * blockDim.x) + 2 * threadIdx.x;
  const int row = y + H * z;
  if (x0 >= W || a.rowBody[row]) return 0.0;
  const float* __restrict__ f = (const float*)a.f;
  const float* __restrict__ lamNext = (const float*)a.lamNext;
  float* __restrict__ lamOut = (float*)a.lamOut;
  const int N = (int)a.N, idx = x0 + W * row;
  float2 g[Q3], lp[Q3];
#pragma unroll
  for (int i = 0; i < Q3; i++) {
    const float* p = f + (idx + a.foff[side][i]);
    g[i] = cx3(i) == 0 ? __ldg(reinterpret_cast<const float2*>(p)) : make_float2(__ldg(p), __ldg(p + 1));
  }
  adj_wait();
#pragma unroll
  for (int i = 0; i < Q3; i++) lp[i] = __ldcg(reinterpret_cast<const float2*>(lamNext + (i * N + idx)));
  const float4* xt = (const float4*)a.xTab + x0;
  const float4 t0 = __ldg(xt), t1 = __ldg(xt + 1);
  float2 lg[Q3], dut;
  collide_adjoint3<float2, true>(g, lp, make_float2(t0.x, t1.x), make_float2(t0.y, t1.y), make_float2(t0.z, t1.z),
                                 (float)a.u, lg, dut);
  const bool on0 = x0 > 0, on1 = x0 + 1 < W - 1;
#pragma unroll
  for (int i = 0; i < Q3; i++) {
    float* p = lamOut + (idx + a.foff[side][i]);
    if (on0) p[0] = lg[i].x;
    if (on1) p[1] = lg[i].y;
  }
  return (on0 ? (double)dut.x : 0.0) + (on1 ? (double)dut.y : 0.0);
}

// L2 prefetch for the tile one plane later: one 128-byte line per thread and turn, of the 19 pulls
// and of lambda^{n+1}, as the forward step does it (a hint: every address is a source of an interior
// row of that plane).
template <class R, int TILEX>
__device__ __forceinline__ void adj_prefetch(const AdjLaunch3& a, int tz, int tid) {
  constexpr int kPer = 128 / (int)sizeof(R), kLines = TILEX / kPer, kRows = kAdjThreads / kAdjTileX;
  constexpr int kSlots = kLines * kRows;  // lines of a tile per array
  const int l = tid % kLines, r = tid / kLines % kRows;
  const int y = 1 + blockIdx.y * kRows + r;
  const int x = (int)blockIdx.x * TILEX + l * kPer + kPer / 2;
  if (y >= a.H - 1 || x >= a.W - 1) return;
  const long long cell = x + (long long)a.W * (y + (long long)a.H * (1 + tz));
#pragma unroll
  for (int q0 = 0; q0 < Q3; q0 += kAdjThreads / kSlots) {
    const int i = q0 + tid / kSlots;
    if (i >= Q3) break;
    const long long o = i * a.N + cell;
    asm volatile("prefetch.global.L2 [%0];" ::"l"((const R*)a.lamNext + o));
    asm volatile("prefetch.global.L2 [%0];" ::"l"((const R*)a.f + (o - a.off[i])));
  }
}

// The flagged fluid cells (faces, inlet, outlet, body), kSlowCells per block in three phases:
// (cell, direction) items pull through the cells' records into shared memory; one thread per cell
// applies the transposed Jacobian of its collision (or of the outlet equilibrium; the inlet only
// feeds dJ/du_n); (cell, direction) items push the plain pulls' adjoints and store the links'
// adjoints (with dJ/dq of Bouzidi links). A thread's five items share a cell; their loads go out
// together, and what the last phase needs of them stays in registers.
constexpr int kSlowCells = 32;

template <class R>
__device__ __forceinline__ double adj_slow_role(const AdjLaunch3& a, int block, int tid) {
  constexpr int kItems = (Q3 * kSlowCells + kAdjThreads - 1) / kAdjThreads;
  constexpr int kDirs = kAdjThreads / kSlowCells;  // directions a round of the block's threads covers
  __shared__ R sg[Q3][kSlowCells + 1];
  __shared__ R slp[Q3][kSlowCells + 1];
  __shared__ R slg[Q3][kSlowCells + 1];
  const int N = (int)a.N;
  const int n = a.nSlow;
  const int c = tid % kSlowCells, i0 = tid / kSlowCells;
  const int s = block * kSlowCells + c;
  const bool on = s < n;
  const R* __restrict__ f = (const R*)a.f;
  const R* __restrict__ lamNext = (const R*)a.lamNext;
  R* __restrict__ lamOut = (R*)a.lamOut;
  const R* sA1 = (const R*)a.sA1;
  const R* sA2 = (const R*)a.sA2;
  const int idx = on ? a.slowCells[s] : 0;
  const uint32_t fl = on ? a.flags[idx] : FLAG3_INLET;
  int e[kItems], tgt[kItems];
  R fj[kItems], f2[kItems], lp[kItems];
#pragma unroll
  for (int k = 0; k < kItems; k++) {
    const int i = i0 + k * kDirs;
    const bool item = on && i < Q3;
    e[k] = item ? a.sE1[i * n + s] : 0;
    tgt[k] = item ? a.sTgt[i * n + s] : 0;
  }
#pragma unroll
  for (int k = 0; k < kItems; k++) {
    fj[k] = f[e[k] & 0x7fffffff];
    f2[k] = R(0);
  }
  adj_wait();
#pragma unroll
  for (int k = 0; k < kItems; k++) {
    const int i = i0 + k * kDirs;
    lp[k] = on && i < Q3 ? __ldcg(&lamNext[i * N + idx]) : R(0);
  }
#pragma unroll
  for (int k = 0; k < kItems; k++) {
    const int i = i0 + k * kDirs;
    if (!on || i >= Q3) continue;
    slp[i][c] = lp[k];
    R v = fj[k];  // one source with coefficient 1: plain pulls, copies, mirrors, bounce-back
    if (e[k] < 0) {  // Bouzidi interpolation: two sources
      const int r = i * n + s;
      f2[k] = f[a.sE2[r]];
      v = sA1[r] * v + sA2[r] * f2[k];
    }
    sg[i][c] = v;
  }
  __syncthreads();
  double du = 0.0;
  if (tid < kSlowCells && on) {
    R g[Q3], lpc[Q3], lg[Q3];
#pragma unroll
    for (int i = 0; i < Q3; i++) {
      g[i] = sg[i][tid];
      lpc[i] = slp[i][tid];
    }
    const R u = (R)a.u;
    if (fl & FLAG3_INLET) {
      // f' = feq(1, u, 0, 0): d/du = w_i (3 c_ix + 9 c_ix^2 u - 3 u); the inlet reads nothing
      R sum = R(0);
#pragma unroll
      for (int i = 0; i < Q3; i++) {
        const R cx = R(cx3(i));
        sum += lpc[i] * w3<R>(i) * (R(3) * cx + R(9) * cx * cx * u - R(3) * u);
        lg[i] = R(0);
      }
      du = (double)sum;
    } else if (fl & FLAG3_OUTLET) {
      outlet_adjoint3<R>(g, lpc, lg);
    } else {
      const R* xt = (const R*)a.xTab + 4 * (idx % a.W);
      R dut = R(0);
      collide_adjoint3<R>(g, lpc, xt[0], xt[1], xt[2], u, lg, dut);
      du = (double)dut;
    }
#pragma unroll
    for (int i = 0; i < Q3; i++) slg[i][tid] = lg[i];
  }
  __syncthreads();
  if (!(fl & FLAG3_INLET)) {
    const R w = (R)a.w;
#pragma unroll
    for (int k = 0; k < kItems; k++) {
      const int i = i0 + k * kDirs;
      if (i >= Q3) continue;
      const R v = slg[i][c];
      if (tgt[k] >= 0) {  // a plain pull: the element's only regular reader
        lamOut[tgt[k]] = v;
      } else {            // a link: its adjoint, and dJ/dq of a Bouzidi link
        const int l = -tgt[k] - 1;
        ((R*)a.lamG)[l] = v;
        const int qk = e[k] < 0 ? a.lqk[l] : 0;  // only a two-source pull depends on q
        if (qk) {
          const R q = ((const R*)a.lq)[l];
          const R dgdq = qk == 1 ? R(2) * (fj[k] - f2[k]) : (f2[k] - fj[k]) / (R(2) * q * q);
          a.dqAcc[l] += (double)((v + w * ((const R*)a.lcF)[l]) * dgdq);
        }
      }
    }
  }
  return du;
}

// PAIR: f32 with an even width. Five blocks per SM for f32 (up to 102 registers).
template <class R, bool PAIR>
__global__ void __launch_bounds__(kAdjThreads, PAIR ? 4 : (sizeof(R) == 4 ? 5 : 3)) adj_step3_kernel(AdjLaunch3 a) {
  __shared__ double red[kAdjThreads / 32];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int tid = threadIdx.x + blockDim.x * threadIdx.y;
  const int slice = a.slice0 + blockIdx.z;
  if (slice < a.roleZ) {
    const int r = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * slice);
    if (r >= a.nSlowBlocks + a.nFaceBlocks) return;
    double du = 0.0;
    if (r < a.nSlowBlocks) {
      du = adj_slow_role<R>(a, r, tid);
    } else if constexpr (PAIR) {
      du = adj_face_pairs_role(a, r - a.nSlowBlocks);
    }
    block_du_partial(du, a.blockPart, a.nCellBlocks + r, red, tid);
  } else {
    const int tz = slice - a.roleZ;
    if (tz + 1 < a.D - 2) adj_prefetch<R, (PAIR ? 2 : 1) * kAdjTileX>(a, tz + 1, tid);
    double du;
    if constexpr (PAIR)
      du = adj_pairs_role(a, tz);
    else
      du = adj_cells_role<R>(a, tz);
    block_du_partial(du, a.blockPart, blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * tz), red, tid);
  }
}

// Elements with an irregular reader or no regular reader: lambda^n[e] (= 0 when no regular reader
// wrote it) plus each link's adjoint times its coefficient, plus the direct force terms.
template <class R>
__global__ void __launch_bounds__(256) adj_rows3_kernel(AdjLaunch3 a) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  const bool on = r < a.nRows;
  // the row's own record does not depend on the step before: it goes out before the wait, with the first
  // entries (few rows have more)
  constexpr int kHead = 4;
  const int e = on ? a.rowElem[r] : 0;
  const int k0 = on ? a.rowStart[r] : 0, k1 = on ? a.rowStart[r + 1] : 0;
  const bool set = on && a.rowSet[r];
  const R phi = on ? ((const R*)a.rowPhi)[r] : R(0);
  const R* lamG = (const R*)a.lamG;
  const R* lcF = (const R*)a.lcF;
  const R* alpha = (const R*)a.entAlpha;
  int link[kHead];
  R al[kHead], cF[kHead];
#pragma unroll
  for (int k = 0; k < kHead; k++) {
    link[k] = k0 + k < k1 ? a.entLink[k0 + k] : 0;
    al[k] = k0 + k < k1 ? alpha[k0 + k] : R(0);
  }
#pragma unroll
  for (int k = 0; k < kHead; k++) cF[k] = k0 + k < k1 ? lcF[link[k]] : R(0);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (!on) return;
  R* lamOut = (R*)a.lamOut;
  const R w = (R)a.w;
  R v = set ? R(0) : lamOut[e];
  R lam[kHead];
#pragma unroll
  for (int k = 0; k < kHead; k++) lam[k] = k0 + k < k1 ? lamG[link[k]] : R(0);
#pragma unroll
  for (int k = 0; k < kHead; k++)
    if (k0 + k < k1) v += al[k] * (lam[k] + w * cF[k]);
  for (int k = k0 + kHead; k < k1; k++) {
    const int L = a.entLink[k];
    v += alpha[k] * (lamG[L] + w * lcF[L]);
  }
  v += w * phi;
  lamOut[e] = v;
}

// After a segment: dJ/du_n of its steps, one block each, from the steps' block sums (strided per
// thread, then in order).
__global__ void __launch_bounds__(256) adj_du3_kernel(const double* __restrict__ part, int nParts,
                                                      double* __restrict__ dudn) {
  __shared__ double red[8];
  const double* p = part + (size_t)blockIdx.x * nParts;
  double s = 0.0;
  for (int k = threadIdx.x; k < nParts; k += 256) s += p[k];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int k = 0; k < 8; k++) t += red[k];
    dudn[blockIdx.x] = t;
  }
}

// A programmatic dependent of the launch before it, or (dependent = false) an ordinary launch.
template <class... Args>
cudaError_t launch_dependent(void (*fn)(Args...), dim3 grid, dim3 block, cudaStream_t s, bool dependent, Args... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = dependent ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, fn, args...);
}

constexpr unsigned kMaxSlices = 65535;  // of a grid's z

// Interior-cell blocks of a step: x tiles of 32 cells (or 32 x-pairs), so each warp still reads
// 128-byte rows and the tiles before the absorbing layer take the collision code without it.
bool adj_pairs(int precision, int W) { return precision == 0 && W % 2 == 0; }

dim3 adj_cell_grid(int precision, int W, int H, int D) {
  const int tileY = kAdjThreads / kAdjTileX, tileX = adj_pairs(precision, W) ? 2 * kAdjTileX : kAdjTileX;
  const unsigned gx = (unsigned)((W + tileX - 1) / tileX);
  if (H < 3 || D < 3) return dim3(gx, 1, 0);  // every cell is flagged
  return dim3(gx, (unsigned)((H - 2 + tileY - 1) / tileY), (unsigned)(D - 2));
}

// Blocks of the face rows: tiles of the two z planes, and of the two y rows of the planes between.
int adj_face_blocks(int precision, int W, int H, int D, dim3 cells) {
  if (!adj_pairs(precision, W) || H < 3 || D < 3) return 0;
  const int rows = kAdjThreads / kAdjTileX;
  return (int)(2 * cells.x * cells.y + 2 * cells.x * ((D - 2 + rows - 1) / rows));
}

template <class R>
cudaError_t launch_adjoint_step3_t(AdjLaunch3 a, bool first, cudaStream_t s) {
  const int precision = sizeof(R) == 4 ? 0 : 3;
  const dim3 cells = adj_cell_grid(precision, a.W, a.H, a.D);
  a.nCellBlocks = (int)(cells.x * cells.y * cells.z);
  for (int i = 0; i < Q3; i++) a.off[i] = (int)off3(i, a.W, a.H);
  a.nSlowBlocks = (a.nSlow + kSlowCells - 1) / kSlowCells;
  a.nFaceBlocks = adj_face_blocks(precision, a.W, a.H, a.D, cells);
  if (a.nCellBlocks + a.nSlowBlocks + a.nFaceBlocks != a.nParts) return cudaErrorInvalidValue;
  for (int side = 0; side < 4; side++) {
    for (int i = 0; i < Q3; i++) {
      const bool out = side == 0 ? cz3(i) == 1 : (side == 1 ? cz3(i) == -1 : (side == 2 ? cy3(i) == 1 : cy3(i) == -1));
      const int pop = !out ? i : (side < 2 ? mirror_z3(i) : mirror_y3(i));
      const int off = !out ? a.off[i] : (side < 2 ? cx3(i) + a.W * cy3(i) : cx3(i) + a.W * a.H * cz3(i));
      a.foff[side][i] = (int)((long long)pop * a.N - off);
    }
  }
  const unsigned slice = cells.x * cells.y;
  a.roleZ = (int)(((unsigned)(a.nSlowBlocks + a.nFaceBlocks) + slice - 1) / slice);
  void (*fn)(AdjLaunch3) = adj_step3_kernel<R, false>;
  if constexpr (sizeof(R) == 4) {
    if (adj_pairs(precision, a.W)) fn = adj_step3_kernel<R, true>;
  }
  // a launch takes 65,535 slices: a thin grid of some 20,000 planes has more
  const unsigned slices = a.roleZ + cells.z;
  for (unsigned z0 = 0; z0 < slices; z0 += kMaxSlices) {
    a.slice0 = (int)z0;
    const cudaError_t e = launch_dependent(fn, dim3(cells.x, cells.y, std::min(slices - z0, kMaxSlices)),
                                           dim3(kAdjTileX, kAdjThreads / kAdjTileX), s, !first || z0 > 0, a);
    if (e != cudaSuccess) return e;
  }
  if (a.nRows == 0) return cudaSuccess;
  return launch_dependent(adj_rows3_kernel<R>, dim3((unsigned)((a.nRows + 255) / 256)), dim3(256), s, true, a);
}

}  // namespace

namespace cells {
cudaError_t launch_adjoint_step3(int precision, const AdjLaunch3& a, bool first, cudaStream_t s) {
  if (precision == 0) return launch_adjoint_step3_t<float>(a, first, s);
  if (precision == 3) return launch_adjoint_step3_t<double>(a, first, s);
  return cudaErrorInvalidValue;
}
}  // namespace cells

// ---------------- the recorded run's tables, built on the device ----------------
//
// Once per recorded run (on the host they took 50 ms of a 128x64x64 gradient, more than the forward
// run of 1,000 steps). The links follow the rules of pullSlow3 (src/shaders/step3d.ts:119-168).
// Rows gather what several readers, or a reader with a coefficient, send to one element; their order
// is of no account, and each row adds its entries in link order.

namespace {

// Whether a flagged fluid cell is listed: all but those adj_face_pairs_role takes.
__device__ __forceinline__ bool adj_listed(const AdjTables3& t, int x, int y, int z, uint32_t fl) {
  if (fl == 0u || (fl & FLAG3_SOLID)) return false;
  const bool zFace = z == 0 || z == t.D - 1, yFace = y == 0 || y == t.H - 1;
  const bool face = t.facePairs && zFace != yFace && x > 0 && x < t.W - 1 && !t.rowBody[y + t.H * z];
  return !face;
}

// Listed cells of each row, one warp per row: their number, or with `offset` the cells themselves.
__global__ void adj_list3_kernel(AdjTables3 t, int* __restrict__ counts, const int* __restrict__ offset,
                                 int* __restrict__ cells) {
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (row >= t.H * t.D) return;
  const int z = row / t.H, y = row - z * t.H;
  int n = offset ? offset[row] : 0;
  for (int x0 = 0; x0 < t.W; x0 += 32) {
    const int x = x0 + lane;
    const bool in = x < t.W && adj_listed(t, x, y, z, t.flags[x + t.W * row]);
    const unsigned m = __ballot_sync(0xffffffffu, in);
    if (in && offset) cells[n + __popc(m & ((1u << lane) - 1u))] = x + t.W * row;
    n += __popc(m);
  }
  if (!offset && lane == 0) counts[row] = n;
}

// Links of each listed cell: its flagged directions (the inlet reads nothing).
__global__ void adj_link_count3_kernel(AdjTables3 t, const int* __restrict__ cells, int n, int* __restrict__ counts) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  const uint32_t fl = t.flags[cells[c]];
  counts[c] = (fl & FLAG3_INLET) ? 0 : __popc(fl & (((1u << Q3) - 1u) & ~1u));
}

// Exclusive scan of n counts by one block, in place; the total to counts[n].
__global__ void __launch_bounds__(1024) adj_scan3_kernel(int* __restrict__ counts, int n) {
  __shared__ int warpSum[32];
  __shared__ int carry;
  const int tid = threadIdx.x, lane = tid & 31;
  if (tid == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < n; base += 1024) {
    const int k = base + tid;
    const int v = k < n ? counts[k] : 0;
    int s = v;
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += u;
    }
    if (lane == 31) warpSum[tid >> 5] = s;
    __syncthreads();
    if (tid < 32) {
      int w = warpSum[tid];
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += u;
      }
      warpSum[tid] = w;
    }
    __syncthreads();
    const int before = carry + (tid >= 32 ? warpSum[(tid >> 5) - 1] : 0) + s - v;
    if (k < n) counts[k] = before;
    __syncthreads();
    if (tid == 1023) carry = before + v;
    __syncthreads();
  }
  if (tid == 0) counts[n] = carry;
}

// The pull records of each listed cell's 19 directions and its links, one thread per cell; every link's
// sources are counted into cnt (per element).
template <class R>
__global__ void adj_links3_kernel(AdjTables3 t, AdjLaunch3 a, const int* __restrict__ linkBase, AdjLinkQ3* __restrict__ linkQ,
                                  int* __restrict__ sE1, int* __restrict__ sE2, int* __restrict__ sTgt,
                                  R* __restrict__ sA1, R* __restrict__ sA2, R* __restrict__ lcF, R* __restrict__ lq,
                                  signed char* __restrict__ lqk, int* __restrict__ cnt) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = a.nSlow;
  if (c >= n) return;
  const int W = t.W, H = t.H, D = t.D;
  const int N = (int)t.N;  // 19 N < 2^31
  const int idx = a.slowCells[c];
  const int z = idx / (W * H), y = idx / W - z * H, x = idx % W;
  const uint32_t fl = t.flags[idx];
  const bool inlet = (fl & FLAG3_INLET) != 0u, outlet = (fl & FLAG3_OUTLET) != 0u;
  auto at = [&](int qx, int qy, int qz) { return qx + W * (qy + H * qz); };
  auto solid = [&](int cell) { return (t.flags[cell] & FLAG3_SOLID) != 0u; };
  int k = linkBase[c];
  for (int i = 0; i < Q3; i++) {
    const int r = i * n + c;
    if (inlet) {  // the inlet reads nothing
      sE1[r] = sE2[r] = sTgt[r] = 0;
      sA1[r] = sA2[r] = R(0);
      continue;
    }
    if (i == 0 || !(fl & (1u << i))) {
      const int e = i * N + idx - a.off[i];
      sE1[r] = sE2[r] = sTgt[r] = e;
      sA1[r] = R(1);
      sA2[r] = R(0);
      continue;
    }
    const int j = opp3(i);
    const int sx = x - cx3(i), sy = y - cy3(i), sz = z - cz3(i);
    const bool outX = sx < 0 || sx >= W, outY = sy < 0 || sy >= H, outZ = sz < 0 || sz >= D;
    const int comp = t.component;
    const int cc = comp == 0 ? cx3(j) : (comp == 1 ? cy3(j) : cz3(j));
    int e1, e2 = -1, cF = 0, qKind = 0;
    R a1 = R(1), a2 = R(0), q = R(0);
    AdjLinkQ3 Q{0.0, 0.0, -1, -1};
    if (outX && outlet) {
      e1 = i * N + at(W - 2, y, z);
    } else if (outY && outZ) {
      e1 = j * N + idx;
    } else if (outY || outZ) {
      const int rs = at(sx, outY ? y : sy, outY ? sz : z);
      if (solid(rs)) {  // a body meets a slip face: bounce-back with force 2 c_j f_j
        e1 = j * N + idx;
        cF = cc;
      } else {
        e1 = (outY ? mirror_y3(i) : mirror_z3(i)) * N + rs;
      }
    } else if (outX) {
      e1 = j * N + idx;
    } else {
      const int s = at(sx, sy, sz);
      if (!solid(s)) {
        e1 = i * N + s;
      } else {
        // Bouzidi: q in the arithmetic type, as the step kernel computes it
        const R dF = (R)t.sdf[idx], dS = (R)t.sdf[s];
        const R den = max(dF - dS, (R)1e-6);
        const R raw = dF / den;
        q = min(max(raw, (R)1e-3), R(1));
        e1 = j * N + idx;
        cF = cc;
        Q.cell = idx;
        Q.solid = s;
        if (raw > (R)1e-3 && raw < R(1) && (dF - dS) > (R)1e-6) {
          Q.dqdF = -(double)dS / ((double)den * (double)den);
          Q.dqdS = (double)dF / ((double)den * (double)den);
        }
        if (q < R(0.5)) {
          const int nx = x + cx3(i), ny = y + cy3(i), nz = z + cz3(i);
          if (nx >= 0 && nx < W && ny >= 0 && ny < H && nz >= 0 && nz < D && !solid(at(nx, ny, nz))) {
            a1 = R(2) * q;
            e2 = j * N + at(nx, ny, nz);
            a2 = R(1) - R(2) * q;
            qKind = 1;
          }
        } else {
          a1 = R(1) / (R(2) * q);
          e2 = i * N + idx;
          a2 = (R(2) * q - R(1)) / (R(2) * q);
          qKind = 2;
        }
        if (qKind == 0) Q.solid = -1;  // its pull does not depend on q
      }
    }
    // one source with coefficient 1 is the plain index; else the sign bit marks the two sources
    sE1[r] = e2 < 0 ? e1 : (int)((uint32_t)e1 | 0x80000000u);
    sE2[r] = e2 >= 0 ? e2 : e1;
    sA1[r] = a1;
    sA2[r] = a2;
    sTgt[r] = -(k + 1);
    lcF[k] = (R)cF;
    lq[k] = q;
    lqk[k] = (signed char)qKind;
    linkQ[k] = Q;
    atomicAdd(cnt + e1, 1);
    if (e2 >= 0) atomicAdd(cnt + e2, 1);
    k++;
  }
}

// Whether a plain store writes element e's adjoint: its regular reader is a fluid cell that pulls e's
// direction without a rule, or e leaves the grid through a slip face and the cell that pulls its mirror
// image is one of adj_face_pairs_role's.
__device__ __forceinline__ bool adj_regular(const AdjTables3& t, int e) {
  const int i = e / (int)t.N, cell = e - i * (int)t.N;
  const int z = cell / (t.W * t.H), y = cell / t.W - z * t.H, x = cell % t.W;
  const int rx = x + cx3(i), ry = y + cy3(i), rz = z + cz3(i);
  if (rx < 0 || rx >= t.W) return false;
  const bool outY = ry < 0 || ry >= t.H, outZ = rz < 0 || rz >= t.D;
  if (outY || outZ) {
    if (!t.facePairs || (outY && outZ)) return false;
    const int my = outY ? y : ry, mz = outZ ? z : rz;
    const uint32_t m = t.flags[rx + t.W * (my + t.H * mz)];
    return m != 0u && !(m & FLAG3_SOLID) && !adj_listed(t, rx, my, mz, m);
  }
  const uint32_t g = t.flags[rx + t.W * (ry + t.H * rz)];
  return !(g & (FLAG3_SOLID | FLAG3_INLET)) && (i == 0 || !(g & (1u << i)));
}

// Links whose only source has no other reader store their adjoint there (their target becomes the
// element). The elements of the others become rows: the first of an element's readers to come takes
// the row's number. Elements that nothing reads keep the zero of the cleared adjoint states.
template <class R>
__global__ void adj_claim3_kernel(AdjTables3 t, int n, const int* __restrict__ sE1, const int* __restrict__ sE2,
                                  int* __restrict__ sTgt, const R* __restrict__ lcF, const int* __restrict__ cnt,
                                  int* __restrict__ rowOf, int* __restrict__ rowElem, int* __restrict__ rowStart,
                                  int* __restrict__ nRows) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
  if (c >= n) return;
  const int r = i * n + c;
  if (sTgt[r] >= 0) return;
  const bool two = sE1[r] < 0;
  const int e1 = sE1[r] & 0x7fffffff;
  if (!two && cnt[e1] == 1 && lcF[-sTgt[r] - 1] == R(0) && !adj_regular(t, e1)) {
    sTgt[r] = e1;
    return;
  }
  for (int s = 0; s < (two ? 2 : 1); s++) {
    const int e = s ? sE2[r] : e1;
    if (atomicCAS(rowOf + e, 0, -1) != 0) continue;
    const int row = atomicAdd(nRows, 1);
    rowElem[row] = e;
    rowStart[row] = cnt[e];
    rowOf[e] = row + 1;
  }
}

template <class R>
__global__ void adj_entries3_kernel(int n, const int* __restrict__ sE1, const int* __restrict__ sE2,
                                    const int* __restrict__ sTgt, const R* __restrict__ sA1, const R* __restrict__ sA2,
                                    const int* __restrict__ rowOf, const int* __restrict__ rowStart,
                                    int* __restrict__ fill, int* __restrict__ entLink, R* __restrict__ entAlpha) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
  if (c >= n) return;
  const int r = i * n + c;
  if (sTgt[r] >= 0) return;
  const bool two = sE1[r] < 0;
  for (int s = 0; s < (two ? 2 : 1); s++) {
    const int row = rowOf[s ? sE2[r] : (sE1[r] & 0x7fffffff)] - 1;
    const int p = rowStart[row] + atomicAdd(fill + row, 1);
    entLink[p] = -sTgt[r] - 1;
    entAlpha[p] = s ? sA2[r] : (two ? sA1[r] : R(1));
  }
}

// Each row's entries in link order (a row has a handful), the sum of its force links' coefficients
// (those that read the element as f_j, their first source), and whether a plain pull writes it.
template <class R>
__global__ void adj_rows_build3_kernel(AdjTables3 t, int nRows, const int* __restrict__ rowElem,
                                       const int* __restrict__ rowStart, int* __restrict__ entLink,
                                       R* __restrict__ entAlpha, const int* __restrict__ le1, const R* __restrict__ lcF,
                                       R* __restrict__ rowPhi, unsigned char* __restrict__ rowSet) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= nRows) return;
  const int k0 = rowStart[row], k1 = rowStart[row + 1], e = rowElem[row];
  for (int k = k0 + 1; k < k1; k++) {
    const int l = entLink[k];
    const R al = entAlpha[k];
    int q = k;
    for (; q > k0 && entLink[q - 1] > l; q--) {
      entLink[q] = entLink[q - 1];
      entAlpha[q] = entAlpha[q - 1];
    }
    entLink[q] = l;
    entAlpha[q] = al;
  }
  double phi = 0.0;
  for (int k = k0; k < k1; k++)
    if (le1[entLink[k]] == e) phi += (double)lcF[entLink[k]];
  rowPhi[row] = (R)phi;
  rowSet[row] = adj_regular(t, e) ? 0 : 1;
}

// First source of each link, for adj_rows_build3_kernel.
__global__ void adj_first_source3_kernel(int n, const int* __restrict__ sE1, const int* __restrict__ sTgt,
                                         int* __restrict__ le1) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
  if (c >= n) return;
  const int r = i * n + c;
  if (sTgt[r] < 0) le1[-sTgt[r] - 1] = sE1[r] & 0x7fffffff;
}

// A device buffer of the recorded run: from the handle's table block while it has room (256-byte
// aligned), else a buffer of its own that the run frees.
void* adj_alloc(Cells3D* h, Adjoint3D* A, size_t bytes, const char* what) {
  bytes = (std::max<size_t>(bytes, 1) + 255) / 256 * 256;
  A->tabNeed += bytes;
  if (h->adjTab && A->tabUsed + bytes <= h->adjTabBytes) {
    void* p = (char*)h->adjTab + A->tabUsed;
    A->tabUsed += bytes;
    return p;
  }
  void* p = h->dev.alloc(bytes, what);
  A->own.push_back(p);
  return p;
}

// Makes the handle's table block hold `bytes` (with room for a somewhat larger body next time),
// before the run has taken anything from it; without the memory for it the run's buffers are
// allocated one by one.
void reserve_adj_tables(Cells3D* h, Adjoint3D* A, size_t bytes) {
  if (h->adjTabBytes >= bytes || A->tabUsed != 0) return;
  if (h->adjTab) h->dev.release(h->adjTab);
  h->adjTab = nullptr;
  h->adjTabBytes = 0;
  const size_t want = bytes + bytes / 8 + ((size_t)1 << 20);
  if (want + (size_t)h->N * 16 < h->dev.free_bytes()) {
    h->adjTab = h->dev.alloc(want, "adjoint tables");
    h->adjTabBytes = want;
  }
}

void release_adjoint(Cells3D* h) {
  if (!h->adj) return;
  Adjoint3D* A = h->adj.get();
  // the checkpoints, recompute buffers and adjoint states live in h->adjStore and the tables in
  // h->adjTab, which both stay; only the run's own buffers go
  if (!h->dev.fake) h->dev.sync();
  if (A->side2) cudaStreamSynchronize(A->side2);
  if (A->fork2) cudaEventDestroy(A->fork2);
  if (A->join2) cudaEventDestroy(A->join2);
  if (A->side2) cudaStreamDestroy(A->side2);
  for (void* p : A->own) h->dev.release(p);
  h->adj.reset();
}

// Block sums of one adjoint step.
int adj_parts(const Cells3D* h, int nSlow) {
  const dim3 cells = adj_cell_grid(h->prec, h->W, h->H, h->D);
  return (int)(cells.x * cells.y * cells.z) + (nSlow + kSlowCells - 1) / kSlowCells +
         adj_face_blocks(h->prec, h->W, h->H, h->D, cells);
}

unsigned blocks_of(size_t n, unsigned b) { return (unsigned)((n + b - 1) / b); }

// The list of flagged cells, their pull records, the links and the rows for the current flags and SDF.
// Three ints come back to the host: the numbers of cells, links and rows. The per-element scratch (cnt and rowOf, a
// count and a row number per population element) lies in the two adjoint states: a backward sweep has to clear them
// before it starts, as it does.
template <class R>
void build_tables(Cells3D* h, Adjoint3D* A, int* cnt, int* rowOf) {
  cells::Device& dev = h->dev;
  cudaStream_t st = dev.stream;
  const int W = h->W, H = h->H, D = h->D, nRowsXY = H * D;
  AdjTables3 t;
  t.flags = h->flags;
  t.sdf = h->sdf;
  t.rowBody = h->rowBody;
  t.N = h->N;
  t.W = W;
  t.H = H;
  t.D = D;
  t.component = A->component;
  t.facePairs = adj_face_blocks(h->prec, W, H, D, adj_cell_grid(h->prec, W, H, D)) > 0;
  // the cell list, and the links of each cell, counted and scanned in scratch
  int* rowCount = rowOf;                     // H D + 1
  adj_list3_kernel<<<blocks_of((size_t)nRowsXY * 32, 256), 256, 0, st>>>(t, rowCount, nullptr, nullptr);
  adj_scan3_kernel<<<1, 1024, 0, st>>>(rowCount, nRowsXY);
  int host[2] = {0, 0};
  dev.d2h(host, rowCount + nRowsXY, 4);
  dev.sync();
  A->nSlow = host[0];
  const size_t ns = (size_t)A->nSlow, nsr = std::max<size_t>(1, 19 * ns);
  int* cells = cnt;                          // the list, then each cell's first link (n + 1)
  int* linkBase = cnt + ns;
  adj_list3_kernel<<<blocks_of((size_t)nRowsXY * 32, 256), 256, 0, st>>>(t, nullptr, rowCount, cells);
  if (ns) adj_link_count3_kernel<<<blocks_of(ns, 256), 256, 0, st>>>(t, cells, A->nSlow, linkBase);
  adj_scan3_kernel<<<1, 1024, 0, st>>>(linkBase, A->nSlow);
  dev.d2h(host, linkBase + ns, 4);
  dev.sync();
  A->nLinks = host[0];
  const size_t nl = std::max<size_t>(1, (size_t)A->nLinks), ne = 2 * nl;  // at most two entries per link
  {
    // every device buffer of the run, as adj_alloc rounds them (these tables, then the forward
    // run's): the handle's table block grows to hold them all before the first is taken
    auto al = [](size_t b) { return (std::max<size_t>(b, 1) + 255) / 256 * 256; };
    const size_t nSeg = (size_t)((A->steps + A->K - 1) / A->K), rb = sizeof(R);
    const size_t segSteps = (size_t)std::min<int64_t>(A->K, A->steps);
    const size_t need = al(ns * 4) + al((ns + 1) * 4) + 3 * al(nsr * 4) + 2 * al(nsr * rb) + al(nl * 4) + 3 * al(nl * rb) +
                        al(nl) + al(nl * sizeof(AdjLinkQ3)) + al(nl * 8) + 2 * al(ne * 4) + al((ne + 1) * 4) + al(ne) +
                        2 * al(ne * rb) + al(ne * 4) + al(64) + al(nSeg * sizeof(DevState3)) + al(sizeof(DevState3)) +
                        al((size_t)adj_parts(h, A->nSlow) * segSteps * 8) + al((size_t)A->steps * 8);
    reserve_adj_tables(h, A, need);
  }
  A->slowCells = (int*)adj_alloc(h, A, ns * 4, "adjoint flagged cells");
  int* base = (int*)adj_alloc(h, A, (ns + 1) * 4, "adjoint link base");
  A->sE1 = (int*)adj_alloc(h, A, nsr * 4, "adjoint flagged-cell records");
  A->sE2 = (int*)adj_alloc(h, A, nsr * 4, "adjoint flagged-cell records");
  A->sTgt = (int*)adj_alloc(h, A, nsr * 4, "adjoint flagged-cell records");
  A->sA1 = adj_alloc(h, A, nsr * sizeof(R), "adjoint flagged-cell records");
  A->sA2 = adj_alloc(h, A, nsr * sizeof(R), "adjoint flagged-cell records");
  int* le1 = (int*)adj_alloc(h, A, nl * 4, "adjoint links");
  A->lcF = adj_alloc(h, A, nl * sizeof(R), "adjoint links");
  A->lq = adj_alloc(h, A, nl * sizeof(R), "adjoint links");
  A->lqk = (signed char*)adj_alloc(h, A, nl, "adjoint links");
  A->linkQ = (AdjLinkQ3*)adj_alloc(h, A, nl * sizeof(AdjLinkQ3), "adjoint links");
  A->lamG = adj_alloc(h, A, nl * sizeof(R), "adjoint link values");
  A->dqAcc = (double*)adj_alloc(h, A, nl * 8, "adjoint dJ/dq");
  A->rowElem = (int*)adj_alloc(h, A, ne * 4, "adjoint rows");
  int* fill = (int*)adj_alloc(h, A, ne * 4, "adjoint rows");
  A->rowStart = (int*)adj_alloc(h, A, (ne + 1) * 4, "adjoint rows");
  A->rowSet = (unsigned char*)adj_alloc(h, A, ne, "adjoint rows");
  A->rowPhi = adj_alloc(h, A, ne * sizeof(R), "adjoint rows");
  A->entAlpha = adj_alloc(h, A, ne * sizeof(R), "adjoint rows");
  A->entLink = (int*)adj_alloc(h, A, ne * 4, "adjoint rows");
  int* nRows = (int*)adj_alloc(h, A, 64, "adjoint rows");
  A->nRows = 0;
  if (ns) {
    check_cuda(cudaMemcpyAsync(A->slowCells, cells, ns * 4, cudaMemcpyDeviceToDevice, st), "adjoint cell list");
    check_cuda(cudaMemcpyAsync(base, linkBase, (ns + 1) * 4, cudaMemcpyDeviceToDevice, st), "adjoint link base");
    dev.memset0(cnt, 19 * (size_t)h->N * 4);
    dev.memset0(rowOf, 19 * (size_t)h->N * 4);
    dev.memset0(nRows, 4);
    dev.memset0(fill, ne * 4);
    AdjLaunch3 a;
    std::memset(&a, 0, sizeof(a));
    a.nSlow = A->nSlow;
    a.slowCells = A->slowCells;
    for (int i = 0; i < Q3; i++) a.off[i] = (int)off3(i, W, H);
    const dim3 items(blocks_of(ns, 256), Q3);
    adj_links3_kernel<R><<<blocks_of(ns, 128), 128, 0, st>>>(t, a, base, A->linkQ, A->sE1, A->sE2, A->sTgt, (R*)A->sA1,
                                                             (R*)A->sA2, (R*)A->lcF, (R*)A->lq, A->lqk, cnt);
    adj_first_source3_kernel<<<items, 256, 0, st>>>(A->nSlow, A->sE1, A->sTgt, le1);
    adj_claim3_kernel<R><<<items, 256, 0, st>>>(t, A->nSlow, A->sE1, A->sE2, A->sTgt, (const R*)A->lcF, cnt, rowOf,
                                                A->rowElem, A->rowStart, nRows);
    check_cuda(cudaGetLastError(), "adjoint table kernels");
    dev.d2h(host, nRows, 4);
    dev.sync();
    A->nRows = host[0];
    if (A->nRows > 0) {
      adj_scan3_kernel<<<1, 1024, 0, st>>>(A->rowStart, A->nRows);
      adj_entries3_kernel<R><<<items, 256, 0, st>>>(A->nSlow, A->sE1, A->sE2, A->sTgt, (const R*)A->sA1,
                                                    (const R*)A->sA2, rowOf, A->rowStart, fill, A->entLink,
                                                    (R*)A->entAlpha);
      adj_rows_build3_kernel<R><<<blocks_of((size_t)A->nRows, 256), 256, 0, st>>>(
          t, A->nRows, A->rowElem, A->rowStart, A->entLink, (R*)A->entAlpha, le1, (const R*)A->lcF, (R*)A->rowPhi,
          A->rowSet);
    }
  }
  check_cuda(cudaGetLastError(), "adjoint table kernels");
  dev.launches += 10;
}

}  // namespace

namespace {

// The launch arguments of the adjoint step kernels for the recorded run (all but f, the adjoint
// buffers, the block sums and the step's inlet speed and objective weight, which enqueue_sweep sets).
AdjLaunch3 adj_args(Cells3D* h, Adjoint3D* A) {
  AdjLaunch3 a;
  std::memset(&a, 0, sizeof(a));
  a.flags = h->flags;
  a.xTab = h->xTab;
  a.rowBody = h->rowBody;
  a.lcF = A->lcF;
  a.lq = A->lq;
  a.lqk = A->lqk;
  a.lamG = A->lamG;
  a.dqAcc = A->dqAcc;
  a.N = h->N;
  a.W = h->W;
  a.H = h->H;
  a.D = h->D;
  a.absorbX0 = h->absorbX0;
  a.slowCells = A->slowCells;
  a.nSlow = A->nSlow;
  a.sE1 = A->sE1;
  a.sE2 = A->sE2;
  a.sTgt = A->sTgt;
  a.sA1 = A->sA1;
  a.sA2 = A->sA2;
  a.nParts = A->nParts;
  a.nRows = A->nRows;
  a.rowElem = A->rowElem;
  a.rowSet = A->rowSet;
  a.rowStart = A->rowStart;
  a.entLink = A->entLink;
  a.entAlpha = A->entAlpha;
  a.rowPhi = A->rowPhi;
  return a;
}

// Recompute a segment's len states into state set `set` from its checkpoint copy in set[0].
void enqueue_recompute(Cells3D* h, Adjoint3D* A, int set, int len, int par0, cudaStream_t stream) {
  for (int t = 0; t + 1 < len; t++) {
    h->enqueue_step_between(A->seg[set][(size_t)t], A->seg[set][(size_t)t + 1], par0 ^ (t & 1), false, stream);
    h->dev.launches++;
  }
}

// The adjoint steps of segment sgi (len steps, states in set `set`), from the last to the first,
// starting from adjoint buffer c; the next (earlier) segment's recompute into the other set, when there
// is one, runs beside them on side2.
void enqueue_sweep(Cells3D* h, Adjoint3D* A, AdjLaunch3& a, int64_t sgi, int set, int len, int c, bool next,
                   int nextLen, int nextPar0, bool terminal) {
  cudaStream_t s = h->dev.stream;
  if (next) {
    check_cuda(cudaEventRecord(A->fork2, s), "cudaEventRecord");
    check_cuda(cudaStreamWaitEvent(A->side2, A->fork2, 0), "cudaStreamWaitEvent");
  }
  for (int t = len - 1; t >= 0; t--) {
    const int64_t n = sgi * A->K + t, label = A->s0 + n + 1;
    a.f = A->seg[set][(size_t)t];
    a.lamNext = A->lam[c];
    a.lamOut = A->lam[c ^ 1];
    a.blockPart = A->blockPart + (size_t)t * A->nParts;
    a.u = A->uStep[(size_t)n];
    a.w = label >= A->w0 && label <= A->w1 ? A->scale / (double)(A->w1 - A->w0 + 1) : 0.0;
    check_cuda(launch_adjoint_step3(h->prec, a, t == len - 1, s), "adjoint step kernel");
    h->dev.launches += 2;
    // elements that nothing reads keep zero, which a terminal adjoint in the first buffer is not
    if (terminal && n + 1 == A->steps) h->dev.memset0(A->lam[c], 19 * h->bpp * (size_t)h->N);
    c ^= 1;
    // the recompute's steps go out between the adjoint steps, so neither stream waits for the host
    const int k = len - 1 - t;
    if (next && k + 1 < nextLen) {
      h->enqueue_step_between(A->seg[set ^ 1][(size_t)k], A->seg[set ^ 1][(size_t)k + 1], nextPar0 ^ (k & 1), false,
                              A->side2);
      h->dev.launches++;
    }
  }
  if (next) {
    for (int k = len; k + 1 < nextLen; k++) {
      h->enqueue_step_between(A->seg[set ^ 1][(size_t)k], A->seg[set ^ 1][(size_t)k + 1], nextPar0 ^ (k & 1), false,
                              A->side2);
      h->dev.launches++;
    }
    check_cuda(cudaEventRecord(A->join2, A->side2), "cudaEventRecord");
  }
  adj_du3_kernel<<<len, 256, 0, s>>>(A->blockPart, A->nParts, A->dudn + sgi * A->K);
  check_cuda(cudaGetLastError(), "adjoint du kernel");
  h->dev.launches++;
  if (next) check_cuda(cudaStreamWaitEvent(s, A->join2, 0), "cudaStreamWaitEvent");
}

// The state set of segment s: the sweep alternates sets, starting with set 0 at the last segment.
int seg_set(const Adjoint3D* A, int64_t s) {
  const int64_t nSeg = (A->steps + A->K - 1) / A->K;
  return (int)((nSeg - 1 - s) & 1);
}

}  // namespace

// ---------------- C ABI ----------------

#define ADJ_TRY(h) try {
#define ADJ_CATCH(h)                                                         \
  }                                                                          \
  catch (const AllocError& e) {                                              \
    release_adjoint(h);                                                      \
    (h)->lastError = std::string("Solver3D allocation failed: ") + e.what(); \
    return CELLS_E_ALLOC;                                                    \
  }                                                                          \
  catch (const Error& e) {                                                   \
    (h)->lastError = e.what();                                               \
    return e.status;                                                         \
  }                                                                          \
  catch (const std::exception& e) {                                          \
    (h)->lastError = e.what();                                               \
    return CELLS_E_INVALID;                                                  \
  }                                                                          \
  return CELLS_OK;

extern "C" {

int cells3d_adjoint_forward(Cells3D* h, const Cells3DAdjointSpec* spec, double* objective) {
  if (!h || !spec) return CELLS_E_INVALID;
  ADJ_TRY(h)
  if (h->dev.fake) throw Error(CELLS_E_INVALID, "the adjoint needs a CUDA device");
  if (h->prec != CELLS_FP32 && h->prec != CELLS_FP64)
    throw Error(CELLS_E_PRECISION_UNSUPPORTED, "the adjoint runs with FP32 or FP64 storage");
  if (h->cfg.smagorinsky != 0.0) throw Error(CELLS_E_INVALID, "the adjoint supports smagorinsky = 0 only");
  if (spec->steps <= 0 || spec->checkpoint_every <= 0) throw Error(CELLS_E_INVALID, "steps and checkpoint_every must be positive");
  if (spec->component < 0 || spec->component > 2) throw Error(CELLS_E_INVALID, "component must be 0, 1 or 2");
  const int64_t s0 = h->step;
  if (spec->window_begin > spec->window_end || spec->window_begin <= s0 || spec->window_end > s0 + spec->steps)
    throw Error(CELLS_E_INVALID, "the objective window must lie within the recorded steps");
  const int64_t nWin = spec->window_end - spec->window_begin + 1;
  if (nWin > HISTORY_LEN) throw Error(CELLS_E_INVALID, "the objective window exceeds the 8192-sample force ring");
  if (19ll * h->N >= (1ll << 31)) throw Error(CELLS_E_INVALID, "the adjoint supports grids of fewer than 2^31 / 19 cells");
  // the previous run's stream and events carry over (detached here, after their work has finished,
  // so release_adjoint keeps them)
  Adjoint3D carry;
  if (Adjoint3D* old = h->adj.get()) {
    if (old->side2) cudaStreamSynchronize(old->side2);
    std::swap(carry.side2, old->side2);
    std::swap(carry.fork2, old->fork2);
    std::swap(carry.join2, old->join2);
  }
  release_adjoint(h);
  h->adj.reset(new Adjoint3D());
  Adjoint3D* A = h->adj.get();
  std::swap(A->side2, carry.side2);
  std::swap(A->fork2, carry.fork2);
  std::swap(A->join2, carry.join2);
  A->s0 = s0;
  A->steps = spec->steps;
  A->w0 = spec->window_begin;
  A->w1 = spec->window_end;
  A->K = spec->checkpoint_every;
  A->component = spec->component;
  A->scale = spec->scale;
  A->parity0 = h->parity;
  cells::Device& dev = h->dev;
  const size_t fBytes = 19ull * h->bpp * (size_t)h->N;
  const int64_t nSeg = (A->steps + A->K - 1) / A->K;
  const int segBufs = (int)std::min<int64_t>(A->K, A->steps);
  // one block for the checkpoints, both sets of recompute buffers and both adjoint states, each
  // at a 256-byte aligned stride; kept for the next recorded run while it fits
  const size_t stride = (fBytes + 255) / 256 * 256;
  const size_t need = (size_t)(nSeg + 2 * segBufs + 2) * stride;
  if (!h->adjStore || h->adjStoreBytes < need) {
    if (h->adjStore) {
      dev.release(h->adjStore);
      h->adjStore = nullptr;
      h->adjStoreBytes = 0;
    }
    if (need + (size_t)h->N * 16 > dev.free_bytes())
      throw AllocError("the adjoint's checkpoints need " + std::to_string(need) + " bytes; the device has " +
                       std::to_string(dev.free_bytes()) + " free");
    h->adjStore = dev.alloc(need, "adjoint checkpoints");
    h->adjStoreBytes = need;
  }
  char* store = (char*)h->adjStore;
  for (int64_t k = 0; k < nSeg; k++) A->ck.push_back(store + (size_t)k * stride);
  for (int set = 0; set < 2; set++)
    for (int k = 0; k < segBufs; k++) A->seg[set].push_back(store + (size_t)(nSeg + set * segBufs + k) * stride);
  // the per-element scratch: the adjoint states' places, the last two of the store (an f32 element is as wide as a
  // count)
  if (h->prec == CELLS_FP64)
    build_tables<double>(h, A, (int*)(store + (size_t)(nSeg + 2 * segBufs) * stride),
                         (int*)(store + (size_t)(nSeg + 2 * segBufs + 1) * stride));
  else
    build_tables<float>(h, A, (int*)(store + (size_t)(nSeg + 2 * segBufs) * stride),
                        (int*)(store + (size_t)(nSeg + 2 * segBufs + 1) * stride));
  A->ckStateBlock = (DevState3*)adj_alloc(h, A, (size_t)nSeg * sizeof(DevState3), "adjoint checkpoint");
  for (int64_t k = 0; k < nSeg; k++) A->ckState.push_back(A->ckStateBlock + k);
  A->endState = adj_alloc(h, A, sizeof(DevState3), "adjoint end state");
  A->lam[0] = store + (size_t)(nSeg + 2 * segBufs) * stride;
  A->lam[1] = store + (size_t)(nSeg + 2 * segBufs + 1) * stride;
  A->nParts = adj_parts(h, A->nSlow);
  A->blockPart = (double*)adj_alloc(h, A, (size_t)A->nParts * segBufs * 8, "adjoint partials");
  A->dudn = (double*)adj_alloc(h, A, (size_t)A->steps * 8, "adjoint du");
  if (!A->side2) check_cuda(cudaStreamCreateWithFlags(&A->side2, cudaStreamNonBlocking), "cudaStreamCreate");
  if (!A->fork2) check_cuda(cudaEventCreateWithFlags(&A->fork2, cudaEventDisableTiming), "cudaEventCreate");
  if (!A->join2) check_cuda(cudaEventCreateWithFlags(&A->join2, cudaEventDisableTiming), "cudaEventCreate");
  // the recorded run: a checkpoint at the start of every segment, force samples in the window
  const uint64_t written0 = h->forceSamplesRead + h->forceSteps.size();
  A->uStep.resize((size_t)A->steps);
  A->rampStep.resize((size_t)A->steps);
  for (int64_t n = 0; n < A->steps; n++) {
    const int64_t s = s0 + n;
    A->uStep[(size_t)n] = h->uin_at(s);
    A->rampStep[(size_t)n] = h->rampKind ? (h->rampTarget != 0.0 ? h->ramp_speed(s) / h->rampTarget : 0.0) : 1.0;
  }
  // (launched step by step: a step takes the GPU several times as long as its launch takes the host,
  // and capturing K-step graphs anew for every recorded run cost more than they saved)
  int samples = 0;
  const bool split = h->split_run(nWin);
  for (int64_t n = 0; n < A->steps; n++) {
    if (n % A->K == 0) {
      const int64_t k = n / A->K;
      check_cuda(cudaMemcpyAsync(A->ck[(size_t)k], h->f[h->parity], fBytes, cudaMemcpyDeviceToDevice, dev.stream),
                 "checkpoint copy");
      check_cuda(cudaMemcpyAsync(A->ckState[(size_t)k], h->st, sizeof(DevState3), cudaMemcpyDeviceToDevice,
                                 dev.stream),
                 "checkpoint copy");
    }
    const int64_t label = s0 + n + 1;
    const bool sample = label >= A->w0 && label <= A->w1;
    h->enqueue_run_step(sample, n + 1 == A->steps, split, samples);
    h->parity ^= 1;
    h->step++;
    if (sample) h->forceSteps.push_back((uint32_t)h->step);
  }
  check_cuda(cudaMemcpyAsync(A->endState, h->st, sizeof(DevState3), cudaMemcpyDeviceToDevice, dev.stream),
             "end state copy");
  // the objective from the window's samples (ring slots written0 .. written0 + nWin - 1)
  std::vector<double4> hist((size_t)nWin);
  size_t got = 0;
  for (uint64_t k = written0; k < written0 + (uint64_t)nWin;) {
    const size_t r = (size_t)(k % HISTORY_LEN);
    const size_t run = (size_t)std::min<uint64_t>(written0 + nWin - k, (uint64_t)(HISTORY_LEN - r));
    dev.d2h(hist.data() + got, h->history + r, run * sizeof(double4));
    got += run;
    k += run;
  }
  dev.sync();
  double sum = 0.0;
  for (const double4& v : hist) sum += A->component == 0 ? v.x : (A->component == 1 ? v.y : v.z);
  A->objective = A->scale * sum / (double)nWin;
  A->endStep = h->step;
  A->argGen = h->argGen;
  if (objective) *objective = A->objective;
  ADJ_CATCH(h)
}

int cells3d_adjoint_backward(Cells3D* h, const void* terminal_adjoint, double* dJ_dsdf, double* dJ_du_in,
                             void* adjoint_out) {
  if (!h) return CELLS_E_INVALID;
  ADJ_TRY(h)
  Adjoint3D* A = h->adj.get();
  if (!A) throw Error(CELLS_E_INVALID, "adjoint_backward needs a recorded adjoint_forward");
  if (h->step != A->endStep || h->argGen != A->argGen)
    throw Error(CELLS_E_INVALID, "the solver changed after adjoint_forward: record the run again");
  cells::Device& dev = h->dev;
  const long long N = h->N;
  const size_t fBytes = 19ull * h->bpp * (size_t)N;
  dev.memset0(A->lam[0], fBytes);
  dev.memset0(A->lam[1], fBytes);
  dev.memset0(A->dqAcc, (size_t)std::max(1, A->nLinks) * 8);
  dev.memset0(A->dudn, (size_t)A->steps * 8);
  int cur = 0;
  if (terminal_adjoint) {
    dev.h2d(A->lam[0], terminal_adjoint, fBytes);
    dev.sync();
  }
  const int64_t nSeg = (A->steps + A->K - 1) / A->K;
  AdjLaunch3 a = adj_args(h, A);
  // restore a segment's device state and first state (its checkpoint) into its state set
  auto restore = [&](int64_t s) {
    check_cuda(cudaMemcpyAsync(h->st, A->ckState[(size_t)s], sizeof(DevState3), cudaMemcpyDeviceToDevice,
                               dev.stream),
               "checkpoint restore");
    check_cuda(cudaMemcpyAsync(A->seg[seg_set(A, s)][0], A->ck[(size_t)s], fBytes, cudaMemcpyDeviceToDevice,
                               dev.stream),
               "checkpoint restore");
  };
  auto seg_len = [&](int64_t s) { return (int)std::min<int64_t>(A->K, A->steps - s * A->K); };
  auto seg_par0 = [&](int64_t s) { return (int)((A->parity0 + s * A->K) & 1); };
  // the last segment's states first; every other segment's recompute runs beside the sweep of the
  // segment after it
  restore(nSeg - 1);
  enqueue_recompute(h, A, seg_set(A, nSeg - 1), seg_len(nSeg - 1), seg_par0(nSeg - 1), dev.stream);
  for (int64_t sgi = nSeg - 1; sgi >= 0; sgi--) {
    const int len = seg_len(sgi);
    const int set = seg_set(A, sgi);
    const bool next = sgi > 0;
    if (next) restore(sgi - 1);
    enqueue_sweep(h, A, a, sgi, set, len, cur, next, next ? seg_len(sgi - 1) : 0, next ? seg_par0(sgi - 1) : 0,
                  terminal_adjoint != nullptr);
    if (len & 1) cur ^= 1;
  }
  check_cuda(cudaMemcpyAsync(h->st, A->endState, sizeof(DevState3), cudaMemcpyDeviceToDevice, dev.stream),
             "end state restore");
  if (adjoint_out) dev.d2h(adjoint_out, A->lam[cur], fBytes);
  std::vector<double> dq((size_t)std::max(1, A->nLinks)), dudn((size_t)A->steps);
  std::vector<AdjLinkQ3> linkQ((size_t)(dJ_dsdf ? A->nLinks : 0));
  dev.d2h(dq.data(), A->dqAcc, dq.size() * 8);
  dev.d2h(dudn.data(), A->dudn, dudn.size() * 8);
  if (!linkQ.empty()) dev.d2h(linkQ.data(), A->linkQ, linkQ.size() * sizeof(AdjLinkQ3));
  dev.sync();
  if (dJ_dsdf) {
    std::fill(dJ_dsdf, dJ_dsdf + N, 0.0);
    for (int k = 0; k < A->nLinks; k++) {
      const AdjLinkQ3& L = linkQ[(size_t)k];
      if (L.solid < 0) continue;
      dJ_dsdf[L.cell] += dq[(size_t)k] * L.dqdF;
      dJ_dsdf[L.solid] += dq[(size_t)k] * L.dqdS;
    }
  }
  if (dJ_du_in) {
    double s = 0.0;
    for (int64_t n = 0; n < A->steps; n++) s += dudn[(size_t)n] * A->rampStep[(size_t)n];
    *dJ_du_in = s;
  }
  ADJ_CATCH(h)
}

int cells3d_adjoint_release(Cells3D* h) {
  if (!h) return CELLS_E_INVALID;
  ADJ_TRY(h)
  release_adjoint(h);
  if (h->adjStore) {
    h->dev.release(h->adjStore);
    h->adjStore = nullptr;
    h->adjStoreBytes = 0;
  }
  if (h->adjTab) {
    h->dev.release(h->adjTab);
    h->adjTab = nullptr;
    h->adjTabBytes = 0;
  }
  ADJ_CATCH(h)
}

}  // extern "C"
