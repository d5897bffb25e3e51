// Several D2Q9 time steps in one launch: a block loads a tile of one tunnel with a margin of k cells on
// every side into shared memory, steps it k times while the margin shrinks by one cell a step, and
// stores the tile. The margins of neighbouring tiles are computed twice instead of exchanged, so a
// launch needs no communication, and a step costs a block barrier instead of a launch and the
// round trips of its loads.
//
// Boundary rules read within one cell of their own, so they need nothing beyond the margin; a periodic
// seam is a margin loaded from the other side. What a flagged direction pulls is resolved per cell into
// a rule word and Bouzidi coefficients when the SDF is set (rules_of2), because evaluating the
// general rules -- eight directions with dependent flag and SDF loads -- took most of a step: 400x100
// cylinder 5.0 us a step with them. The arithmetic is the one-step kernel's (step2d.cuh); k is odd, so
// a launch ends in the other population buffer as a single step does.
//
// Where every tile is resident at once, a step waits for the tile with the most boundary: with the rules
// inside each cell's code a step of 128x128 cells took 1.1 us without boundaries and 2.7 with a cylinder. There
// (LIST) a block first collects its flagged directions into a list of links; a step works the list off, one
// link per thread, into the places that the pulls read, and then every cell takes the same plain path: 2.05
// us, and 400x100 2.8 -> 2.4. With more tiles than SMs the work counts, and the rules stay with the cells.
//
// Force: a tile's owned cells, each summed link by link, sum in f64 per sampled step (warp shuffles, then
// the warps in order) into one partial per step and tile; after the launches of a run sum_samples2_kernel
// adds the tiles up in order into the ring.
#include <algorithm>

#include "step2d.cuh"

namespace cells {
namespace CELLS_NS {

template <class R>
struct Vec2T;
template <>
struct Vec2T<float> {
  using T = float2;
};
template <>
struct Vec2T<double> {
  using T = double2;
};

template <class C, int RX, int RY>
struct TileSource2 {
  const typename C::S* p;  // population 0 of the cell
  __device__ __forceinline__ typename C::R at(int pop, long long, int, int, int dx, int dy) const {
    return (typename C::R)p[pop * (RX * RY) + dy * RX + dx];
  }
};

// The pulls of the flagged directions by the cell's rule word; fj of a rule i is the cell's population
// opposite to i. coef: the (c1, c2) of the cell's body rules, one per direction.
template <class C, class Source>
__device__ __forceinline__ void rules2(uint32_t w, const Tunnel2& T, const Source& src,
                                       const typename Vec2T<typename C::R>::T* __restrict__ coef, typename C::R (&f)[Q2],
                                       typename C::R force[2]) {
  using R = typename C::R;
#pragma unroll
  for (int i = 1; i < Q2; i++) {
    const uint32_t rule = (w >> (3 * (i - 1))) & 7u;
    if (rule == RULE2_PULL) continue;
    const int j = opp2(i);
    if (rule == RULE2_SLIP || rule == RULE2_SLIP_HERE) {
      f[i] = src.at(mirror_y2(i), 0, 0, 0, rule == RULE2_SLIP ? -cx2(i) : 0, 0);
      continue;
    }
    const R fj = src.at(j, 0, 0, 0, 0, 0);
    R fi = fj;
    if (rule == RULE2_MOVING) {
      f[i] = fj + R(6) * w2<R>(i) * R(cx2(i)) * prm<R>(T, P2_ULID);
      continue;
    }
    if (rule >= RULE2_BODY_N) {
      if (rule != RULE2_BODY_0) {
        const auto c = coef[i - 1];
        if (rule == RULE2_BODY_N)
          fi = c.x * fj + c.y * src.at(j, 0, 0, 0, cx2(i), cy2(i));
        else
          fi = fj / c.x + c.y * src.at(i, 0, 0, 0, 0, 0);
      }
      const R t = fj + fi;
      force[0] += R(cx2(j)) * t;
      force[1] += R(cy2(j)) * t;
    }
    f[i] = fi;
  }
}

// A flagged direction of a tile's cell, collected when the block starts: offsets in the tile's buffer of f_j
// (a, low 15 bits), of the place that the pull reads, population i of x - c_i, solid or outside (a, next 15
// bits), and of the rule's second source (b, low 15 bits); the rule (b, bits 15-17); c_j + 1 in x and y (b, bits
// 18-19 and 20-21); on the first link of a cell whose force counts in this tile, the number of the cell's
// links (b, bits 22-25); and the Bouzidi coefficients, or the moving wall's term in c1.
template <class R>
struct __align__(16) Link2 {
  uint32_t a, b;
  R c1, c2;
};

// Links per tile: what 64 x 48 cells of f32 leave of shared memory, or a tile's walls and a body of its size.
template <int RX, int RY>
constexpr int kTileLinks2 = RX * RY >= 3072 ? 352 : 512;

// The links of the cell at offset c with rule word w, the first of which is number pos.
template <class R, int RX, int RY>
__device__ __forceinline__ void write_links2(Link2<R>* links, int pos, uint32_t w, int c, uint32_t head, R ulid,
                                             const typename Vec2T<R>::T* __restrict__ coef) {
  constexpr int cells = RX * RY;
#pragma unroll
  for (int i = 1; i < Q2; i++) {
    const uint32_t rule = (w >> (3 * (i - 1))) & 7u;
    if (rule == RULE2_PULL) continue;
    const int j = opp2(i);
    int g = j * cells + c;
    if (rule == RULE2_SLIP) g = mirror_y2(i) * cells + c - cx2(i);
    if (rule == RULE2_SLIP_HERE) g = mirror_y2(i) * cells + c;
    if (rule == RULE2_BODY_N) g = j * cells + c + cy2(i) * RX + cx2(i);
    if (rule == RULE2_BODY_H) g = i * cells + c;
    Link2<R> L;
    L.a = (uint32_t)(j * cells + c) | (uint32_t)(i * cells + c - cy2(i) * RX - cx2(i)) << 15;
    L.b = (uint32_t)g | rule << 15 | (uint32_t)(cx2(j) + 1) << 18 | (uint32_t)(cy2(j) + 1) << 20;
    L.c1 = R(6) * w2<R>(i) * R(cx2(i)) * ulid;
    L.c2 = R(0);
    if (rule == RULE2_BODY_N || rule == RULE2_BODY_H) {
      L.c1 = coef[i - 1].x;
      L.c2 = coef[i - 1].y;
    }
    L.b |= head << 22;
    head = 0u;
    links[pos++] = L;
  }
}

// One link of a step: the pulled value goes where the pull reads it, and the momentum exchange f_j + f_i is
// returned. The cell is that place's only reader: the place is solid or outside the grid (cells at the seam of a
// side that is periodic alone are not listed), and a slip row that mirrors a solid's population reads one that
// points out of the grid, which no link writes.
template <class S, class R>
__device__ __forceinline__ R link2(const Link2<R>& L, S* cur) {
  const uint32_t rule = (L.b >> 15) & 7u;
  if (rule == RULE2_PULL) return R(0);
  const R fj = (R)cur[L.a & 0x7fffu], g = (R)cur[L.b & 0x7fffu];
  R v = fj;
  if (rule == RULE2_SLIP || rule == RULE2_SLIP_HERE) v = g;
  if (rule == RULE2_MOVING) v = fj + L.c1;
  if (rule == RULE2_BODY_N) v = L.c1 * fj + L.c2 * g;
  if (rule == RULE2_BODY_H) v = fj / L.c1 + L.c2 * g;
  cur[L.a >> 15] = (S)v;
  return fj + v;
}

// The force on the cell whose links begin with number l, in their order.
template <class R>
__device__ __forceinline__ void cell_force2(const Link2<R>* links, const R* linkT, int l, R& fx, R& fy) {
  const int count = (int)((links[l].b >> 22) & 0xfu);
  fx = fy = R(0);
  if (count == 0) return;
  uint32_t b[Q2 - 1];
  R t[Q2 - 1];
#pragma unroll
  for (int q = 0; q < Q2 - 1; q++) {
    const int e = q < count ? l + q : l;
    b[q] = links[e].b;
    t[q] = linkT[e];
  }
#pragma unroll
  for (int q = 0; q < Q2 - 1; q++) {
    if (q >= count || ((b[q] >> 15) & 7u) < RULE2_BODY_N) continue;
    fx += R((int)((b[q] >> 18) & 3u) - 1) * t[q];
    fy += R((int)((b[q] >> 20) & 3u) - 1) * t[q];
  }
}

// The warp's sum of (x, y): x in the even lanes, y in the odd ones.
__device__ __forceinline__ double warp_sum2(double x, double y, int lane) {
  const double send = (lane & 1) ? x : y;
  double keep = (lane & 1) ? y : x;
  keep += __shfl_xor_sync(0xffffffffu, send, 1);
#pragma unroll
  for (int o = 2; o < 32; o <<= 1) keep += __shfl_xor_sync(0xffffffffu, keep, o);
  return keep;
}

// A coordinate v in [-k, n - 1 + k] of the margin's frame as one of the grid, or -1 outside it.
__device__ __forceinline__ int real_coord2(int v, int n, bool wrapLow, bool wrapHigh) {
  if (v < 0) return wrapLow ? v + n : -1;
  if (v >= n) return wrapHigh ? v - n : -1;
  return v;
}

// Region RX x RY cells, ROWS rows per thread; tiles of (RX - 2 K) x (RY - 2 K) cells. LAST: a run's last launch, of
// several steps.
template <class C, int RX, int RY, int ROWS, bool LIST, bool LAST>
__global__ void __launch_bounds__(RX * RY / ROWS, 1)
    block2d_kernel(const Tunnel2* __restrict__ tunnels, const Block2Tunnel* __restrict__ layout,
                   const unsigned short* __restrict__ tileTunnel, int K, int k, int par, double2* __restrict__ partials,
                   int j0) {
  using S = typename C::S;
  using R = typename C::R;
  extern __shared__ __align__(16) unsigned char smemRaw[];
  __shared__ double sU[kBlockSteps2];
  __shared__ unsigned sStep;
  __shared__ double sWarp[kBlockSteps2][32][2];
  __shared__ int sLinkCount[32];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int b = blockIdx.x;
  const int t = __ldg(&tileTunnel[b]);
  const Tunnel2& T = tunnels[t];
  const int lb = b - layout[t].first;
  const int tyi = lb / layout[t].tilesX, txi = lb - tyi * layout[t].tilesX;
  constexpr int BY = RY / ROWS, cells = RX * RY;
  const int tid = threadIdx.x + RX * threadIdx.y;
  const int W = T.W, H = T.H;
  const int ox = txi * (RX - 2 * K) - K, oy = tyi * (RY - 2 * K) - K;  // the region's corner
  const int vx = ox + (int)threadIdx.x;
  const int rx = real_coord2(vx, W, T.left == X2_PERIODIC, T.right == X2_PERIODIC);
  const int cut = K - k;  // margin cells that k < K steps do not need
  const bool colIn = rx >= 0 && rx < W && (int)threadIdx.x >= cut && (int)threadIdx.x < RX - cut;
  const bool colOwn = (int)threadIdx.x >= K && (int)threadIdx.x < RX - K && vx < W;
  const uint32_t* __restrict__ flags = T.flags;
  typename XTab2<R>::T xt = {};
  if (colIn) xt = ((const typename XTab2<R>::T*)T.xtab)[rx];
  uint32_t fl[ROWS];  // rule words
  int ry[ROWS];
  bool slots = false;
#pragma unroll
  for (int m = 0; m < ROWS; m++) {
    const int r = threadIdx.y + m * BY, vy = oy + r;
    ry[m] = real_coord2(vy, H, T.bottom == Y2_PERIODIC, T.top == Y2_PERIODIC);
    const bool in = colIn && ry[m] >= 0 && ry[m] < H && r >= cut && r < RY - cut;
    fl[m] = CODE2_SOLID;
    if (in) {
      fl[m] = __ldg(&T.code[ry[m] * W + rx]);
      slots = slots || (colOwn && r >= K && r < RY - K && vy < H && (fl[m] & CODE2_SLOT));
    } else {
      ry[m] = -1;
    }
  }
  const Geo2 g{W, H, T.left, T.right, T.bottom, T.top};
  const int forcing = T.forcing, every = partials ? T.forceEvery : 0;
  const R smagC2 = prm<R>(T, P2_SMAGC2), lambda = prm<R>(T, P2_LAMBDA);
  const int parabolic = T.parabolic;
  // The tile's links, cell by cell and direction by direction, in a fixed order: a scan over the block's
  // counts. A listed cell drops its rules; where the list is full they stay with the cell (rules2).
  constexpr int LINKS = kTileLinks2<RX, RY>, WARPS = RX * BY / 32;
  Link2<R>* const links = (Link2<R>*)(smemRaw + 2 * Q2 * cells * sizeof(S));
  R* const linkT = (R*)(links + LINKS);  // each link's momentum exchange in the current step
  int nLinks = 0;
  if constexpr (LIST) {
    int mine[ROWS], sum = 0;
    const bool left = T.left == X2_PERIODIC, bottom = T.bottom == Y2_PERIODIC;
    const int seamX0 = left ? -1 : W - 1, seamY0 = bottom ? -1 : H - 1;
    const bool seamX = left != (T.right == X2_PERIODIC) && (vx == seamX0 || vx == seamX0 + 1);
    const bool seamY = bottom != (T.top == Y2_PERIODIC);
#pragma unroll
    for (int m = 0; m < ROWS; m++) {
      const uint32_t w = fl[m] & CODE2_RULES;
      // only of cells that a step computes: their neighbours are places in the tile
      const int r = threadIdx.y + m * BY, vy = oy + r;
      const bool steps = (int)threadIdx.x > cut && (int)threadIdx.x < RX - 1 - cut && r > cut && r < RY - 1 - cut;
      // With one side of an axis periodic, the margin behind it continues the grid with cells whose own far side is
      // a wall or open: what they would pull from there is a real cell in the tile, no place for a link's value.
      // The cells on both sides of that seam keep their rules.
      const bool seam = seamX || (seamY && (vy == seamY0 || vy == seamY0 + 1));
      mine[m] = !steps || seam || (fl[m] & CODE2_SOLID) ? 0 : __popc((w | w >> 1 | w >> 2) & 0x249249u);
      sum += mine[m];
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if ((tid & 31) >= o) incl += v;
    }
    if ((tid & 31) == 31) sLinkCount[tid >> 5] = incl;
    __syncthreads();
    const int n = (tid & 31) < WARPS ? sLinkCount[tid & 31] : 0;
    int pos = __reduce_add_sync(0xffffffffu, (tid & 31) < (tid >> 5) ? n : 0) + incl - sum;
    nLinks = min(__reduce_add_sync(0xffffffffu, n), LINKS);
#pragma unroll
    for (int m = 0; m < ROWS; m++) {
      if (mine[m] == 0) continue;
      if (pos + mine[m] <= LINKS) {
        const auto* coef = (const typename Vec2T<R>::T*)T.qCoef;
        if (fl[m] & CODE2_SLOT) coef += ((size_t)(__ldg(&flags[ry[m] * W + rx]) >> BIDX2_SHIFT) - 1) * 8;
        const int r = threadIdx.y + m * BY;
        const bool counts = (fl[m] & CODE2_SLOT) && colOwn && r >= K && r < RY - K && oy + r < H;
        write_links2<R, RX, RY>(links, pos, fl[m], r * RX + threadIdx.x, counts ? mine[m] : 0, prm<R>(T, P2_ULID), coef);
        fl[m] &= CODE2_INLET | CODE2_OUTLET;
      } else {
        for (int q = pos; q < LINKS; q++) links[q].b = RULE2_PULL << 15;
      }
      pos += mine[m];
    }
  }
  DevState2* st = T.st;
  // what the launch before wrote: populations, step counter and inlet speed
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (tid == 0) {
    const unsigned step = __ldcg(&st->step[par]);
    const double u0 = __ldcg(&st->uIn[par]);
    sStep = step;
    for (int j = 0; j <= k; j++) {
      const double u = T.rampKind != 0 && j > 0
                           ? ramp_speed2(T.rampKind, T.rampTarget, T.rampSteps, T.rampEvery, step + (unsigned)j)
                           : u0;
      if (j < k)
        sU[j] = u;
      else if (lb == 0) {
        // the counter and inlet speed after the k steps (slot par ^ 1; this launch reads slot par)
        st->step[par ^ 1] = step + (unsigned)k;
        st->uIn[par ^ 1] = u;
      }
    }
  }
  S* const buf = (S*)smemRaw;
  const int N = W * H;  // 9 N < 2^31: checked when the tunnel is created
  const S* __restrict__ src = (const S*)T.f[par];
  S* __restrict__ dst = (S*)T.f[par ^ 1];
  // A slip row may mirror a solid's populations. No step writes them, and the two buffers differ where the cell
  // became solid between steps: the steps find them in turn, as step by step. (Through L2: this launch writes that
  // buffer's other cells.)
  auto solid_half = [&](int m, int c, int idx) {
    if (!(fl[m] & CODE2_SOLID) || (ry[m] != 0 && ry[m] != H - 1)) return;
#pragma unroll
    for (int i = 0; i < Q2; i++) buf[(Q2 + i) * cells + c] = __ldcg((const S*)T.f[par ^ 1] + (i * N + idx));
  };
#pragma unroll
  for (int m = 0; m < ROWS; m++) {
    if (ry[m] < 0) continue;
    const int c = (threadIdx.y + m * BY) * RX + threadIdx.x, idx = ry[m] * W + rx;
    S v[Q2];
#pragma unroll
    for (int i = 0; i < Q2; i++) v[i] = C::ld(src + (i * N + idx));
#pragma unroll
    for (int i = 0; i < Q2; i++) buf[i * cells + c] = v[i];
    if constexpr (!LIST) solid_half(m, c, idx);
  }
  if constexpr (LIST) {  // after all rows' loads are out: 700x180 2.66 -> 2.62 us a step (without a list 4% slower)
#pragma unroll
    for (int m = 0; m < ROWS; m++)
      if (ry[m] >= 0) solid_half(m, (threadIdx.y + m * BY) * RX + threadIdx.x, ry[m] * W + rx);
  }
  // whether the tile has cells with a force, and whether some of them are not in the list
  bool unlisted = false;
#pragma unroll
  for (int m = 0; m < ROWS; m++) unlisted = unlisted || (!(fl[m] & CODE2_SOLID) && (fl[m] & CODE2_SLOT));
  slots = __syncthreads_or(slots ? 1 : 0) != 0;
  unlisted = LIST ? __syncthreads_or(unlisted ? 1 : 0) != 0 : slots;
  for (int j = 0; j < k; j++) {
    S* cur = buf + (j & 1) * (Q2 * cells);
    S* nxt = buf + ((j + 1) & 1) * (Q2 * cells);
    const int lo = cut + j + 1;  // the margin that is still exact after this step begins here
    const bool colOn = (int)threadIdx.x >= lo && (int)threadIdx.x < RX - lo;
    const R u = (R)sU[j];
    auto sampled = [&]() { return slots && every > 0 && (sStep + (unsigned)j + 1u) % (unsigned)every == 0u; };
    if (LIST && nLinks > 0) {
      for (int l = tid; l < nLinks; l += RX * BY) linkT[l] = link2<S, R>(links[l], cur);
      __syncthreads();
    }
    const bool listed = LIST && sampled();  // without a list it is asked late, for want of registers
    if (listed) {
      double v = 0.0;
      if ((tid & ~31) < nLinks) {
        double ax = 0.0, ay = 0.0;
        for (int l = tid; l < nLinks; l += RX * BY) {
          R lx, ly;
          cell_force2<R>(links, linkT, l, lx, ly);
          ax += (double)lx;
          ay += (double)ly;
        }
        v = warp_sum2(ax, ay, tid & 31);
      }
      if ((tid & 31) < 2) sWarp[j][tid >> 5][tid & 31] = v;
    }
    double fx = 0.0, fy = 0.0;
#pragma unroll
    for (int m = 0; m < ROWS; m++) {
      const int r = threadIdx.y + m * BY;
      if (!colOn || r < lo || r >= RY - lo || (fl[m] & CODE2_SOLID)) continue;
      // opaque to the compiler in every step: what the boundary rules derive from them would otherwise be
      // hoisted out of the step loop into spilled registers
      uint32_t flag = fl[m];
      int x = rx, y = ry[m];
      asm volatile("" : "+r"(flag), "+r"(x), "+r"(y));
      const S* p = cur + r * RX + threadIdx.x;
      R f[Q2], o[Q2];
#pragma unroll
      for (int i = 0; i < Q2; i++) f[i] = (R)p[i * cells - cy2(i) * RX - cx2(i)];
      const int idx = y * W + x;
      if (flag != 0u) {
        R force[2] = {R(0), R(0)};
        const TileSource2<C, RX, RY> ts{p};
        if (flag & CODE2_GENERAL) {
          boundary2<C>(T, g, ts, flags, u, x, y, (long long)idx, __ldg(&flags[idx]), f, force);
        } else {
          if (flag & CODE2_RULES) {
            const auto* coef = (const typename Vec2T<R>::T*)T.qCoef;
            if (flag & CODE2_SLOT) coef += ((size_t)(__ldg(&flags[idx]) >> BIDX2_SHIFT) - 1) * 8;
            rules2<C>(flag, T, ts, coef, f, force);
          }
          if (flag & (CODE2_INLET | CODE2_OUTLET)) zou_he2<C>(LIST ? parabolic : T.parabolic, H, (flag & CODE2_INLET) != 0u, u, y, f);
        }
        if ((flag & CODE2_SLOT) && colOwn && r >= K && r < RY - K && oy + r < H) {
          fx += (double)force[0];
          fy += (double)force[1];
        }
      }
      if constexpr (kExact2)
        collide2<C>(T, xt, forcing, smagC2, H, u, y, f, [&](int i, R v) { o[i] = v; });
      else
        collide2_lean<R>(T, xt, forcing, smagC2, lambda, H, LIST ? parabolic : T.parabolic, u, y, f, o);
      if (j + 1 < k) {
#pragma unroll
        for (int i = 0; i < Q2; i++) nxt[i * cells + r * RX + threadIdx.x] = (S)o[i];
      } else if (colOwn && r >= K && r < RY - K && oy + r < H) {
#pragma unroll
        for (int i = 0; i < Q2; i++) dst[i * N + idx] = (S)o[i];
      }
    }
    if (LIST ? listed && unlisted : sampled()) {
      const double v = warp_sum2(fx, fy, tid & 31);
      if ((tid & 31) < 2) sWarp[j][tid >> 5][tid & 31] = LIST ? sWarp[j][tid >> 5][tid & 31] + v : v;
    }
    __syncthreads();
  }
  if (every > 0 && tid < k && (sStep + (unsigned)tid + 1u) % (unsigned)every == 0u) {
    double ax = 0.0, ay = 0.0;
    if (slots) {
      for (int w = 0; w < WARPS; w++) {
        ax += sWarp[tid][w][0];
        ay += sWarp[tid][w][1];
      }
    }
    partials[(size_t)(j0 + tid) * gridDim.x + b] = make_double2(ax, ay);
  }
  // The step before the last, still in the half that the last one read. The source buffer should hold it, as after
  // single steps, for the cells that become solid next (flags2_kernel); it holds the k-th before, and other
  // blocks may still read it. Bound by its stores, once a run: 100 steps of 2000x500 1,431 -> 1,437 us, 5 steps of
  // 4000x1000 288 -> 316. A variant of its own, because as a branch it cost the launches that skip it (400x100
  // 2.40 -> 2.45 us a step).
  if constexpr (LAST) {
    const S* cur = buf + ((k - 1) & 1) * (Q2 * cells);
    S* __restrict__ prev = (S*)T.prev;
#pragma unroll
    for (int m = 0; m < ROWS; m++) {
      const int r = threadIdx.y + m * BY;
      if (!colOwn || r < K || r >= RY - K || oy + r >= H) continue;
#pragma unroll
      for (int i = 0; i < Q2; i++) __stcs(&prev[i * N + ry[m] * W + rx], cur[i * cells + r * RX + threadIdx.x]);
    }
  }
}

// After a run of n steps that ended on parity par: one block per tunnel, one warp per sampled step, adds
// up the tiles' partials (strided over the lanes, then shuffles) into the force ring.
__global__ void __launch_bounds__(512) sum_samples2_kernel(const Tunnel2* __restrict__ tunnels,
                                                           const Block2Tunnel* __restrict__ layout,
                                                           const double2* __restrict__ partials, int tiles, int n,
                                                           int par) {
  const Tunnel2& T = tunnels[blockIdx.x];
  const unsigned every = (unsigned)T.forceEvery;
  if (every == 0u) return;
  const Block2Tunnel L = layout[blockIdx.x];
  DevState2* st = T.st;
  const unsigned end = st->step[par], step0 = end - (unsigned)n, base = st->sample;
  for (int j = threadIdx.x >> 5; j < n; j += blockDim.x >> 5) {
    const unsigned label = step0 + (unsigned)j + 1u;
    if (label % every != 0u) continue;
    double ax = 0.0, ay = 0.0;
    for (int q = threadIdx.x & 31; q < L.tiles; q += 32) {
      const double2 v = partials[(size_t)j * tiles + L.first + q];
      ax += v.x;
      ay += v.y;
    }
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
      ax += __shfl_down_sync(0xffffffffu, ax, s);
      ay += __shfl_down_sync(0xffffffffu, ay, s);
    }
    if ((threadIdx.x & 31) == 0) {
      T.history[(base + label / every - step0 / every - 1u) % HISTORY2_LEN] = make_double2(ax, ay);
      if (!isfinite(ax) || !isfinite(ay)) atomicOr(&st->status, 1u);
    }
  }
  __syncthreads();  // every warp has read the counter
  if (threadIdx.x == 0) st->sample = base + end / every - step0 / every;
}

template <class C>
static cudaError_t launch_block2_t(const Block2Launch& a, cudaStream_t s) {
  using Kernel = void (*)(const Tunnel2*, const Block2Tunnel*, const unsigned short*, int, int, int, double2*, int);
  Kernel fn = nullptr;
  const int shape = a.regionX * 1000 + a.regionY * 10 + a.rows;
  const bool last = a.last && a.k > 1;
#define SHAPE2(RX, RY, ROWS, LIST) \
  (last ? block2d_kernel<C, RX, RY, ROWS, LIST, true> : block2d_kernel<C, RX, RY, ROWS, LIST, false>)
  if constexpr (sizeof(typename C::R) == 4) {
    switch (shape) {
      case 32241: fn = SHAPE2(32, 24, 1, true); break;
      case 32321: fn = SHAPE2(32, 32, 1, true); break;
      case 64322: fn = SHAPE2(64, 32, 2, true); break;
      case 64483: fn = a.list ? SHAPE2(64, 48, 3, true) : SHAPE2(64, 48, 3, false); break;
    }
  } else {
    switch (shape) {
      case 32242: fn = SHAPE2(32, 24, 2, true); break;
      case 32322: fn = a.list ? SHAPE2(32, 32, 2, true) : SHAPE2(32, 32, 2, false); break;
    }
  }
#undef SHAPE2
  if (!fn) return cudaErrorInvalidValue;
  const size_t links = !a.list ? 0 : (size_t)a.regionX * a.regionY >= 3072 ? kTileLinks2<64, 48> : kTileLinks2<32, 32>;
  const size_t smem = 2 * Q2 * sizeof(typename C::S) * (size_t)a.regionX * a.regionY +
                      links * (sizeof(Link2<typename C::R>) + sizeof(typename C::R));
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(a.nTiles);
  cfg.blockDim = dim3(a.regionX, a.regionY / a.rows);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = a.first ? 0 : 1;  // a run's first launch waits for everything before it: the tables are read early
  return cudaLaunchKernelEx(&cfg, fn, a.tunnels, a.layout, a.tileTunnel, a.K, a.k, a.par, a.partials, a.j0);
}

cudaError_t launch_block2(int precision, const Block2Launch& a, cudaStream_t s) {
  // Populations through L2: a launch is resident while the one before it still writes them, which the read-only
  // path does not allow for; a block reads each once.
  if (precision == 0) return launch_block2_t<Store2F32P>(a, s);
  if (precision == 3) return launch_block2_t<Store2F64P>(a, s);
  return cudaErrorInvalidValue;
}

cudaError_t launch_sum_samples2(const Tunnel2* tunnels, const Block2Tunnel* layout, int nTunnels, const double2* partials,
                                int tiles, int n, int par, cudaStream_t s) {
  sum_samples2_kernel<<<nTunnels, 512, 0, s>>>(tunnels, layout, partials, tiles, n, par);
  return cudaGetLastError();
}

}  // namespace CELLS_NS
}  // namespace cells
