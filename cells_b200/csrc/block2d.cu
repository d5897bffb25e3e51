// Several D2Q9 time steps in one launch: a block loads a tile of one tunnel with a margin of k cells on
// every side into shared memory, steps it k times while the margin shrinks by one cell a step, and
// stores the tile. The margins of neighbouring tiles are computed twice instead of exchanged, so a
// launch needs no communication, and a step costs a block barrier instead of a launch and the
// round trips of its loads.
//
// Boundary rules read within one cell of their own, so they need nothing beyond the margin; a periodic
// seam is a margin loaded from the other side. What a flagged direction pulls is resolved per cell into
// a rule word and Bouzidi coefficients when the SDF is set (rules2_kernel), because evaluating the
// general rules -- eight directions with dependent flag and SDF loads -- took most of a step: 400x100
// cylinder 5.0 us a step with them. The arithmetic is the one-step kernel's (step2d.cuh); k is odd, so
// a launch ends in the other population buffer as a single step does.
//
// Force: a tile's owned cells sum in f64 per sampled step (warp shuffles, then the warps in order) into
// one partial per step and tile; after the launches of a run sum_samples2_kernel adds the tiles up in
// order into the ring.
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
  __device__ __forceinline__ typename C::R at(int pop, int, int, int dx, int dy) const {
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
      f[i] = src.at(mirror_y2(i), 0, 0, rule == RULE2_SLIP ? -cx2(i) : 0, 0);
      continue;
    }
    const R fj = src.at(j, 0, 0, 0, 0);
    R fi = fj;
    if (rule == RULE2_MOVING) {
      f[i] = fj + R(6) * w2<R>(i) * R(cx2(i)) * prm<R>(T, P2_ULID);
      continue;
    }
    if (rule >= RULE2_BODY_N) {
      if (rule != RULE2_BODY_0) {
        const auto c = coef[i - 1];
        if (rule == RULE2_BODY_N)
          fi = c.x * fj + c.y * src.at(j, 0, 0, cx2(i), cy2(i));
        else
          fi = fj / c.x + c.y * src.at(i, 0, 0, 0, 0);
      }
      const R t = fj + fi;
      force[0] += R(cx2(j)) * t;
      force[1] += R(cy2(j)) * t;
    }
    f[i] = fi;
  }
}

// A coordinate v in [-k, n - 1 + k] of the margin's frame as one of the grid, or -1 outside it.
__device__ __forceinline__ int real_coord2(int v, int n, bool wrapLow, bool wrapHigh) {
  if (v < 0) return wrapLow ? v + n : -1;
  if (v >= n) return wrapHigh ? v - n : -1;
  return v;
}

// Region RX x RY cells, ROWS rows per thread; tiles of (RX - 2 K) x (RY - 2 K) cells.
template <class C, int RX, int RY, int ROWS>
__global__ void __launch_bounds__(RX * RY / ROWS, 1)
    block2d_kernel(const Tunnel2* __restrict__ tunnels, const Block2Tunnel* __restrict__ layout,
                   const unsigned short* __restrict__ tileTunnel, int K, int k, int par, double2* __restrict__ partials,
                   int j0) {
  using S = typename C::S;
  using R = typename C::R;
  extern __shared__ __align__(16) unsigned char smemRaw[];
  __shared__ double sU[kBlockSteps2];
  __shared__ unsigned sStep;
  __shared__ double2 sWarp[kBlockSteps2][32];
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
#pragma unroll
  for (int m = 0; m < ROWS; m++) {
    if (ry[m] < 0) continue;
    const int c = (threadIdx.y + m * BY) * RX + threadIdx.x, idx = ry[m] * W + rx;
    S v[Q2];
#pragma unroll
    for (int i = 0; i < Q2; i++) v[i] = C::ld(src + (i * N + idx));
#pragma unroll
    for (int i = 0; i < Q2; i++) buf[i * cells + c] = v[i];
    if (fl[m] & CODE2_SOLID) {  // a slip row may mirror a solid's populations: they are in both halves
#pragma unroll
      for (int i = 0; i < Q2; i++) buf[(Q2 + i) * cells + c] = v[i];
    }
  }
  slots = __syncthreads_or(slots ? 1 : 0) != 0;
  for (int j = 0; j < k; j++) {
    const S* cur = buf + (j & 1) * (Q2 * cells);
    S* nxt = buf + ((j + 1) & 1) * (Q2 * cells);
    const int lo = cut + j + 1;  // the margin that is still exact after this step begins here
    const bool colOn = (int)threadIdx.x >= lo && (int)threadIdx.x < RX - lo;
    const R u = (R)sU[j];
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
          if (flag & (CODE2_INLET | CODE2_OUTLET)) zou_he2<C>(T, H, (flag & CODE2_INLET) != 0u, u, y, f);
        }
        if ((flag & CODE2_SLOT) && colOwn && r >= K && r < RY - K && oy + r < H) {
          fx += (double)force[0];
          fy += (double)force[1];
        }
      }
      if constexpr (kExact2)
        collide2<C>(T, xt, forcing, smagC2, H, u, y, f, o);
      else
        collide2_lean<R>(T, xt, forcing, smagC2, lambda, H, u, y, f, o);
      if (j + 1 < k) {
#pragma unroll
        for (int i = 0; i < Q2; i++) nxt[i * cells + r * RX + threadIdx.x] = (S)o[i];
      } else if (colOwn && r >= K && r < RY - K && oy + r < H) {
#pragma unroll
        for (int i = 0; i < Q2; i++) dst[i * N + idx] = (S)o[i];
      }
    }
    if (slots && every > 0 && (sStep + (unsigned)j + 1u) % (unsigned)every == 0u) {
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) {
        fx += __shfl_down_sync(0xffffffffu, fx, s);
        fy += __shfl_down_sync(0xffffffffu, fy, s);
      }
      if ((tid & 31) == 0) sWarp[j][tid >> 5] = make_double2(fx, fy);
    }
    __syncthreads();
  }
  if (every > 0 && tid < k && (sStep + (unsigned)tid + 1u) % (unsigned)every == 0u) {
    double ax = 0.0, ay = 0.0;
    if (slots) {
      for (int w = 0; w < RX * BY / 32; w++) {
        ax += sWarp[tid][w].x;
        ay += sWarp[tid][w].y;
      }
    }
    partials[(size_t)(j0 + tid) * gridDim.x + b] = make_double2(ax, ay);
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
  if constexpr (sizeof(typename C::R) == 4) {
    switch (shape) {
      case 32281: fn = block2d_kernel<C, 32, 28, 1>; break;
      case 32321: fn = block2d_kernel<C, 32, 32, 1>; break;
      case 64322: fn = block2d_kernel<C, 64, 32, 2>; break;
      case 64483: fn = block2d_kernel<C, 64, 48, 3>; break;
    }
  } else {
    switch (shape) {
      case 32242: fn = block2d_kernel<C, 32, 24, 2>; break;
      case 32322: fn = block2d_kernel<C, 32, 32, 2>; break;
    }
  }
  if (!fn) return cudaErrorInvalidValue;
  const size_t smem = 2 * Q2 * sizeof(typename C::S) * (size_t)a.regionX * a.regionY;
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
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, fn, a.tunnels, a.layout, a.tileTunnel, a.K, a.k, a.par, a.partials, a.j0);
}

cudaError_t launch_block2(int precision, const Block2Launch& a, cudaStream_t s) {
  if (precision == 0) return launch_block2_t<Store2F32>(a, s);
  if (precision == 3) return launch_block2_t<Store2F64>(a, s);
  return cudaErrorInvalidValue;
}

cudaError_t launch_sum_samples2(const Tunnel2* tunnels, const Block2Tunnel* layout, int nTunnels, const double2* partials,
                                int tiles, int n, int par, cudaStream_t s) {
  sum_samples2_kernel<<<nTunnels, 512, 0, s>>>(tunnels, layout, partials, tiles, n, par);
  return cudaGetLastError();
}

}  // namespace CELLS_NS
}  // namespace cells
