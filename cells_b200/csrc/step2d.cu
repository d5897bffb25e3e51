// The D2Q9 step kernel: pull streaming, every boundary rule of the reference's 2D solver, Zou-He
// inlet and outlet, TRT collision with Smagorinsky, absorbing layers and the Guo body force, and
// the momentum-exchange force of the step reduced in f64 — for every tunnel of a batch in one
// launch (src/shaders/step.ts:9-229, src/shaders/common.ts:39-57, src/shaders/aux.ts:143-172).
//
// Each block updates one tile (blockDim.x x blockDim.y cells) of one tunnel; the tiles of all
// tunnels of a batch form one grid, so tunnels of different sizes advance in the same launch. A
// cell whose flag word is 0 pulls its 9 populations straight from the neighbours; any other cell
// resolves each direction with the reference's pullSlow rules. The arithmetic follows the
// reference's expressions operation by operation; the exact build (-fmad=false) reproduces the
// oracle's bits.
//
// Force: every tile of a sampled step writes the f64 sum of its cells' forces to its partial slot;
// the tunnel's last tile to finish (an atomic count) sums the partials in slot order into the
// history ring. The reference sums f32 slots in atomic order instead (src/shaders/aux.ts:143-172).
//
// This file is compiled twice: into cells::fast (contraction allowed) and, with
// -fmad=false -DCELLS_EXACT_ARITH, into cells::exact.
#include "step2d.cuh"

namespace cells {
namespace CELLS_NS {

// The fields of a tunnel that every cell of a tile reads, loaded once per thread.
template <class C>
struct Hot2 {
  const typename C::S* __restrict__ src;
  typename C::S* __restrict__ dst;
  const uint32_t* __restrict__ flags;
  const typename XTab2<typename C::R>::T* __restrict__ xtab;
  int W, H, N;
  int forcing;
  typename C::R smagC2;
};

// The loads of the cell (x, y): its flag word and the fast path's nine pulls, issued together (one
// memory round trip per cell, not two); a flagged cell replaces the pulls in cell2. Every address is
// inside the allocation: the largest, direction 8 on the top row, is at most W - 1 elements past the
// nine arrays, which the host pads.
template <class C>
__device__ __forceinline__ uint32_t load2(const Hot2<C>& h, int x, int y, typename C::R (&f)[Q2]) {
  using R = typename C::R;
  const int idx = y * h.W + x;
#pragma unroll
  for (int i = 0; i < Q2; i++) f[i] = (R)C::ld(h.src + (i * h.N + idx - cy2(i) * h.W - cx2(i)));
  return __ldg(&h.flags[idx]);
}

// main, src/shaders/step.ts:177-227, for the cell (x, y) of tunnel T, whose loads load2 made.
// Returns whether the cell has a force slot (its force is then in force[0..1]).
template <class C>
__device__ __forceinline__ bool cell2(const Tunnel2& T, const Hot2<C>& h, typename C::R uIn, int x, int y,
                                      uint32_t fl, typename C::R (&f)[Q2], typename C::R force[2]) {
  using R = typename C::R;
  using S = typename C::S;
  const int N = h.N;  // 9 N < 2^31: checked when the tunnel is created
  S* __restrict__ dst = h.dst;
  const int idx = y * h.W + x;
  bool slot = false;
  if (fl != 0u) {
    if (fl & FLAG2_SOLID) return false;
    const Geo2 g{h.W, h.H, T.left, T.right, T.bottom, T.top};
    const GridSource2<C> src{h.src, (long long)N, h.W};
    slot = boundary2<C>(T, g, src, h.flags, uIn, x, y, (long long)idx, fl, f, force);
  }
  // f32 stores each population as it is known, for want of registers, f64 all of them at the end: us per step of
  // 4000x1000 f32 68.8 and 71.0, f64 187 and 156.
  if constexpr (sizeof(R) == 4) {
    collide2<C>(T, h.xtab[x], h.forcing, h.smagC2, h.H, uIn, y, f, [&](int i, R v) { dst[i * N + idx] = (S)v; });
  } else {
    R o[Q2];
    const auto xt = h.xtab[x];  // read-only for the whole launch
    collide2<C>(T, xt, h.forcing, h.smagC2, h.H, uIn, y, f, [&](int i, R v) { o[i] = v; });
#pragma unroll
    for (int i = 0; i < Q2; i++) dst[i * N + idx] = (S)o[i];
  }
  return slot;
}

// One tile (lb-th of its tunnel t) of the step of parity par.
template <class C, int ROWS>
__device__ __forceinline__ void tile2(const Tunnel2* __restrict__ tunnels, int t, int lb, int par, int allowSample) {
  using R = typename C::R;
  const Tunnel2& T = tunnels[t];
  __shared__ double2 warpSum[32];
  __shared__ int lastTile;
  const int tid = threadIdx.x + blockDim.x * threadIdx.y;
  const int nthreads = blockDim.x * blockDim.y;
  const int tilesX = T.tilesX;
  const int tyi = lb / tilesX;
  const int txi = lb - tyi * tilesX;
  const int x = txi * blockDim.x + threadIdx.x;
  const int y = tyi * (ROWS * blockDim.y) + threadIdx.y;  // this thread's rows: y (+ blockDim.y)
  DevState2* st = T.st;
  const unsigned step = __ldcg(&st->step[par]);
  const double uInD = __ldcg(&st->uIn[par]);
  const int every = T.forceEvery;
  const bool sample = allowSample && every > 0 && ((step + 1u) % (unsigned)every) == 0u;
  if (lb == 0 && tid == 0) {
    // the next step's counter and inlet speed (slot par^1; this step reads slot par only)
    st->step[par ^ 1] = step + 1u;
    st->uIn[par ^ 1] = T.rampKind != 0 ? ramp_speed2(T.rampKind, T.rampTarget, T.rampSteps, T.rampEvery, step + 1u)
                                       : uInD;
  }
  // each cell's force stays in its own accumulator and is widened to f64 before the two are added,
  // as every cell's force enters the f64 tile sum on its own
  R force[2] = {R(0), R(0)}, force1[2] = {R(0), R(0)};
  bool slot = false, slot1 = false;
  if (x < T.W && y < T.H) {
    Hot2<C> h;
    h.W = T.W;
    h.H = T.H;
    h.N = h.W * h.H;
    h.src = (const typename C::S*)T.f[par];
    h.dst = (typename C::S*)T.f[par ^ 1];
    h.flags = T.flags;
    h.xtab = (const typename XTab2<R>::T*)T.xtab;
    h.forcing = T.forcing;
    h.smagC2 = prm<R>(T, P2_SMAGC2);
    R f0[Q2];
    const uint32_t fl0 = load2<C>(h, x, y, f0);
    if constexpr (ROWS == 2) {
      // both rows' loads go out before either cell computes
      const int y1 = y + blockDim.y;
      const bool second = y1 < h.H;
      R f1[Q2];
      uint32_t fl1 = 0u;
      if (second) fl1 = load2<C>(h, x, y1, f1);
      slot = cell2<C>(T, h, (R)uInD, x, y, fl0, f0, force);
      if (second) slot1 = cell2<C>(T, h, (R)uInD, x, y1, fl1, f1, force1);
    } else {
      slot = cell2<C>(T, h, (R)uInD, x, y, fl0, f0, force);
    }
  }
  if (!sample) return;
  // f64 sum of the tile's forces: warp shuffles, then warps in order
  if (__syncthreads_or((slot || slot1) ? 1 : 0)) {
    double sx = slot ? (double)force[0] : 0.0, sy = slot ? (double)force[1] : 0.0;
    if (slot1) {
      sx += (double)force1[0];
      sy += (double)force1[1];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sx += __shfl_down_sync(0xffffffffu, sx, o);
      sy += __shfl_down_sync(0xffffffffu, sy, o);
    }
    if ((tid & 31) == 0) warpSum[tid >> 5] = make_double2(sx, sy);
    __syncthreads();
    if (tid == 0) {
      double ax = 0.0, ay = 0.0;
      for (int w = 0; w < (nthreads + 31) / 32; w++) {
        ax += warpSum[w].x;
        ay += warpSum[w].y;
      }
      T.partials[lb] = make_double2(ax, ay);
    }
  } else if (tid == 0) {
    T.partials[lb] = make_double2(0.0, 0.0);
  }
  if (tid == 0) {
    __threadfence();
    const unsigned prev = atomicAdd(&st->done, 1u);
    lastTile = prev == (unsigned)(T.nTiles - 1);
  }
  __syncthreads();
  if (!lastTile) return;
  // the tunnel's last tile: partials in slot order, strided per thread, then threads in order
  __threadfence();
  double ax = 0.0, ay = 0.0;
  for (int k = tid; k < T.nTiles; k += nthreads) {
    const double2 v = __ldcg(&T.partials[k]);
    ax += v.x;
    ay += v.y;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ax += __shfl_down_sync(0xffffffffu, ax, o);
    ay += __shfl_down_sync(0xffffffffu, ay, o);
  }
  __syncthreads();
  if ((tid & 31) == 0) warpSum[tid >> 5] = make_double2(ax, ay);
  __syncthreads();
  if (tid == 0) {
    double bx = 0.0, by = 0.0;
    for (int w = 0; w < (nthreads + 31) / 32; w++) {
      bx += warpSum[w].x;
      by += warpSum[w].y;
    }
    const unsigned s = __ldcg(&st->sample);
    T.history[s % HISTORY2_LEN] = make_double2(bx, by);
    st->sample = s + 1u;
    st->done = 0u;
    if (!isfinite(bx) || !isfinite(by)) atomicOr(&st->status, 1u);
  }
}

// Register cap of the f32 kernel (blocks of 256 threads per SM it must fit): 3 (up to 85
// registers); measured against 4 (64 registers, a few spilled words) the batch is as fast and one
// tunnel at a time 3% faster, while 5 and 6 (51 and 42 registers) spill and lose 12-28%. The f64
// kernel keeps its registers.
template <class C>
constexpr int min_blocks2() {
  return sizeof(typename C::R) == 4 ? 3 : 1;
}

template <class C, int ROWS>
__global__ void __launch_bounds__(256, min_blocks2<C>()) step2d_kernel(const Tunnel2* __restrict__ tunnels,
                                                     const unsigned short* __restrict__ tileTunnel, int par,
                                                     int allowSample) {
  // programmatic dependent launch, as in the 3D step: the next step's grid is scheduled during
  // this one's tail and waits here for the previous grid to complete
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int b = blockIdx.x;
  const int t = __ldg(&tileTunnel[b]);
  tile2<C, ROWS>(tunnels, t, b - __ldg(&tunnels[t].firstTile), par, allowSample);
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Grid-wide barrier of the persistent kernel: arrivals count up a counter that the host zeroes
// before each launch; barrier k of the launch waits for k * gridDim.x arrivals. The wait is
// bounded by one second of the global timer and, as a backstop, by 2^23 polls; on time-out the
// block sets *error and the kernel winds down (every other block's wait then ends at its next
// poll).
__device__ __forceinline__ bool grid_barrier2(unsigned* counter, unsigned target, int* error) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0 && threadIdx.y == 0) {
    ok = 1;
    __threadfence();
    atomicAdd(counter, 1u);
    long long spins = 0;
    const unsigned long long t0 = global_ns();
    while (true) {
      unsigned seen;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(counter) : "memory");
      if (seen >= target) break;
      if (*(volatile int*)error != 0 || ++spins > (1ll << 23) || global_ns() - t0 > 1000000000ull) {
        atomicExch(error, 1);
        ok = 0;
        break;
      }
      __nanosleep(100);
    }
    __threadfence();
  }
  __syncthreads();
  return ok != 0;
}

// nSteps steps of every tunnel in one launch: each resident block walks the tiles with a grid
// stride, then all blocks meet at the barrier before the next step.
template <class C, int ROWS>
__global__ void __launch_bounds__(256, min_blocks2<C>()) step2d_persistent_kernel(const Tunnel2* __restrict__ tunnels,
                                                                const unsigned short* __restrict__ tileTunnel,
                                                                int nTiles, int par, int nSteps, int allowSample,
                                                                unsigned* barrier, int* error, unsigned extra) {
  for (int s = 0; s < nSteps; s++) {
    for (int b = blockIdx.x; b < nTiles; b += gridDim.x) {
      const int t = __ldg(&tileTunnel[b]);
      tile2<C, ROWS>(tunnels, t, b - __ldg(&tunnels[t].firstTile), par, allowSample);
      __syncthreads();
    }
    par ^= 1;
    if (s + 1 < nSteps && !grid_barrier2(barrier, (unsigned)(s + 1) * gridDim.x + extra, error)) return;
  }
}

template <class C>
static cudaError_t launch_step2_t(const Step2Launch& a, cudaStream_t s) {
  if (a.nTiles <= 0) return cudaSuccess;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(a.nTiles);
  cfg.blockDim = dim3(a.tileX, a.tileY);
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, a.rows == 2 ? step2d_kernel<C, 2> : step2d_kernel<C, 1>, a.tunnels, a.tileTunnel,
                            a.par, a.allowSample);
}

template <class C>
static cudaError_t launch_step2_persistent_t(const Step2Launch& a, cudaStream_t s) {
  if (a.nTiles <= 0 || a.nSteps <= 0) return cudaSuccess;
  dim3 block(a.tileX, a.tileY);
  const Tunnel2* tunnels = a.tunnels;
  const unsigned short* tileTunnel = a.tileTunnel;
  int nTiles = a.nTiles, par = a.par, nSteps = a.nSteps, allowSample = a.allowSample;
  unsigned* barrier = a.barrier;
  int* error = a.error;
  unsigned extra = a.barrierExtra;
  void* args[] = {&tunnels, &tileTunnel, &nTiles, &par, &nSteps, &allowSample, &barrier, &error, &extra};
  cudaError_t e = cudaMemsetAsync(barrier, 0, sizeof(unsigned), s);
  if (e != cudaSuccess) return e;
  const void* fn = a.rows == 2 ? (const void*)step2d_persistent_kernel<C, 2> : (const void*)step2d_persistent_kernel<C, 1>;
  return cudaLaunchCooperativeKernel(fn, dim3(a.gridBlocks), block, args, 0, s);
}

template <class C>
static int persistent_blocks2_t(int threads) {
  int dev = 0, sms = 0, perSm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  // resident blocks of either rows variant (the smaller, so that both launch cooperatively)
  int perSm2 = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, step2d_persistent_kernel<C, 1>, threads, 0) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm2, step2d_persistent_kernel<C, 2>, threads, 0) != cudaSuccess)
    return 0;
  if (perSm2 < perSm) perSm = perSm2;
  return perSm * sms;
}

cudaError_t launch_step2(int precision, const Step2Launch& a, cudaStream_t s) {
  if (precision == 0) return launch_step2_t<Store2F32>(a, s);
  if (precision == 3) return launch_step2_t<Store2F64>(a, s);
  return cudaErrorInvalidValue;
}

cudaError_t launch_step2_persistent(int precision, const Step2Launch& a, cudaStream_t s) {
  if (precision == 0) return launch_step2_persistent_t<Store2F32P>(a, s);
  if (precision == 3) return launch_step2_persistent_t<Store2F64P>(a, s);
  return cudaErrorInvalidValue;
}

int persistent_blocks2(int precision, int threads) {
  if (precision == 0) return persistent_blocks2_t<Store2F32P>(threads);
  if (precision == 3) return persistent_blocks2_t<Store2F64P>(threads);
  return 0;
}

}  // namespace CELLS_NS
}  // namespace cells
