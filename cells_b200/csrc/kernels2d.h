// Host-visible declarations of the 2D kernels' launchers (step2d.cu and aux2d.cu).
#pragma once

#include "d2q9.cuh"

namespace cells {

// One step (or, persistent, nSteps steps) of every tunnel of a batch. A tile is one block's cells:
// tileX x (rows tileY) cells of one tunnel, each thread taking rows y and, with rows = 2, y + tileY;
// the tiles of all tunnels are numbered consecutively.
struct Step2Launch {
  const Tunnel2* tunnels;            // device array, one per tunnel
  const unsigned short* tileTunnel;  // device array: the tunnel of each tile
  int nTiles;                        // tiles of all tunnels
  int tileX, tileY;                  // block shape
  int rows;                          // cell rows per thread: 1 or 2
  int par;                           // parity of the first step
  int allowSample;                   // 0: no force sampling (autotuner trials)
  int nSteps;                        // persistent launch: steps per launch
  int gridBlocks;                    // persistent launch: resident blocks
  unsigned* barrier;                 // persistent launch: grid barrier counter (zeroed per launch)
  int* error;                        // persistent launch: set to 1 when a barrier wait ran out
  unsigned barrierExtra;             // persistent launch: arrivals added to every barrier's target
                                     // (0; 1 only to test the time-out path)
};

// k steps of every tunnel of a batch in one launch, tiles in shared memory (block2d.cu). A tile is
// (regionX - 2 K) x (regionY - 2 K) cells of one tunnel; the launch's k steps are odd and at most K.
constexpr int kBlockSteps2 = 7;  // largest K
struct Block2Tunnel {
  int tilesX, tiles, first;  // tiles per row, of the tunnel, and its first in the batch
};
struct Block2Launch {
  const Tunnel2* tunnels;
  const Block2Tunnel* layout;        // device array, one per tunnel
  const unsigned short* tileTunnel;  // device array: the tunnel of each tile
  int nTiles;
  int regionX, regionY, rows;        // region of a block and cell rows per thread
  bool list;                         // the tile's boundary links are collected and go ahead of the cells
  int K, k;
  int par;                           // parity of the first step
  double2* partials;                 // force partials [step of the run][tile]; NULL: no sampling
  int j0;                            // the launch's first step in the run
  bool first;                        // the first launch of a run: it starts after all work before it
  bool last;                         // the last one: it leaves the step before its last in Tunnel2::prev
};

// precision: 0 f32, 3 f64. fast: FMA contraction allowed; exact: every operation rounds as written.
namespace fast {
cudaError_t launch_block2(int precision, const Block2Launch& a, cudaStream_t s);
// The force samples of a run of n steps that ended on parity par, from its partials.
cudaError_t launch_sum_samples2(const Tunnel2* tunnels, const Block2Tunnel* layout, int nTunnels, const double2* partials,
                                int tiles, int n, int par, cudaStream_t s);
cudaError_t launch_step2(int precision, const Step2Launch& a, cudaStream_t s);
cudaError_t launch_step2_persistent(int precision, const Step2Launch& a, cudaStream_t s);
int persistent_blocks2(int precision, int threads);  // resident blocks of the persistent kernel
}
namespace exact {
cudaError_t launch_block2(int precision, const Block2Launch& a, cudaStream_t s);
// The force samples of a run of n steps that ended on parity par, from its partials.
cudaError_t launch_sum_samples2(const Tunnel2* tunnels, const Block2Tunnel* layout, int nTunnels, const double2* partials,
                                int tiles, int n, int par, cudaStream_t s);
cudaError_t launch_step2(int precision, const Step2Launch& a, cudaStream_t s);
cudaError_t launch_step2_persistent(int precision, const Step2Launch& a, cudaStream_t s);
int persistent_blocks2(int precision, int threads);
}

struct AuxLaunch2 {
  int W, H, N;
  int left, right, bottom, top;
  int forcing;
  double fx, fy;
};

// The block kernel's rule words and Bouzidi coefficients (Tunnel2::code, qCoef); cells whose force slot exceeds qCap
// keep the general rules. code NULL: there are none.
struct Rules2 {
  uint32_t* code;
  void* qCoef;
  int qCap;
};
// flagsShader (src/shaders/aux.ts:22-88): flags with force slots from *counter (zeroed first), the rules that follow
// from them, and the refill of uncovered cells from mac.
// A cell that becomes solid keeps the populations of the last step and of the one before it, one in each buffer.
// prev: those of the step before it, where the buffer that should hold them (older: 0 fA, 1 fB) holds an earlier
// step because the last launch took several; else NULL. It is kept in step with the refill of uncovered cells.
cudaError_t launch_flags2(int precision, const AuxLaunch2& a, const float* sdf, uint32_t* flags, void* fA, void* fB,
                          const float4* mac, unsigned* counter, void* prev, int older, const Rules2& rules,
                          cudaStream_t s);
// Cells of a tunnel; x0 and y0 may be -1 and the far ends one beyond the grid: its other side.
struct Box2 {
  int x0, y0, w, h;
};
// The rules of a box's cells from the flags and the SDF, for edits of the SDF that leave the flags.
cudaError_t launch_rules2(int precision, const AuxLaunch2& a, const Box2& box, const float* sdf, const uint32_t* flags,
                          const Rules2& rules, cudaStream_t s);
// initShader (src/shaders/aux.ts:92-111): both buffers to feq(rho, ux, uy) of mac.
cudaError_t launch_init2(int precision, const AuxLaunch2& a, const float4* mac, void* fA, void* fB, cudaStream_t s);
// macroShader (src/shaders/aux.ts:115-140); sets status bit 1 on a non-finite value.
cudaError_t launch_macro2(int precision, const AuxLaunch2& a, const void* f, const uint32_t* flags, float4* mac,
                          DevState2* st, cudaStream_t s);
// sum(rho) over fluid cells in f64, per-block partials then one ordered sum.
cudaError_t launch_mass2(int precision, const AuxLaunch2& a, const void* f, const uint32_t* flags, double* partials,
                         int nPartials, double* out, cudaStream_t s);
// brushShader (src/shaders/aux.ts:177-194) over the box [x0, x0 + w) x [y0, y0 + h).
cudaError_t launch_brush2(float* sdf, int W, int H, float cx, float cy, float r, int erase, int x0, int y0, int w,
                          int h, cudaStream_t s);
// Writes parts of a tunnel's device state: bit 0 both step counters, bit 1 both inlet speeds,
// bit 2 clears the force sample counter, bit 3 clears the status word.
cudaError_t launch_set_state2(DevState2* st, int which, unsigned step, double uIn, cudaStream_t s);

}  // namespace cells
