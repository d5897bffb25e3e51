// Discrete adjoint of the D3Q19 step (no counterpart in the reference): the recorded forward run
// and the buffers of the backward sweep.
//
// The forward map of one step is f^{n+1} = C(P(f^n)): P pulls every population (a plain copy from
// the upstream node, or at boundaries a combination of one or two source elements: outlet copy,
// bounce-back, slip mirror, Bouzidi interpolation with link fraction q from the SDF), C collides
// each cell (TRT with sponge and absorbing layer; the inlet stores feq(1, u_n); the outlet stores
// feq(1, u)). The objective is J = scale * mean_{n in window} F_c(n), F the momentum-exchange force.
// The backward sweep runs lambda^n = P^T (dC/dg)^T lambda^{n+1} + dJ_n/df^n from lambda^T down to
// lambda^0 over states recomputed segment by segment from checkpoints taken every K steps, and
// accumulates dJ/dq per Bouzidi link (then dJ/dsdf) and dJ/du_n per step (then dJ/du_in).
#pragma once

#include <cstdint>
#include <vector>

#include "kernels3d.h"

// How a link's fraction q depends on the SDF: dq/dsdf at the cell and at the solid node (0 where q is
// clamped). solid < 0: the link's pull does not depend on q.
struct AdjLinkQ3 {
  double dqdF, dqdS;
  int cell, solid;
};

struct Adjoint3D {
  // recorded run
  int64_t s0 = 0;         // step count when the recorded forward run started
  int64_t steps = 0;
  int64_t w0 = 0, w1 = 0;  // objective window (inclusive step labels)
  int K = 100;
  int component = 0;
  double scale = 1.0;
  double objective = 0.0;
  int parity0 = 0;
  uint64_t argGen = 0;     // the handle's argument generation at record time
  int64_t endStep = 0;     // the handle's step after the recorded run
  std::vector<double> uStep;    // inlet speed of each recorded step
  std::vector<double> rampStep; // d u_n / d u_in of each recorded step

  // checkpoints: the populations and device state at the start of every segment
  std::vector<void*> ck;       // into the handle's adjStore
  std::vector<void*> ckState;  // into ckStateBlock
  cells::DevState3* ckStateBlock = nullptr;
  void* endState = nullptr;  // device state after the run (restored after the backward sweep)
  std::vector<void*> seg[2];  // two sets of K recomputed states: the segment being swept and the next

  // link tables (device). A link is a flagged direction of a listed cell: g = a1 f[e1] + a2 f[e2].
  // Force links add cF (f[e1] + g) to the objective's force component, cF = c_{j, component}.
  int nLinks = 0;
  AdjLinkQ3* linkQ = nullptr;
  void* lcF = nullptr;          // R, 0 for a link without force
  void* lq = nullptr;           // R
  signed char* lqk = nullptr;   // 0: g does not depend on q; 1: q < 1/2 with a fluid node behind; 2: q >= 1/2
  void* lamG = nullptr;         // R, the adjoint of each link's pulled value in the current step
  double* dqAcc = nullptr;      // dJ/dq per link, summed over the steps

  // transposed map: elements that a link reads beside other readers, with a coefficient or for a force
  int nRows = 0;
  int* rowElem = nullptr;
  unsigned char* rowSet = nullptr;  // 1: the element has no regular reader (its adjoint is set, not added)
  int* rowStart = nullptr;          // nRows + 1
  int* entLink = nullptr;
  void* entAlpha = nullptr;         // R
  void* rowPhi = nullptr;           // R: sum of cF of the force links whose fj is this element

  // adjoint state
  void* lam[2] = {nullptr, nullptr};  // R, 19 N each
  double* blockPart = nullptr;       // dJ/du_n block sums of a segment's steps: K x nParts
  double* dudn = nullptr;            // dJ/du_n per recorded step
  // device buffers of this run: carved from the handle's adjTab block while it has room (tabUsed
  // bytes taken), else allocated on their own (own, freed with the run); tabNeed is the total
  size_t tabUsed = 0, tabNeed = 0;
  std::vector<void*> own;
  cudaStream_t side2 = nullptr;          // the next segment's recompute, beside the sweep
  cudaEvent_t fork2 = nullptr, join2 = nullptr;
  int* slowCells = nullptr;  // listed flagged fluid cells (device), in index order: all but the face rows'
  int nSlow = 0;
  int* sE1 = nullptr;        // [19][nSlow] pull records of the flagged cells
  int* sE2 = nullptr;
  int* sTgt = nullptr;
  void* sA1 = nullptr;       // R
  void* sA2 = nullptr;       // R
  int nParts = 0;            // block sums of one adjoint step
};

namespace cells {

struct AdjLaunch3 {
  const void* f;         // f^n (storage type == arithmetic type: f32 or f64)
  const void* lamNext;   // lambda^{n+1}
  void* lamOut;          // lambda^n
  const uint32_t* flags;
  const void* xTab;      // per x: omega+, omega-, sigma, 1 / omega+
  const uint8_t* rowBody;
  const void* lcF;
  const void* lq;
  const signed char* lqk;
  void* lamG;
  double* dqAcc;
  double* blockPart;     // the step's dJ/du_n block sums
  double u, w;           // the step's inlet speed, and the objective weight of its force
  long long N;
  int W, H, D;
  int off[cells::Q3];    // cell offset of each direction
  int absorbX0;          // first x of the absorbing layer (W when there is none)
  int nCellBlocks, nSlowBlocks, nFaceBlocks;  // blocks of the roles
  int roleZ;                                  // grid slices of the last two
  int slice0;                                 // first slice of this launch
  int foff[4][cells::Q3];                     // face rows: element offset of direction i's source from the cell
  const int* slowCells;  // the flagged fluid cells, in index order
  int nSlow;
  const int* sE1;        // [19][nSlow]: the source of a one-source pull (coefficient 1), or the first
                         // of two sources with the sign bit set (then sE2, sA1, sA2 apply)
  const int* sE2;
  const int* sTgt;       // [19][nSlow]: element of a plain pull's adjoint, or -(link + 1)
  const void* sA1;       // R: coefficients (a2 = 0 for one source)
  const void* sA2;
  int nParts;            // blockPart entries: nCellBlocks + nSlowBlocks + nFaceBlocks
  // transposed map
  int nRows;
  const int* rowElem;
  const unsigned char* rowSet;
  const int* rowStart;
  const int* entLink;
  const void* entAlpha;
  const void* rowPhi;
};

// What the table kernels read.
struct AdjTables3 {
  const uint32_t* flags;
  const float* sdf;
  const uint8_t* rowBody;
  long long N;
  int W, H, D;
  int component;
  int facePairs;  // the face rows go to the x-pair role
};

constexpr int kAdjThreads = 128;
constexpr int kAdjTileX = 32;
// One adjoint step (precision 0 or 3): the interior and flagged cells in one launch, then the
// boundary-element kernel. The step reads f^n before it waits for the launch before it; first: the step starts
// after all work before it on the stream (the recompute of its segment's states).
cudaError_t launch_adjoint_step3(int precision, const AdjLaunch3& a, bool first, cudaStream_t s);

}  // namespace cells
