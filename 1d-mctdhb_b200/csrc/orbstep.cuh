// orbstep.cuh -- the orbital side of one MCTDHB step of one system by one
// cluster of thread blocks (orbstep.cu): Runge-Kutta step of the orbital
// equation, Gram-Schmidt, h_kl, g_ksql and the pair matrix, for 2..8 orbitals
// on up to 4096 grid points.  The batched engine runs one cluster per slot,
// the single-system solver one cluster (solver.cu).
#pragma once
#include "batch.h"

namespace mctdhb {

// parts of a step (orb_step_kernel), in execution order
constexpr int kOrbPeriodic = 1;   // f[G-1] = f[0] first (periodic grids)
constexpr int kOrbRk = 2;         // orbitals advanced (Runge-Kutta; split: its nonlinear part)
constexpr int kOrbHalf = 4;       // split: the linear half steps around it as well
constexpr int kOrbGs = 8;         // Gram-Schmidt in imaginary time
constexpr int kOrbPost = 16;      // periodic copy again, overlap residual in real time
constexpr int kOrbMatrices = 32;  // h, g, the pair matrix, Lanczos set-up
constexpr int kOrbStep = 63;

// A cluster of `blocks` per slot of the list: 1, 2, 4 or 8, on which the results
// do not depend, or 0 for eight by code made for eight; mon: the count block's monitor flags, cleared by the first block
// (nullptr: none)
int orb_step_launch(const BatchSlot* slots, const int* list, const int* nlist, int nslots,
                    int parts, int* mon, int blocks, cudaStream_t st);
// launch attributes (call before any stream capture) of the batch's instance or
// the single system's (each is seven orbital counts of code to load)
int orb_step_prepare(bool batch);
// clusters that run at a time (cluster_blocks)
int orb_step_waves(int (&at)[kClusterSizes]);
inline bool orb_step_eligible(int M, int G) {
    return M >= kBatchMinOrb && M <= kBatchMaxOrb && G <= kBatchMaxGrid;
}

}  // namespace mctdhb
