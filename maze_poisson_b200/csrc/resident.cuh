// Field solves whose vectors stay on the SMs between iterations (see resident.cu).
#pragma once

#include "engine.cuh"

namespace mzb {

// Bytes of the work area `EngineArgs::halo` must hold for grids of n points per side, 0 when
// the resident kernels do not serve that size.
size_t resident_halo_bytes(int n);

// Launch a CG program (PROG_CG, PROG_PCG with Jacobi, PROG_INIT_FIELD, PROG_LCG_UPDATE,
// PROG_MAZE_LCG with the implicit or Jacobi preconditioner; the Laplacian or the
// Poisson-Boltzmann operator) on the resident kernel; false when the size, the program or
// the device does not allow it, or without a work area.
bool resident_cg_launch(const EngineArgs& a, cudaStream_t stream);

// Launch PROG_MG_UPDATE or PROG_MAZE_MG (either operator) on the resident multigrid kernel;
// false when the grid is not a multiple of 4, too large, or has no work area.
bool resident_mg_launch(const EngineArgs& a, cudaStream_t stream);

}  // namespace mzb
