// Teams of blocks of the persistent Jacobi-PCG (persistent.cu), and what happens when the device cannot place
// one. Host code only.
#pragma once

#include <cuda_runtime_api.h>

namespace cstg {

// From the smallest systems up: one cluster; one block per SM with the matrix in shared memory; one block per SM
// that streams it (by wide or narrow groups of rows); and, for the meshes that none of these holds, all
// vectors in global memory (persistent_grid.cu).
enum class PcgTeam { kFirst = -1, kCluster = 0, kResident, kStream, kStreamNarrow, kGrid, kNone };

// A launch that asks for more blocks at once than the process or stream has SMs for.
inline bool unplaced(cudaError_t e) {
  return e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorInvalidClusterSize ||
         e == cudaErrorLaunchOutOfResources;
}

// Launches on `team`, or on the first team after it that the device can place (kNone: on none of them, nothing
// was launched and the caller's other path takes the solve).
template <class Launch, class Next>
cudaError_t launch_first_team(PcgTeam& team, Launch launch, Next next) {
  while (team != PcgTeam::kNone) {
    const cudaError_t e = launch(team);
    if (!unplaced(e)) return e;
    cudaGetLastError();  // (reported: not the next call's error)
    team = next(team);
  }
  return cudaSuccess;
}

}  // namespace cstg
