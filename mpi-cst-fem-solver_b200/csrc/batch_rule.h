// Which of the two batch kernels (batch.cu) a batch runs on. Host code only.
#pragma once

#include <cmath>

namespace cstg {

// clusters: how many the device takes at a time of k_batch_pcg and of k_batch_halo. The first runs every batch
// (and what the second leaves), so only it is a must.
inline bool batch_shape_runs(const int (&clusters)[2]) { return clusters[0] >= 1; }

// k_batch_halo, when p of the largest plate fits its blocks' shared memory (`smem` bytes each) for R load cases, by
// a halo of a few rows of nodes (a plate that then does not fit is left to k_batch_pcg).
inline bool batch_halo_runs(const int (&clusters)[2], int largest, int cluster, int R, unsigned smem) {
  const double own = std::ceil((double)largest / cluster), nodes = own + 3.0 * std::sqrt((double)largest) + 64.0;
  return clusters[1] >= 1 && nodes * (16.0 * R + 4.0) + 4096.0 <= (double)smem;
}

}  // namespace cstg
