// Launch of a kernel whose blocks wait for one another (host code).
#pragma once

#include <cuda_runtime_api.h>

#include <algorithm>

namespace tea {

// launch(blocks) makes a cooperative launch and returns its error.  The loops
// ask for a block per SM; a process that may use only part of the SMs has no
// room for that many at once, and the launch is refused before anything runs.
// Any smaller grid gives the same results (a block takes supertiles b, b +
// grid, ...), so it is tried an eighth smaller until it fits.
template <class Launch>
cudaError_t launch_resident(int blocks, Launch launch) {
  cudaError_t e = launch(blocks);
  while (e == cudaErrorCooperativeLaunchTooLarge && blocks > 1) {
    cudaGetLastError();  // not to be found by a later check
    blocks -= std::max(1, blocks / 8);
    e = launch(blocks);
  }
  return e;
}

}  // namespace tea
