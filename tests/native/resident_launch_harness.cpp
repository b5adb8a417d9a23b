// tea_resident_launch.h on the host, with a launch that is too large above a
// given number of blocks.
#include "tea_resident_launch.h"

static int g_cleared;
extern "C" cudaError_t cudaGetLastError(void) {
  g_cleared++;
  return cudaSuccess;
}

// Tries launch_resident from `blocks`; writes the grids tried to tried[0..),
// returns the last error, and the count of tries and of cleared errors.
extern "C" int try_launch(int blocks, int room, int other_error, int* tried, int* n, int* cleared) {
  *n = g_cleared = 0;
  const cudaError_t e = tea::launch_resident(blocks, [&](int b) {
    tried[(*n)++] = b;
    if (other_error) return (cudaError_t)other_error;
    return b > room ? cudaErrorCooperativeLaunchTooLarge : cudaSuccess;
  });
  *cleared = g_cleared;
  return (int)e;
}
