/* The shared-memory claim of long rows (copy.cu, spread) where a process
 * takes the engine from one device to another, on the host: the calls of the
 * CUDA runtime that ask for the claim are recorded here for the device that
 * is current, and a launch counts as refused where its device was never
 * asked.  The launches themselves fail on a machine without a GPU, which
 * nothing here looks at. */
#include <cuda_runtime.h>
#include <stdarg.h>
#include <stdio.h>

#include "b200shm.h"

static int g_device, g_asked[2], g_launches, g_refused;
template <class K>
static cudaError_t record_attribute(K *, cudaFuncAttribute, int bytes) {
  g_asked[g_device] = bytes;
  return cudaSuccess;
}
#define cudaFuncSetAttribute record_attribute
#include "copy.cu"

namespace b200 {
static State g_state;
State &st() { return g_state; }
int fail(int code, const char *, ...) { return code; }
int cuda_fail(cudaError_t, const char *) { return B200SHM_ERR_CUDA; }
void count_launch(unsigned) {
  g_launches++;
  if (!g_asked[g_device]) g_refused++;
}
int finish(void *, const char *) { return B200SHM_OK; }
int check_team(int, int, int) { return B200SHM_OK; }
int check_extent(uint64_t, uint64_t, const char *) { return B200SHM_OK; }
int grid_sms() { return g_state.sm_count; }
}  // namespace b200

int main() {
  State &s = st();
  s.up = true;
  s.npes = 128;
  s.slice = 64ull << 20;
  s.base = (char *)0x100000000ull;
  uint64_t sizes[128];
  for (uint64_t &x : sizes) x = 65536;
  for (g_device = 0; g_device < 2; g_device++) {
    fcollect_launch(0, 1, 128, 0, 32ull << 20, 65536, nullptr);
    broadcast_launch(0, 0, 1, 128, 0, 32ull << 20, 16ull << 20, nullptr);
    collect_launch(0, 1, 128, 0, 32ull << 20, sizes, nullptr);
  }
  printf("%d launches, %d on a device that was not asked\n", g_launches, g_refused);
  return g_launches == 6 && g_refused == 0 ? 0 : 1;
}
