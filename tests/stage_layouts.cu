// Host program of tests/test_stage_layouts.py: checks the compile-time layouts
// of the stage kernels, taken from the kernels' own header.  Prints one line per
// fault and returns their number (at most 100).
#include <cstdio>
#include "stage_kernels.cuh"

using namespace psdns;

static int faults = 0;
#define CHECK(ok, ...)               \
  do {                               \
    if (!(ok)) {                     \
      faults++;                      \
      std::printf(__VA_ARGS__);      \
      std::printf("\n");             \
    }                                \
  } while (0)

// fft1024_lines overwrites its lines' storage up to the next multiple of four
// lines, and the tail with the B operands comes right after the storage
static void tc_storage(const char* name, int lines, size_t smem) {
  const size_t line = sizeof(float2) * LS<float, 1024>::value, tw = sizeof(float2) * FFTPlan<float, 1024>::TWSIZE;
  const size_t need = tw + (size_t)((lines + 3) / 4 * 4) * line + kTcTail;
  CHECK(smem >= need, "%s: %d lines need %zu bytes, have %zu", name, lines, need, smem);
  CHECK(smem <= 227 * 1024, "%s: %zu bytes of shared memory", name, smem);
}

int main() {
  tc_storage("K3", 6, K3Launch<float, 1024, 0, true>::SMEM_TC);
  tc_storage("K3 scalar", 12, K3Launch<float, 1024, 1, true>::SMEM_TC);
  tc_storage("K5", K5Launch<float, 1024, 0>::LINES_TC, K5Launch<float, 1024, 0>::SMEM_TC);
  tc_storage("K5 scalar", K5Launch<float, 1024, 1>::LINES_TC, K5Launch<float, 1024, 1>::SMEM_TC);
  return faults < 100 ? faults : 100;
}
