// Host program of tests/test_stage_layouts.py: checks the compile-time layouts
// of the stage kernels, taken from the kernels' own header.  Prints one line per
// fault and returns their number (at most 100).
#include <cstdio>
#include <vector>
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

// elements a + r STEP (r < R) of the line at byte offset o, as panel_read and
// panel_write address them
template <typename PA, bool XCH, int R, int STEP, int r = 0>
static void panel_set(const char* name, unsigned panel, unsigned x, unsigned a) {
  if constexpr (r < R) {
    const unsigned o = panel + x * PA::LX, oa = o ^ PA::template off<XCH>(a);
    const unsigned got = PA::template addr<XCH, (unsigned)r * STEP>(oa, o, a);
    const unsigned want = panel + (PA::template off<XCH>(a + r * STEP) ^ (x * PA::LX));
    CHECK(got == want, "%s order %d line %u: element %u + %d * %d at %u, not %u", name, (int)XCH, x, a, r, STEP, got,
          want);
    panel_set<PA, XCH, R, STEP, r + 1>(name, panel, x, a);
  }
}

// the accesses of panel_load, panel_fft and panel_store by every thread of a line
template <typename PA, int p = 0>
static void panel_passes(const char* name, unsigned panel, unsigned x) {
  using PL = typename PA::PL;
  constexpr int N = PA::N, R = PL::rad(p), NS = PL::ns(p), LAST = PL::NPASS - 1;
  for (int j = 0; j < N / R; j++) {
    const unsigned w = j / NS * NS * R + j % NS;   // first result of butterfly j
    if constexpr (p == 0) panel_set<PA, false, R, N / R>(name, panel, x, j);
    if constexpr (p > 0) panel_set<PA, true, R, N / R>(name, panel, x, j);
    if constexpr (p < LAST) panel_set<PA, true, R, NS>(name, panel, x, w);
    if constexpr (p == LAST) panel_set<PA, false, R, NS>(name, panel, x, w);
  }
  if constexpr (p < LAST) panel_passes<PA, p + 1>(name, panel, x);
}

// every element of every line has its own place, in both orders
template <typename PA, bool XCH>
static void panel_places(const char* name) {
  std::vector<char> used(PA::BYTES / sizeof(typename PA::C), 0);
  for (unsigned x = 0; x < (unsigned)PA::PW; x++)
    for (unsigned i = 0; i < (unsigned)PA::N; i++) {
      const unsigned b = PA::template off<XCH>(i) ^ (x * PA::LX), e = b / sizeof(typename PA::C);
      const bool ok = b % sizeof(typename PA::C) == 0 && e < used.size() && !used[e];
      CHECK(ok, "%s order %d: element %u of line %u at byte %u", name, (int)XCH, i, x, b);
      if (ok) used[e] = 1;
    }
}

template <typename PA>
static void panel(const char* type, const char* kind) {
  char name[64];
  std::snprintf(name, sizeof name, "%s panel of n = %d, %s", kind, PA::N, type);
  panel_places<PA, false>(name);
  panel_places<PA, true>(name);
  for (unsigned k = 0; k < 2; k++)
    for (unsigned x = 0; x < (unsigned)PA::PW; x++) panel_passes<PA>(name, k * PA::BYTES, x);
}

template <int N>
static void panels() {
  panel<Panel<float, N>>("FP32", "z");
  panel<Panel<double, N>>("FP64", "z");
  if constexpr (N >= 512) {
    panel<Panel<float, N, true>>("FP32", "one-slot");
    panel<Panel<double, N, true>>("FP64", "one-slot");
  }
}

int main() {
  panels<16>();
  panels<32>();
  panels<48>();
  panels<64>();
  panels<96>();
  panels<128>();
  panels<256>();
  panels<512>();
  panels<1024>();
  tc_storage("K3", 6, K3Launch<float, 1024, 0, true>::SMEM_TC);
  tc_storage("K3 scalar", 12, K3Launch<float, 1024, 1, true>::SMEM_TC);
  tc_storage("K5", K5Launch<float, 1024, 0>::LINES_TC, K5Launch<float, 1024, 0>::SMEM_TC);
  tc_storage("K5 scalar", K5Launch<float, 1024, 1>::LINES_TC, K5Launch<float, 1024, 1>::SMEM_TC);
  return faults < 100 ? faults : 100;
}
