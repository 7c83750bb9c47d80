// The kernels' launchers on several devices of one process (see fake_cuda.cpp).
#include <cstdio>

#include "lvg_internal.cuh"

struct FakeDevice {
  int sms, coop, per_sm;
};
extern const FakeDevice fake_devices[4];
extern int fake_current, fake_refused, fake_launches;

namespace lvg {
void exclusive_scan_u32(const uint32_t *, uint32_t *, size_t, uint32_t *, uint32_t *, cudaStream_t) {}
}  // namespace lvg

int main() {
  using namespace lvg;
  Level lv;
  lv.colors = 1;
  for (int b = 0; b <= NUM_BINS; ++b) lv.bin_start[b] = size_t(b) * 100000;  // work for any number of blocks
  int bad = 0;
  auto check = [&](bool ok, const char *what, int i) {
    if (ok) return;
    std::printf("device %d: %s %d\n", fake_current, what, i);
    ++bad;
  };
  // every call twice on each device, the devices in turn
  for (int turn = 0; turn < 2; ++turn)
    for (fake_current = 0; fake_current < 2; ++fake_current) {
      for (int v = 0; v < 16; ++v) {
        const bool sync = v & 1, unit = v & 2, whole = v & 4, totals = v & 8;
        PhaseArgs a{};
        const uint32_t grid = phase_grid(lv, sync, unit, whole, totals);
        check(grid == unsigned(fake_devices[fake_current].sms), "phase grid", int(grid));
        try { launch_phase(sync, unit, whole, totals, grid, a, nullptr); } catch (...) { check(false, "phase", v); }
      }
      for (int v = 0; v < 3; ++v) {
        AggArgs a{};
        a.count = 1000;
        a.unit = v == 1;
        a.whole = v >= 1;
        for (int b = 1; b < NUM_BINS - 1; ++b)
          try { launch_aggregate_bin(b, a, nullptr); } catch (...) { check(false, "aggregate bin", b); }
        try { launch_aggregate_chunks(a, AggChunks{}, 10, 10, AGG_MAX_PARTS, nullptr); } catch (...) { check(false, "aggregate chunks", v); }
      }
      for (int v = 0; v < 4; ++v) {
        MoveArgs a{};
        a.count = 1000;
        a.unit = v & 1;
        a.hub.hub_begin[1] = a.hub.chunk_begin[1] = 10;
        for (int b = 1; b < NUM_BINS - 1; ++b)
          try { launch_move_bin(b, v & 2, a, nullptr); } catch (...) { check(false, "move bin", b); }
        try { launch_move_hubs(v & 2, a, nullptr); } catch (...) { check(false, "hubs", v); }
      }
    }
  // no cooperative launch, or no block that fits: the phase goes launch by launch
  for (fake_current = 2; fake_current < 4; ++fake_current)
    for (int v = 0; v < 16; ++v) check(phase_grid(lv, v & 1, v & 2, v & 4, v & 8) == 0, "phase grid", v);
  std::printf("launches %d refused %d\n", fake_launches, fake_refused);
  return bad || fake_refused ? 1 : 0;
}
