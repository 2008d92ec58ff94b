// What the sea-level workspace keeps after an allocation failed, on a host
// without a device, where every allocation fails: nothing that a later solve
// on the grid would take for made.
#include <cstdio>

#include "sealevel.cu"

int main() {
  bool good = true;
  auto check = [&](bool ok, const char* what) {
    std::printf("%s: %s\n", ok ? "ok" : "FAIL", what);
    good = good && ok;
  };
  Dev<double> d;
  check(d.Alloc(5) != cudaSuccess && d.p == nullptr && d.n == 0, "a failed allocation counts no values");
  SleWorkspace ws;
  ws.mixerMemory = 5;  // as after a solve with five columns
  check(ws.ResetMixer(6) != SL3DGPU_OK, "six columns fail");
  check(ws.ResetMixer(5) != SL3DGPU_OK, "five columns are not taken for made");
  // as after the first of the nonlinear solve's buffers, the next having failed
  ws.nlOcean.p = reinterpret_cast<double*>(256);
  check(ws.PrepareNonlinear() != SL3DGPU_OK, "the rest of the nonlinear buffers are not taken for made");
  return good ? 0 : 1;
}
