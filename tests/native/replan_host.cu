// The replanning of the pressure solve along grid lines when CUDA calls fail (no device is visible to
// this program): called from a destructor, as the grouping of an ensemble does, it must return, and the
// context goes on without the plan.
#include <cstdio>

#include "../../ressim_b200/csrc/rf_ops.hpp"

namespace {

struct Replan {
  rf::Ctx& c;
  ~Replan() { rf::pencil_replan(c); }
};

}  // namespace

int main() {
  static_assert(noexcept(rf::pencil_replan(*static_cast<rf::Ctx*>(nullptr))), "called from a destructor");
  int devices = 0;
  if (cudaGetDeviceCount(&devices) == cudaSuccess && devices > 0) {
    std::puts("a device is visible");
    return 2;
  }
  static rf::Ctx c;
  c.nx = 10, c.ny = 8, c.nz = 6, c.n = 480;
  c.pen.built = 1;
  for (int f = 0; f < 2; ++f)
    for (int k = 0; k < 5; ++k) c.pen.fits[f][k] = -1;
  { Replan r{c}; }
  std::printf("built %d, CTAs %d\n", c.pen.built, c.pen.cs);
  return c.pen.built == 0 && c.pen.cs == 0 ? 0 : 1;
}
