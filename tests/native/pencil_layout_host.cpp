// Host build of the shared-memory layout of the pressure solve along grid lines
// (ressim_b200/csrc/rf_pencil_layout.hpp) for the CPU tests.  Places of a CTA that other CTAs of its
// cluster store to are addressed by the storing CTA's own offsets, so they must not depend on how
// many listed rows (wells) and entries a CTA has.
#include <cstdint>

#include "../../ressim_b200/csrc/rf_pencil_layout.hpp"

namespace {

template <class T>
void remote_places(int nx, int nz, int cols, int cs, int chunk, int nvw, int wells, int entries, int64_t* out) {
  const rf::PenLayout o = rf::pen_layout<T>(nx, nz, cols, cs, chunk, nvw, wells, entries);
  const size_t places[] = {o.nbr, o.mbar, o.red, o.bad};
  for (int k = 0; k < 4; ++k) out[k] = int64_t(places[k]);
  out[4] = int64_t(o.total);
}

}  // namespace

extern "C" void rfh_pencil_remote_places(int32_t bytes, int32_t nx, int32_t nz, int32_t cols, int32_t cs, int32_t chunk,
                                         int32_t nvw, int32_t wells, int32_t entries, int64_t* out) {
  if (bytes == 4)
    remote_places<float>(nx, nz, cols, cs, chunk, nvw, wells, entries, out);
  else
    remote_places<double>(nx, nz, cols, cs, chunk, nvw, wells, entries, out);
}
