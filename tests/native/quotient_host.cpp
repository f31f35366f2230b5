// Host build of the quotients of the pressure solve along grid lines (ressim_b200/csrc/rf_quotient.hpp)
// for the CPU tests: counts the pairs whose quotient it accepts and those that differ from the
// division's (a zero's sign apart).
#include <cstdint>

#include "../../ressim_b200/csrc/rf_quotient.hpp"

namespace {

template <class T>
void count(const T* s, const T* d, int64_t n, int64_t* accepted, int64_t* differ, int64_t* first) {
  for (int64_t i = 0; i < n; ++i) {
    bool ok;
    const T q = rf::pen_div(s[i], d[i], rf::pen_recip(d[i]), ok), ref = s[i] / d[i];
    if (!ok) continue;
    ++*accepted;
    if (q != ref && !(q != q && ref != ref)) {
      if (*differ == 0) *first = i;
      ++*differ;
    }
  }
}

}  // namespace

extern "C" void rfh_quotients32(const float* s, const float* d, int64_t n, int64_t* out) {
  count(s, d, n, out, out + 1, out + 2);
}
extern "C" void rfh_quotients64(const double* s, const double* d, int64_t n, int64_t* out) {
  count(s, d, n, out, out + 1, out + 2);
}
