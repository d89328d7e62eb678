// The instantiations of potential5_kernel, one translation unit per part (SPO_POT5_PART), compiled in parallel.
#include "spo_pot5.cuh"

namespace spo {
namespace pot5 {

template <>
Kernel kernel_of_part<SPO_POT5_PART>(int nphi, int h) {
#define SPO_POT5_CASE(n) \
  if (nphi == n) return h == 1 ? potential5_kernel<n, 1> : potential5_kernel<n, 2>;
#if SPO_POT5_PART == 0
  SPO_POT5_CASE(32)
#elif SPO_POT5_PART == 1
  SPO_POT5_CASE(30)
  SPO_POT5_CASE(8)
#elif SPO_POT5_PART == 2
  SPO_POT5_CASE(28)
  SPO_POT5_CASE(6)
#elif SPO_POT5_PART == 3
  SPO_POT5_CASE(24)
  SPO_POT5_CASE(10)
#elif SPO_POT5_PART == 4
  SPO_POT5_CASE(22)
  SPO_POT5_CASE(12)
  SPO_POT5_CASE(14)
#else
  SPO_POT5_CASE(20)
  SPO_POT5_CASE(18)
  SPO_POT5_CASE(16)
#endif
#undef SPO_POT5_CASE
  return nullptr;
}

}  // namespace pot5
}  // namespace spo
