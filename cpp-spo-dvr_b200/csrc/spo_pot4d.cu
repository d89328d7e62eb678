// The instantiations of potential4_dmma_kernel, one translation unit per part (SPO_POT4D_PART), compiled in parallel.
#include "spo_pot4d.cuh"

namespace spo {
namespace pot4d {

template <>
Kernel kernel_of_part<SPO_POT4D_PART>(int nphi, int h) {
#define SPO_POT4D_CASE(n) \
  if (nphi == n) return h == 1 ? potential4_dmma_kernel<n, 1> : potential4_dmma_kernel<n, 2>;
#if SPO_POT4D_PART == 0
  SPO_POT4D_CASE(32)
  SPO_POT4D_CASE(8)
  SPO_POT4D_CASE(6)
#elif SPO_POT4D_PART == 1
  SPO_POT4D_CASE(30)
  SPO_POT4D_CASE(16)
  SPO_POT4D_CASE(10)
#elif SPO_POT4D_PART == 2
  SPO_POT4D_CASE(28)
  SPO_POT4D_CASE(20)
  SPO_POT4D_CASE(12)
#else
  SPO_POT4D_CASE(24)
  SPO_POT4D_CASE(22)
  SPO_POT4D_CASE(18)
  SPO_POT4D_CASE(14)
#endif
#undef SPO_POT4D_CASE
  return nullptr;
}

}  // namespace pot4d
}  // namespace spo
