// One kernel family of one precision form per translation unit: SPO_LAUNCH_T (float or double) and SPO_LAUNCH_PART.
#include "spo_launch.cuh"

namespace spo_host {

using T = SPO_LAUNCH_T;

#if SPO_LAUNCH_PART == 0
template bool launch_axis2<T>(int, const spo::Axis2Args<T>&, long long, cudaStream_t);
#elif SPO_LAUNCH_PART == 1
template bool launch_xy2<T>(const spo::XyArgs<T>&, long long, cudaStream_t);
#elif SPO_LAUNCH_PART == 2
template void launch_pot2<T>(int, const spo::Pot2Args<T>&, unsigned, std::size_t, cudaStream_t);
#elif SPO_LAUNCH_PART == 3
template void launch_pot3<T>(int, const spo::Pot2Args<T>&, dim3, unsigned, std::size_t, cudaStream_t);
#elif SPO_LAUNCH_PART == 5
template KinLaunch<T> kin_configure<T>(int, int, int, bool, int, long long);
#elif SPO_LAUNCH_PART == 6
template KinLaunch<float> kin_configure<spo::Wide>(int, int, int, bool, int, long long);
#else
template Pot4Kernel<T> pot4_kernel_for<T>(int, int);
#endif

}  // namespace spo_host
