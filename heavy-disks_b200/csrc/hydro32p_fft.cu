// The packed hydro step of disks on FFT gravity (hydro32p_launch.cuh).
#include "hydro32p_launch.cuh"

namespace dg {

template <> cudaError_t launch_hydro32p<false>(const Hydro32pArgs &a, int fm, cudaStream_t st) {
  return launch_hydro32p_as<false>(a, fm, st);
}
template <> cudaError_t prepare_hydro32p<false>() { return prepare_hydro32p_as<false>(); }

}  // namespace dg
