// The FP64 gravity passes of lengths known at run time (fft_smem.cuh).
#include "fft_smem_launch.cuh"

namespace dg {

template <> bool make_fft_plan<double2>(int n, FftPlan *pl) { return make_plan<double2>(n, pl); }
template cudaError_t build_fft_tables<double2>(int, int, FftTables<double2> *);
template cudaError_t launch_phi_fwd<double2>(const FftDisk<double2> &, int, int, int, const FftTables<double2> &, cudaStream_t);
template cudaError_t launch_u_conv<double2>(const FftDisk<double2> &, int, int, const FftTables<double2> &, cudaStream_t);
template cudaError_t launch_phi_inv<double2>(const FftDisk<double2> &, int, int, const FftTables<double2> &, cudaStream_t);

}  // namespace dg
