// The FP32 gravity passes of lengths known at run time (fft_smem.cuh).
#include "fft_smem_launch.cuh"

namespace dg {

template <> bool make_fft_plan<float2>(int n, FftPlan *pl) { return make_plan<float2>(n, pl); }
template cudaError_t build_fft_tables<float2>(int, int, FftTables<float2> *);
template cudaError_t launch_phi_fwd<float2>(const FftDisk<float2> &, int, int, int, const FftTables<float2> &, cudaStream_t);
template cudaError_t launch_u_conv<float2>(const FftDisk<float2> &, int, int, const FftTables<float2> &, cudaStream_t);
template cudaError_t launch_phi_inv<float2>(const FftDisk<float2> &, int, int, const FftTables<float2> &, cudaStream_t);

}  // namespace dg
