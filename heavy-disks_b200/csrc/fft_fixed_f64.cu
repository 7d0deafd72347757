// Compile-time lengths of the FP64 gravity passes (fft_fixed.cuh).
#include "fft_fixed_launch.cuh"

namespace dg {

using V = double2;
#define DG_LENGTHS(X) \
  X(64) X(128) X(256) X(384) X(512) X(768) X(1024) X(2048)

template <> bool fixed_length<V>(int n) {
  switch (n) {
#define X(N) case N: return true;
    DG_LENGTHS(X)
#undef X
    default: return false;
  }
}
template <> void fixed_radices<V>(int n, int *R) {
  switch (n) {
#define X(N) case N: for (int k = 0; k < 5; ++k) R[k] = FixedPlan<V, N>::R[k]; break;
    DG_LENGTHS(X)
#undef X
  }
}
template <> cudaError_t fixed_attrs<V>(int n) {
  switch (n) {
#define X(N) case N: return FixedLen<V, N>::attrs();
    DG_LENGTHS(X)
#undef X
    default: return cudaErrorInvalidValue;
  }
}
template <> cudaError_t fixed_phi_fwd<V>(int n, const FftDisk<V> &d, int b,
                                         int nrows, int ldw, const V *tw, cudaStream_t st) {
  switch (n) {
#define X(N) case N: return FixedLen<V, N>::phi_fwd(d, b, nrows, ldw, tw, st);
    DG_LENGTHS(X)
#undef X
    default: return cudaErrorInvalidValue;
  }
}
template <> cudaError_t fixed_u_conv<V>(int n, const FftDisk<V> &d, int Nc,
                                        int ldw, const V *tw, const V *half, cudaStream_t st) {
  switch (n) {
#define X(N) case N: return FixedLen<V, N>::u_conv(d, Nc, ldw, tw, half, st);
    DG_LENGTHS(X)
#undef X
    default: return cudaErrorInvalidValue;
  }
}
template <> cudaError_t fixed_phi_inv<V>(int n, const FftDisk<V> &d, int nrows,
                                         int ldw, const V *tw, cudaStream_t st) {
  switch (n) {
#define X(N) case N: return FixedLen<V, N>::phi_inv(d, nrows, ldw, tw, st);
    DG_LENGTHS(X)
#undef X
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace dg
