// Instantiation unit: Dirac-operator kernels of representation dimension d = 8
// (declarations in yg_kernels.h, device code in yg_dirac_impl.cuh).
#include "yg_dirac_impl.cuh"

namespace yg {
template void DK<8>::hop(const HopArgs<double> &, int, cudaStream_t);
template void DK<8>::hop(const HopArgs<float> &, int, cudaStream_t);
template void DK<8>::clover(double2 *, const double2 *, const double2 *, Geom, double, double, int, int, int, cudaStream_t);
template void DK<8>::clover_inv(double2 *, const double2 *, const double2 *, Geom, int, cudaStream_t);
template void DK<8>::ldl_inverse(double2 *, double2 *, const double2 *, Geom, double, double, int, cudaStream_t);
template void DK<8>::cinv_float(float2 *, const double2 *, int, cudaStream_t);
template void DK<8>::logdet(double *, const double2 *, int, cudaStream_t);
}  // namespace yg
