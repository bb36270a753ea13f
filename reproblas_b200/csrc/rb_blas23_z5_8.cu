// rb_blas23_z5_8.cu -- FP64 complex gemv / gemm kernels, folds 5..8.
#include "rb_blas23_impl.cuh"

namespace rb {
const XOps<double> xops_z_f5 = make_xops<double, true, 5>();
const XOps<double> xops_z_f6 = make_xops<double, true, 6>();
const XOps<double> xops_z_f7 = make_xops<double, true, 7>();
const XOps<double> xops_z_f8 = make_xops<double, true, 8>();
}  // namespace rb
