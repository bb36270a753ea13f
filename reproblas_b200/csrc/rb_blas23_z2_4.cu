// rb_blas23_z2_4.cu -- FP64 complex gemv / gemm kernels, folds 2..4.
#include "rb_blas23_impl.cuh"

namespace rb {
const XOps<double> xops_z_f2 = make_xops<double, true, 2>();
const XOps<double> xops_z_f3 = make_xops<double, true, 3>();
const XOps<double> xops_z_f4 = make_xops<double, true, 4>();
}  // namespace rb
