// rb_blas23_d2_4.cu -- FP64 real gemv / gemm kernels, folds 2..4.
#include "rb_blas23_impl.cuh"

namespace rb {
const XOps<double> xops_d_f2 = make_xops<double, false, 2>();
const XOps<double> xops_d_f3 = make_xops<double, false, 3>();
const XOps<double> xops_d_f4 = make_xops<double, false, 4>();
}  // namespace rb
