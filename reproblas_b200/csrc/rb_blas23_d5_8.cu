// rb_blas23_d5_8.cu -- FP64 real gemv / gemm kernels, folds 5..8.
#include "rb_blas23_impl.cuh"

namespace rb {
const XOps<double> xops_d_f5 = make_xops<double, false, 5>();
const XOps<double> xops_d_f6 = make_xops<double, false, 6>();
const XOps<double> xops_d_f7 = make_xops<double, false, 7>();
const XOps<double> xops_d_f8 = make_xops<double, false, 8>();
}  // namespace rb
