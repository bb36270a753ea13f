// rb_blas23_c5_8.cu -- FP32 complex gemv / gemm kernels, folds 5..8.
#include "rb_blas23_impl.cuh"

namespace rb {
const XOps<float> xops_c_f5 = make_xops<float, true, 5>();
const XOps<float> xops_c_f6 = make_xops<float, true, 6>();
const XOps<float> xops_c_f7 = make_xops<float, true, 7>();
const XOps<float> xops_c_f8 = make_xops<float, true, 8>();
}  // namespace rb
