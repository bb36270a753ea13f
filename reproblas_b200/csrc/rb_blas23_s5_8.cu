// rb_blas23_s5_8.cu -- FP32 real gemv / gemm kernels, folds 5..8.
#include "rb_blas23_impl.cuh"

namespace rb {
const XOps<float> xops_s_f5 = make_xops<float, false, 5>();
const XOps<float> xops_s_f6 = make_xops<float, false, 6>();
const XOps<float> xops_s_f7 = make_xops<float, false, 7>();
const XOps<float> xops_s_f8 = make_xops<float, false, 8>();
}  // namespace rb
