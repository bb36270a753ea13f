// rb_blas23_s2_4.cu -- FP32 real gemv / gemm kernels, folds 2..4.
#include "rb_blas23_impl.cuh"

namespace rb {
const XOps<float> xops_s_f2 = make_xops<float, false, 2>();
const XOps<float> xops_s_f3 = make_xops<float, false, 3>();
const XOps<float> xops_s_f4 = make_xops<float, false, 4>();
}  // namespace rb
