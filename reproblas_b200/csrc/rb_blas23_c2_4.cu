// rb_blas23_c2_4.cu -- FP32 complex gemv / gemm kernels, folds 2..4.
#include "rb_blas23_impl.cuh"

namespace rb {
const XOps<float> xops_c_f2 = make_xops<float, true, 2>();
const XOps<float> xops_c_f3 = make_xops<float, true, 3>();
const XOps<float> xops_c_f4 = make_xops<float, true, 4>();
}  // namespace rb
