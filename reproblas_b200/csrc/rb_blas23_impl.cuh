// rb_blas23_impl.cuh -- the gemv / gemm kernels of one element type and fold, as a table
// (instantiated in rb_blas23_<type><folds>.cu; one fold's kernels take a while to compile).
#pragma once
#include "rb_gemm_tile.cuh"
#include "rb_gemv_stream.cuh"

namespace rb {

template <typename E, bool CX, int F>
constexpr XOps<E> make_xops() {
  return XOps<E>{gs::gemv_streams<E, CX, F>, gs::launch_gemv<E, CX, F>, gt::plan_gemm<E, CX, F>,
                 gt::launch_gemm<E, CX, F>};
}

}  // namespace rb
