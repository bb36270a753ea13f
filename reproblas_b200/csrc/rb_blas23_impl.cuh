// rb_blas23_impl.cuh -- binned dgemv on sm_100a, and the table of the FP64 gemv / gemm
// kernels of a fold (the gemm tile is in rb_gemm_tile.cuh).
//
// Every output entry is one binned dot product, so the state of each entry depends only on
// the multiset of its products (plus the beta*y / beta*C initial value), exactly as in the
// reference, where the entry is accumulated by blocked binnedBLAS_dbddot calls:
//   dgemv  y_i <- conv( binned(beta*y_i) + sum_j fl(A_ij * fl(alpha*x_j)) )
//          (src/reproBLAS/rdgemv.c:35-87, src/binnedBLAS/dbdgemv.ccog:57-162: alpha scales x)
//   dgemm  C_ij <- conv( binned(beta*C_ij) + sum_k fl(fl(alpha*A_ik) * B_kj) )
//          (src/reproBLAS/rdgemm.c:41-105, src/binnedBLAS/dbdgemm.ccog:61-420: alpha scales A)
// beta == 0 starts from the empty state, beta == 1 from binned(y) without a multiply, other
// betas from binned(fl(y*beta)); alpha == 1 skips the alpha multiply; alpha == 0 deposits no
// products (the host passes an empty reduction).
#pragma once
#include "rb_binned.cuh"
#include "rb_gemm_tile.cuh"
#include "rb_kernels.cuh"
#include "rb_ptx.cuh"

namespace rb {

// Initial state of an output entry (rdgemv.c:47-57 / rdgemm.c:57-75): binned_dbdconv of
// beta*y, or of y when beta == 1, or the empty state when beta == 0.
template <int F>
__device__ __forceinline__ void init_from_value(Acc<double, F>& a, double y, double beta) {
  a.zero();
  if (beta == 0.0) return;
  double v[1] = {beta == 1.0 ? y : __dmul_rn(y, beta)};
  a.template tile<1>(v, 1);
  a.renorm();
}

// Epilogue shared by the BLAS2/3 kernels: combine the products' state `a` (renormalised)
// with the entry's initial state and write the result. `yv` is *out_value, loaded by the
// caller (kOutValue only), so that the load can be issued early.
template <int F>
__device__ __forceinline__ void finish_entry_pre(Acc<double, F>& a, int mode, double yv,
                                                 double* out_value, double beta,
                                                 double* out_binned) {
  if (mode == kOutValue) {
    Acc<double, F> init;
    init_from_value(init, yv, beta);
    init.merge(a);
    init.renorm();
    double p[F], c[F];
    init.store(p, c, 1);
    *out_value = conv<F>(p, c, 1);
  } else {
    Acc<double, F> prev;
    prev.load(out_binned, out_binned + F, 1);
    prev.merge(a);
    prev.renorm();
    prev.store(out_binned, out_binned + F, 1);
  }
}

template <int F>
__device__ __forceinline__ void finish_entry(Acc<double, F>& a, int mode, double* out_value,
                                             double beta, double* out_binned) {
  finish_entry_pre<F>(a, mode, mode == kOutValue ? *out_value : 0.0, out_value, beta, out_binned);
}

__device__ __forceinline__ void ld2(const double* p, double& a, double& b) {
  double2 v = __ldg((const double2*)p);
  a = v.x;
  b = v.y;
}

// Merge `count` records (pri F, car F, flags) at `rec` (shared memory) into `t`.
template <int F>
__device__ __forceinline__ void merge_records(Acc<double, F>& t, const double* rec, int count) {
  constexpr int REC = 2 * F + 2;
  for (int p = 0; p < count; p++) {
    const double* r = rec + p * REC;
    Acc<double, F> o;
    o.zero();
#pragma unroll
    for (int i = 0; i < F; i++) { o.pri[i] = r[i]; o.car[i] = r[F + i]; }
    o.flags = (unsigned)__double_as_longlong(r[2 * F]);
    o.set_idx_from_pri();
    t.merge(o);
  }
}

// ---------------------------------------------------------------------------------------
// gemv, reduction along contiguous rows: out_r = sum_c A[r*lda + c] * bx_c, r < R, c < C.
// S warps share a row (S = 1, 2, 4, 8); a CTA of 8 warps covers 8/S rows. With g.vec (row
// starts and x 16-byte aligned, incx 1) lanes read 16-byte pairs: 512 contiguous bytes per
// warp load; the row is cut into chunks of a multiple of 8 elements so they stay aligned.
// ---------------------------------------------------------------------------------------
template <int F>
__global__ void __launch_bounds__(256) gemv_rows_kernel(GemvArgs g) {
  constexpr int REC = 2 * F + 2;
  __shared__ double smem[8 * REC];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int S = g.split;
  const int rows_per_cta = 8 / S;
  const int rloc = warp / S, part = warp % S;
  const long long r = (long long)blockIdx.x * rows_per_cta + rloc;
  Acc<double, F> a;
  a.zero();
  if (r < g.R) {
    const double* row = g.A + r * g.lda;
    const long long chunk = ((g.C + S - 1) / S + 7) / 8 * 8;
    const long long c0 = part * chunk < g.C ? part * chunk : g.C;
    const long long c1 = c0 + chunk < g.C ? c0 + chunk : g.C;
    if (g.vec) {
      const long long npair = (c1 - c0) / 2;
      constexpr int K = 4;
#pragma unroll 1
      for (long long pb = lane; pb < npair; pb += 32 * K) {
        double v[2 * K];
        int nv = 0;
#pragma unroll
        for (int k = 0; k < K; k++) {
          const long long pi = pb + 32 * k;
          v[2 * k] = v[2 * k + 1] = 0.0;
          if (pi < npair) {
            double a0, a1, x0, x1;
            ld2(row + c0 + 2 * pi, a0, a1);
            ld2(g.x + c0 + 2 * pi, x0, x1);
            if (g.alpha != 1.0) { x0 = __dmul_rn(x0, g.alpha); x1 = __dmul_rn(x1, g.alpha); }
            v[2 * k] = __dmul_rn(a0, x0);
            v[2 * k + 1] = __dmul_rn(a1, x1);
            nv = 2 * k + 2;
          }
        }
        a.template tile<2 * K>(v, nv);
      }
      if (((c1 - c0) & 1) && lane == 0) {
        double xv = __ldg(g.x + (c1 - 1));
        if (g.alpha != 1.0) xv = __dmul_rn(xv, g.alpha);
        double v[1] = {__dmul_rn(__ldg(row + (c1 - 1)), xv)};
        a.template tile<1>(v, 1);
      }
    } else {
      constexpr int K = 4;
#pragma unroll 1
      for (long long b = c0 + lane; b < c1; b += 32 * K) {
        double v[K];
        int nv = 0;
#pragma unroll
        for (int k = 0; k < K; k++) {
          long long c = b + 32 * k;
          v[k] = 0.0;
          if (c < c1) {
            double xv = __ldg(g.x + c * g.incx);
            if (g.alpha != 1.0) xv = __dmul_rn(xv, g.alpha);
            v[k] = __dmul_rn(__ldg(row + c), xv);
            nv = k + 1;
          }
        }
        a.template tile<K>(v, nv);
      }
    }
  }
  a.renorm();
  warp_merge_all(a);
  if (lane == 0) {
    double* rec = smem + warp * REC;
#pragma unroll
    for (int i = 0; i < F; i++) { rec[i] = a.pri[i]; rec[F + i] = a.car[i]; }
    rec[2 * F] = __longlong_as_double((long long)a.flags);
  }
  __syncthreads();
  if (threadIdx.x < rows_per_cta) {
    const long long rr = (long long)blockIdx.x * rows_per_cta + threadIdx.x;
    if (rr < g.R) {
      Acc<double, F> t;
      t.zero();
      merge_records<F>(t, smem + threadIdx.x * S * REC, S);
      finish_entry<F>(t, g.mode, g.y + rr * g.incy, g.beta, g.ybin + rr * g.incy * 2 * F);
    }
  }
}

// ---------------------------------------------------------------------------------------
// gemv, reduction along strided columns: out_c = sum_r A[r*lda + c] * bx_r, c < C, r < R.
// A CTA of 256 threads is G = g.split row groups (1, 2, 4, 8) of T = 256/G threads; thread
// t of a group owns W columns (W = 2 with g.vec, A and lda 16-byte aligned: one 16-byte load
// per row; else 1), so a CTA covers T*W columns and a warp reads 32*W contiguous doubles of
// a row. grid = (column blocks, row chunks); inside a chunk, group q takes rows q, q+G, ...
// The groups' states are merged through shared memory, group 0 writes the chunk's partial
// state to scratch (structure of arrays), and the last chunk-CTA to arrive for a column
// block merges the partials (group q takes chunks q, q+G, ...; then the groups merge once
// more) and finishes the entries. More groups mean narrower column blocks, more of them and
// fewer chunks, which shortens that final serial merge.
// ---------------------------------------------------------------------------------------

// Tree merge of the G row groups' states (each renormalised) through shared memory laid out
// as sm[i * 256 + thread], i < 2F+1; group 0 ends with the merged state. Every thread of the
// CTA must call it.
template <int F>
__device__ __forceinline__ void merge_row_groups(Acc<double, F>& a, double* sm, int grp, int t,
                                                 int G, int T) {
#pragma unroll 1
  for (int s = 1; s < G; s <<= 1) {
    const int m = grp & (2 * s - 1);
    if (m == s) {
#pragma unroll
      for (int i = 0; i < F; i++) {
        sm[i * 256 + threadIdx.x] = a.pri[i];
        sm[(F + i) * 256 + threadIdx.x] = a.car[i];
      }
      sm[2 * F * 256 + threadIdx.x] = __longlong_as_double((long long)a.flags);
    }
    __syncthreads();
    if (m == 0) {
      const int src = (grp + s) * T + t;
      Acc<double, F> o;
      o.zero();
#pragma unroll
      for (int i = 0; i < F; i++) {
        o.pri[i] = sm[i * 256 + src];
        o.car[i] = sm[(F + i) * 256 + src];
      }
      o.flags = (unsigned)__double_as_longlong(sm[2 * F * 256 + src]);
      o.set_idx_from_pri();
      a.merge(o);
    }
    __syncthreads();
  }
}

template <int F, int W>
__device__ __forceinline__ void gemv_cols_body(const GemvArgs& g, double* sm) {
  const int G = g.split, T = 256 / G;
  const int lgT = __ffs(T) - 1;
  const int grp = threadIdx.x >> lgT, t = threadIdx.x & (T - 1);
  const long long cbase = ((long long)blockIdx.x * T + t) * W;
  const int chunk = blockIdx.y, nchunks = gridDim.y;
  const long long rows_per = (g.R + nchunks - 1) / nchunks;
  const long long r0 = (long long)chunk * rows_per;
  const long long r1 = r0 + rows_per < g.R ? r0 + rows_per : g.R;
  const long long stride = (long long)nchunks * g.C;
  Acc<double, F> a[W];
#pragma unroll
  for (int w = 0; w < W; w++) a[w].zero();
  if (cbase < g.C) {
    constexpr int K = 4;
#pragma unroll 1
    for (long long b = r0 + grp; b < r1; b += (long long)G * K) {
      double v[W][K];
      int nv = 0;
#pragma unroll
      for (int k = 0; k < K; k++) {
        const long long r = b + (long long)k * G;
#pragma unroll
        for (int w = 0; w < W; w++) v[w][k] = 0.0;
        if (r < r1) {
          double xv = __ldg(g.x + r * g.incx);
          if (g.alpha != 1.0) xv = __dmul_rn(xv, g.alpha);
          if constexpr (W == 2) {
            double a0, a1;
            ld2(g.A + r * g.lda + cbase, a0, a1);
            v[0][k] = __dmul_rn(a0, xv);
            v[1][k] = __dmul_rn(a1, xv);
          } else {
            v[0][k] = __dmul_rn(__ldg(g.A + r * g.lda + cbase), xv);
          }
          nv = k + 1;
        }
      }
#pragma unroll
      for (int w = 0; w < W; w++) a[w].template tile<K>(v[w], nv);
    }
  }
#pragma unroll
  for (int w = 0; w < W; w++) {
    a[w].renorm();
    merge_row_groups<F>(a[w], sm, grp, t, G, T);
  }
  if (grp == 0) {
#pragma unroll
    for (int w = 0; w < W; w++) {
      const long long c = cbase + w;
      if (c < g.C) {
        double* s = g.scratch + (long long)chunk * g.C + c;
#pragma unroll
        for (int i = 0; i < F; i++) {
          s[(long long)i * stride] = a[w].pri[i];
          s[(long long)(F + i) * stride] = a[w].car[i];
        }
        s[(long long)(2 * F) * stride] = __longlong_as_double((long long)a[w].flags);
      }
    }
  }
  // last chunk-CTA of this column block merges
  __shared__ unsigned s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned tk = atomicAdd(g.tickets + blockIdx.x, 1u);
    s_last = (tk == (unsigned)nchunks - 1) ? 1u : 0u;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
#pragma unroll
  for (int w = 0; w < W; w++) a[w].zero();
  if (cbase < g.C) {
#pragma unroll 1
    for (int ch = grp; ch < nchunks; ch += G) {
#pragma unroll
      for (int w = 0; w < W; w++) {
        const long long c = cbase + w;
        if (c < g.C) {
          const double* s = g.scratch + (long long)ch * g.C + c;
          Acc<double, F> o;
          o.zero();
#pragma unroll
          for (int i = 0; i < F; i++) {
            o.pri[i] = __ldcg(s + (long long)i * stride);
            o.car[i] = __ldcg(s + (long long)(F + i) * stride);
          }
          o.flags = (unsigned)__double_as_longlong(__ldcg(s + (long long)(2 * F) * stride));
          o.set_idx_from_pri();
          a[w].merge(o);
        }
      }
    }
  }
#pragma unroll
  for (int w = 0; w < W; w++) merge_row_groups<F>(a[w], sm, grp, t, G, T);
  if (grp == 0) {
#pragma unroll
    for (int w = 0; w < W; w++) {
      const long long c = cbase + w;
      if (c < g.C) finish_entry<F>(a[w], g.mode, g.y + c * g.incy, g.beta, g.ybin + c * g.incy * 2 * F);
    }
  }
  if (threadIdx.x == 0) g.tickets[blockIdx.x] = 0u;
}

template <int F>
__global__ void __launch_bounds__(256, F <= 3 ? 3 : 2) gemv_cols_kernel(GemvArgs g) {
  __shared__ double sm[(2 * F + 1) * 256];
  if (g.vec) gemv_cols_body<F, 2>(g, sm);
  else gemv_cols_body<F, 1>(g, sm);
}

template <int F>
cudaError_t launch_gemv(const GemvArgs& g, bool rows, dim3 grid, cudaStream_t s) {
  if (rows) gemv_rows_kernel<F><<<grid, 256, 0, s>>>(g);
  else gemv_cols_kernel<F><<<grid, 256, 0, s>>>(g);
  return cudaGetLastError();
}

}  // namespace rb

#include "rb_gemv_stream.cuh"

namespace rb {

template <int F>
Blas23FoldOps make_blas23_ops() {
  Blas23FoldOps o;
  o.gemv = launch_gemv<F>;
  o.gemm_plan = gt::plan_gemm<double, false, F>;
  o.gemm = gt::launch_gemm<double, false, F>;
  // the TMA-fed gemv kernels fit their registers (17 warps per SM) up to fold 3
  if constexpr (F <= 3) {
    o.gemv_stream = gs::launch_gemv_stream<F>;
    o.gemv_stream_prepare = gs::prepare_gemv_stream<F>;
  } else {
    o.gemv_stream = nullptr;
    o.gemv_stream_prepare = nullptr;
  }
  return o;
}

}  // namespace rb
