// rb_api_blas23.cu -- C ABI for the binned gemv / gemm of every element type:
// reproBLAS_r[dszc]gemv, r[dszc]gemm, [dszc]gemv, [dszc]gemm and binnedBLAS_dbdgemv, sbsgemv,
// zbzgemv, cbcgemv, dbdgemm, sbsgemm, zbzgemm, cbcgemm (include/reproBLAS.h:61-93, 130-161;
// include/binnedBLAS.h:99-133).
//
// Orders and transposes map onto the kernels' forms the way the reference does it:
// column-major is row-major with the transpose flipped (dbdgemv.ccog:146-158,
// zbzgemv.ccog:184-196), gemm takes general operand strides. TransA / TransB: 'n'/'N' no transpose, 't'/'T' transpose, anything else the
// conjugate transpose (the reference's default branches; for real elements every non-'n'
// form is the transpose). Complex alpha and beta are read from host memory as two adjacent
// reals, like the reference does. Host operands are copied to a device workspace first;
// outputs are copied back before returning.
//
// One deliberate difference: the reference's column-major conjugate-transpose zbzgemv /
// cbcgemv cut each column's dot into blocks of MIN(X_BLOCK, N - j) elements while j runs
// over the M rows (zbzgemv.ccog:214-218, cbcgemv.ccog:214-218), which equals the mathematical
// A^H x only when M == N. Here every entry is the full A^H x.
#include <algorithm>
#include <cstring>
#include <string>

#include "rb_gemv_stream.cuh"
#include "rb_host.h"
#include "../../include/reproblas_b200.h"

namespace rb {
namespace {

bool xrow(char o) { return o == 'r' || o == 'R'; }
bool xnt(char t) { return t == 'n' || t == 'N'; }
bool xplain_t(char t) { return t == 't' || t == 'T'; }

// The fixed-fold kernels (folds 2..8); nullptr above them, where the run-time fold path runs.
template <typename E, bool CX>
const XOps<E>* xops_for(int fold) {
  if (fold < 2 || fold > kMaxFold) return nullptr;
  if constexpr (sizeof(E) == 8) {
    static const XOps<double>* const d[] = {&xops_d_f2, &xops_d_f3, &xops_d_f4, &xops_d_f5,
                                            &xops_d_f6, &xops_d_f7, &xops_d_f8};
    static const XOps<double>* const z[] = {&xops_z_f2, &xops_z_f3, &xops_z_f4, &xops_z_f5,
                                            &xops_z_f6, &xops_z_f7, &xops_z_f8};
    return (CX ? z : d)[fold - 2];
  } else {
    static const XOps<float>* const s[] = {&xops_s_f2, &xops_s_f3, &xops_s_f4, &xops_s_f5,
                                           &xops_s_f6, &xops_s_f7, &xops_s_f8};
    static const XOps<float>* const c[] = {&xops_c_f2, &xops_c_f3, &xops_c_f4, &xops_c_f5,
                                           &xops_c_f6, &xops_c_f7, &xops_c_f8};
    return (CX ? c : s)[fold - 2];
  }
}

// alpha / beta: real scalars, or the two reals a complex pointer addresses
template <typename E, bool CX>
struct Scalar {
  E r, i;
};
template <typename E, bool CX>
Scalar<E, CX> read_scalar(E v) { return {v, E(0)}; }
template <typename E, bool CX>
Scalar<E, CX> read_scalar(const void* p) {
  const E* q = (const E*)p;
  return {q[0], q[1]};
}

template <typename E, bool CX>
struct XGemvReq {
  int fold;
  char order, trans;
  int M, N;
  Scalar<E, CX> alpha;
  const void* A;
  int lda;
  const void* X;
  int incX;
  Scalar<E, CX> beta;
  void* Y;          // values (kOutValue) or binned states (kOutBinned)
  int incY;
  int mode;
};

unsigned gemv_slot(bool rows, int G, int es, int phases) {
  return rows ? gs::slot_bytes<true>(G, es, phases) : gs::slot_bytes<false>(G, es, phases);
}

// Tensor maps of the stored Rs x Cs matrix, one per phase of its rows, in 8-byte words (the
// copies move bits, whatever the element type): phase h starts at the 16-byte boundary at or
// before row h and its rows span the elements' bytes from there.
bool gemv_maps(GemvMaps* maps, const void* A, size_t es, long long Rs, long long Cs, long long lda,
               int phases, bool rows, int G) {
  auto enc = tensor_map_encoder();
  if (!enc) {
    set_error(RB_ERR_CUDA, "gemv: cuTensorMapEncodeTiled is unavailable");
    return false;
  }
  // box: a stage's rows of one phase, slots of the width the kernel expects (slot_bytes); rows
  // kernel, one phase: 128 bytes of a group's rows, swizzled
  const bool swz = rows && phases == 1;
  const cuuint32_t slot = swz ? 128u : gemv_slot(rows, G, (int)es, phases);
  const cuuint32_t stage_rows = rows ? 512u / G : (cuuint32_t)(128 / es) * G;
  for (int h = 0; h < phases && h < Rs; h++) {
    const uintptr_t row = (uintptr_t)A + (size_t)h * lda * es;
    const size_t shift = row % 16;
    cuuint64_t dims[2] = {(cuuint64_t)((shift + (size_t)Cs * es + 7) / 8),
                          (cuuint64_t)((Rs - h + phases - 1) / phases)};
    cuuint64_t strides[1] = {(cuuint64_t)phases * lda * es};
    cuuint32_t box[2] = {slot / 8, stage_rows / phases};
    cuuint32_t estr[2] = {1u, 1u};
    const CUresult r = enc(&maps->m[h], CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, (void*)(row - shift), dims,
                           strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           swz ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
      set_error(RB_ERR_CUDA, "gemv: cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
      return false;
    }
  }
  // fewer rows than phases: the other phases hold no row (their boxes are loaded all the same,
  // into slots that nothing reads)
  for (int h = (int)Rs; h < phases; h++) maps->m[h] = maps->m[0];
  return true;
}

// Decomposition of the streaming gemv (rb_gemv_stream.cuh): G thread groups per output, units of P
// = 512/G outputs, stages of 128/es*G elements of the reduction, and the split of the stages
// over at most one CTA per SM.
struct GemvShape {
  int G, grid, q, rem, parts;
  long long nunits, nb;
  size_t records, tickets;   // partial states and tickets of what is cut between CTAs (0: nothing is)
};
// `uncut`: no unit is cut between CTAs (no scratch).
GemvShape gemv_shape(bool rows, long long nout, long long nred, int es, bool cx, int fold, int phases,
                     int sms, bool uncut) {
  // Cost in us, from a sweep over G and the grid on the shapes of 128 MiB and below. A stage takes
  // its CTA 1.45 us (64 KB at the SM's share of HBM) or the deposits' issue time: measured 3.1 at
  // fold 3 for complex elements. Behind the last stage: 5 us when no unit is cut, 8 when
  // every CTA has one part of one unit, 10 when the ranges cut anywhere (two runs per CTA), and
  // about 0.4 per part a lane merges.
  const double work = (es == 8 && !cx) || es == 16 ? (3 * fold - 1) * 2 + 2 * fold : (3 * fold - 1) + fold;
  const double dep = cx ? 4.0 * (128 / es) : 128 / es;
  double stage = dep * work * 4 / 1900 * (cx ? 2.0 : 1.15);
  if (stage < 1.45) stage = 1.45;
  GemvShape best{};
  double best_cost = 0;
  for (int G = 2; G <= 8; G *= 2) {
    // columns: a box is at most 256 words of 8 bytes wide, and a thread's rows are of one phase
    if (!rows && (gemv_slot(false, G, es, phases) > 2048 || G < phases)) continue;
    // bank conflicts between a warp's groups
    const double m = G == 8 ? (rows ? (phases > 1 ? 1.2 : 1.0) : es == 16 ? 0.98 : es == 4 ? 1.4 : cx ? 1.04 : 1.13)
                            : (G == 2 ? 1.05 : 1.0);
    GemvShape s{};
    s.G = G;
    const long long P = 512 / G, SC = (long long)(128 / es) * G;
    s.nunits = (nout + P - 1) / P;
    s.nb = (nred + SC - 1) / SC;
    const long long T = s.nunits * s.nb;
    for (int way = uncut ? 1 : 0; way < 2; way++) {
      double ends;
      long long per;   // stages of the busiest CTA
      bool cut;        // some unit is cut between CTAs
      long long share = 1;   // at most so many
      if (way == 0) {
        s.parts = 0;
        s.grid = (int)(T < sms ? T : sms);
        s.q = (int)(T / s.grid);
        s.rem = (int)(T % s.grid);
        per = (T + s.grid - 1) / s.grid;
        cut = s.rem != 0 || s.q % s.nb != 0;
        share = s.nb / s.q + 2;   // a unit meets at most ceil((nb-1) / q) + 1 ranges
        ends = s.grid == s.nunits && s.rem == 0 ? 5 : 10 + 0.4 * (double)(share / G);
      } else if (s.nunits <= sms && !uncut) {
        long long p = sms / s.nunits;
        if (p > s.nb) p = s.nb;
        s.parts = (int)p;
        s.grid = (int)(s.nunits * p);
        s.q = 1;
        s.rem = (int)s.nunits;
        per = (s.nb + p - 1) / p;
        cut = p > 1;
        share = p;
        ends = p == 1 ? 5 : 8 + 0.4 * (double)((p + G - 1) / G);
      } else {
        const long long wu = (s.nunits + sms - 1) / sms;
        s.parts = 1;
        s.q = (int)wu;
        s.rem = (int)s.nunits;
        s.grid = (int)((s.nunits + wu - 1) / wu);
        per = wu * s.nb;
        cut = false;
        ends = 5;
      }
      s.records = cut ? (size_t)2 * s.grid * P : 0;           // see Ends
      s.tickets = cut && share <= gs::kWide ? (size_t)s.grid * (gs::kConsumers / 32) : 0;   // none: see gemv_sum_parts_kernel
      const double cost = (double)per * stage * m + ends;
      if (best.G == 0 || cost < best_cost) {
        best = s;
        best_cost = cost;
      }
    }
  }
  return best;
}

// Shape of the direct columns kernel: G row groups per CTA and `parts` row chunks. Cost model in
// units of one row per thread: the streaming part (waves of CTAs, two per SM, times rows per
// thread, plus the groups' merge) and the sum of the chunks' partial states.
// `uncut`: one chunk (no scratch).
GemvShape gemv_cols_direct_shape(long long nout, long long nred, int sms, bool uncut) {
  GemvShape best{};
  long long best_cost = -1;
  const long long slots = (long long)sms * 2;
  for (int G = 1, lg = 0; G <= 8; G *= 2, lg++) {
    const long long cb = (nout + 256 / G - 1) / (256 / G);
    const long long most = (nred + 8 * G - 1) / (8 * G);   // at least 8 rows per group
    for (long long ch : {slots / cb, (slots + cb - 1) / cb}) {
      if (ch > most) ch = most;
      if (ch > 1024) ch = 1024;
      if (ch < 1 || uncut) ch = 1;
      const long long rpt = ((nred + ch - 1) / ch + G - 1) / G;
      const long long waves = (cb * ch + slots - 1) / slots;
      const long long cost = waves * (rpt + 8 * lg) + 4 * ((ch + G - 1) / G + 2 * lg);
      if (best_cost < 0 || cost < best_cost) {
        best_cost = cost;
        best.G = G;
        best.grid = (int)cb;
        best.parts = (int)ch;
        best.nunits = cb;
        best.records = ch > 1 ? (size_t)ch * nout : 0;
        best.tickets = ch > 1 ? (size_t)cb : 0;
      }
    }
  }
  return best;
}

// Matrices whose rows the direct kernel reduces sooner than the streaming one (us a call, direct /
// streaming). Small ones, up to 48 MB of FP64: 1000x4195 16.1 / 20.1, 4000x1573 20.1 / 22.7, 200x20971
// 22.7 / 28.6; up to 32 MB of the others: FP32 4000x2097 21.6 / 24.6, but 4000x3145 28.2 / 26.8; FP64
// complex 4000x525 26.1 / 30.7, 4000x787 32.7 / 34.7; FP32 complex 1000x4195 26.7 / 27.7, 1000x6291
// 34.8 / 37.0. Many rows fill the streaming kernel's units: FP64 20000x64 20.6 / 11.4, FP32
// 8192x1000 23.0 / 16.5, FP64 complex 8000x131 22.6 / 14.4, but 5000x209 18.5 / 24.7. And few rows of any length, which fill
// a band of the streaming kernel (64 rows or more) badly: FP64 1x3000000 18.5 / 156, 8x8000000 121 / 391,
// 48x400000 47.5 / 51.8, FP32 16x500000 26.7 / 28.8 but 32x500000 39.0 / 35.4, FP64 complex 16x500000
// 58.7 / 94.8 but 32x500000 111 / 107, FP32 complex 48x400000 79.8 / 89.2. And FP64 complex rows from fold 6
// on, whose accumulators spill in the streaming kernel: fold 6 8192^2 479 / 551, fold 7 8192^2 528 / 707,
// 20000x500 121 / 141, fold 8 8192^2 591 / 768, 300x100000 363 / 403, but fold 8 100000x100 467 / 191.
bool gemv_rows_direct(long long nout, long long nred, int es, bool cx, int fold) {
  if (es == 16 && fold > 5 && nred >= 500) return true;
  const long long bytes = nout * nred * es;
  if (nout > 6144) return nout <= 8192 && bytes <= 8ll << 20;
  return nout <= (es == 8 ? 48 : 24) || bytes <= (es == 8 && !cx ? 48ll << 20 : 32ll << 20);
}

// Shape of the direct rows kernel: S warps to a row, enough to fill the device with at least 64
// elements to each, and `parts` CTAs to a row where rows alone leave it idle: 8 CTAs per SM in
// all (4 of FP64 complex, of which 2 are resident), each with four steps of its 8 warps or more, two
// while there are two CTAs per SM. us a call with 4 / 8 / 16 / 32 CTAs per SM (an earlier form of the
// kernel): FP64 8x8000000 164 / 153 / 162 / 172, FP32 32x500000 43.4 / 41.0 / 43.4 / 53.4, FP64 complex
// 16x500000 61.5 / 71.1 / 84.0 / 118.
// `uncut`: one part (no scratch).
GemvShape gemv_rows_direct_shape(long long nout, long long nred, int es, int sms, bool uncut) {
  GemvShape s{};
  int S = 1;
  while (S < 8 && nout * S < (long long)sms * 16 && nred >= 128 * S) S *= 2;
  s.G = S;
  s.grid = (int)((nout + 8 / S - 1) / (8 / S));
  s.parts = 1;
  if (S == 8 && !uncut) {
    const long long steps = nred / 1024;   // of a whole CTA: 4 elements a lane
    const long long most = ((long long)sms * (es == 16 ? 4 : 8) + nout - 1) / nout, once = (long long)sms * 2 / nout;
    const long long p = std::min(most, std::max(steps / 4, std::min(steps / 2, once)));
    if (p > 1 && steps - steps / p >= 6) {   // the sum of the parts takes as long as about five steps
      s.parts = (int)p;
      s.records = (size_t)nout * p;
      s.tickets = (size_t)nout;
    }
  }
  return s;
}

// Whether TMA can address every stage of the matrix: a box's coordinates are ints, in 8-byte words
// along a row (two per FP64 complex element) and in rows of a phase. A box is at most 130 words wide
// and 256 rows high, and its end is kept within int as well. Longer rows (16 GiB and more) and
// taller matrices take the direct kernels, whose addresses are 64-bit.
bool gemv_in_reach(long long Rs, long long Cs, int es, int phases) {
  constexpr long long most = (1ll << 31) - 512;
  return Cs * es / 8 + 2 <= most && Rs / phases <= most;
}

template <typename E, bool CX>
bool run_xgemv(const XGemvReq<E, CX>& q) {
  constexpr int NC = CX ? 2 : 1;
  if (q.M == 0 || q.N == 0) return true;   // r[szc]gemv.c: early return
  const int maxf = sizeof(E) == 8 ? kMaxFoldD : kMaxFoldS;
  if (q.fold < 2 || q.fold > maxf) {
    set_error(RB_ERR_INVALID_ARG, "fold must be in [2, " + std::to_string(maxf) + "]");
    return false;
  }
  const XOps<E>* o = xops_for<E, CX>(q.fold);
  if (q.M < 0 || q.N < 0 || q.lda < 1 || q.incX < 0 || q.incY < 1) {
    set_error(RB_ERR_INVALID_ARG, "gemv: negative size, lda < 1, incX < 0 or incY < 1");
    return false;
  }
  // row-major view of the stored matrix: Rs rows x Cs columns
  bool nt = xnt(q.trans);
  const bool conj = CX && !nt && !xplain_t(q.trans);
  long long Rs = q.M, Cs = q.N;
  if (!xrow(q.order)) { Rs = q.N; Cs = q.M; nt = !nt; }
  if (q.lda < Cs) { set_error(RB_ERR_INVALID_ARG, "gemv: lda smaller than the row length"); return false; }
  const long long nout = nt ? Rs : Cs, nred = nt ? Cs : Rs;
  const bool alpha_zero = q.alpha.r == E(0) && q.alpha.i == E(0);
  const long long nred_eff = alpha_zero ? 0 : nred;            // [szc]b[szc]gemv: alpha == 0
  if (q.mode == kOutBinned && nred_eff == 0) return true;       // binned form touches nothing
  if (!o) {
    // folds above the register-resident kernels: one thread per entry (rb_foldn.cu)
    EntryReq<E> e{};
    e.fold = q.fold;
    e.mode = q.mode;
    e.M = nout; e.N = 1; e.K = nred_eff;
    e.A = q.A; e.sai = nt ? q.lda : 1; e.sak = nt ? 1 : q.lda;
    e.B = q.X; e.sbk = q.incX; e.sbj = 0;
    e.ar = q.alpha.r; e.ai = q.alpha.i; e.br = q.beta.r; e.bi = q.beta.i;
    e.alpha_on_b = true;
    e.conja = conj;
    e.C = q.Y; e.sci = q.incY; e.scj = 0;
    return run_entries_n<E, CX>(e);
  }

  std::unique_lock<std::mutex> lock;
  Workspace* w = acquire_workspace(&lock);
  if (!w) return false;
  cudaStream_t s = w->stream;
  DeviceInfo di;
  if (!device_info(&di)) return false;

  const size_t es = sizeof(E) * NC;
  const size_t per_state = (size_t)2 * q.fold * es;
  const size_t a_bytes = nred_eff > 0 ? ((size_t)(Rs - 1) * q.lda + Cs) * es : 0;
  const size_t x_bytes = span(nred_eff, q.incX, es);
  const size_t y_bytes = q.mode == kOutValue ? span(nout, q.incY, es)
                                             : ((size_t)(nout - 1) * q.incY + 1) * per_state;
  // phases the rows are taken in: the fewest whose pitch is a multiple of 16 bytes, at least
  // two when A itself is misaligned (host operands are copied to aligned device memory)
  const bool a_dev = a_bytes && on_device(q.A);
  const uintptr_t a_mis = a_dev ? (uintptr_t)q.A % 16 : 0;
  int phases = 1;
  while (((size_t)phases * q.lda * es) % 16 != 0) phases *= 2;
  if (phases == 1 && a_mis != 0) phases = 2;
  // the streaming kernels want a reduction, and tensor maps that hold it
  bool streams = false;
  if (!cuda_ok(o->gemv_streams(nt, &streams), "gemv kernel attributes")) return false;
  const bool reach = streams && nred_eff > 0 && gemv_in_reach(Rs, Cs, (int)es, phases);
  const bool rows_direct = nt && (!reach || gemv_rows_direct(nout, nred_eff, (int)es, CX, q.fold));
  // (bounds: see gemv_cols_direct_kernel)
  const bool cols_direct =
      !nt && (!reach || gs::direct_cols<E, CX>(nout, nred_eff));
  GemvShape sh{};
  const auto shape = [&](bool uncut) {
    if (cols_direct) sh = gemv_cols_direct_shape(nout, nred_eff, di.sms, uncut);
    else if (rows_direct) sh = gemv_rows_direct_shape(nout, nred_eff, (int)es, di.sms, uncut);
    else sh = gemv_shape(nt, nout, nred_eff, (int)es, CX, q.fold, phases, di.sms, uncut);
  };
  shape(false);
  CutScratch cs{};
  if (sh.records && !cut_scratch(w, sh.records * NC * (2 * q.fold + 1) * sizeof(E), sh.tickets, &cs)) shape(true);
  const bool a_host = a_bytes && !a_dev, x_host = x_bytes && !on_device(q.X);
  const bool y_host = !on_device(q.Y);
  const size_t need = (a_host ? a_bytes : 0) + (x_host ? x_bytes : 0) + (y_host ? y_bytes : 0) + 3 * 256;
  if (need > 3 * 256 && !w->ensure_big(need)) return false;
  Bump b{w->big};
  bool ok = true;
  const E* dA = (const E*)to_device(q.A, a_bytes, &b, s, &ok);
  const E* dX = (const E*)to_device(q.X, x_bytes, &b, s, &ok);
  E* dY = (E*)to_device(q.Y, y_bytes, &b, s, &ok);
  if (!ok) return false;

  XGemvArgs<E> g{};
  g.R = nt ? nout : nred_eff;
  g.C = nt ? nred_eff : nout;
  g.A = dA;
  g.lda = q.lda;
  g.x = dX;
  g.incx = q.incX;
  g.ar = q.alpha.r;
  g.ai = q.alpha.i;
  g.br = q.beta.r;
  g.bi = q.beta.i;
  g.alpha_one = q.alpha.r == E(1) && q.alpha.i == E(0);
  g.conj = conj ? 1 : 0;
  g.mode = q.mode;
  g.y = q.mode == kOutValue ? dY : nullptr;
  g.ybin = q.mode == kOutBinned ? dY : nullptr;
  g.incy = q.incY;
  g.nb = (int)sh.nb;
  g.q = sh.q;
  g.rem = sh.rem;
  g.parts = sh.parts;
  g.scratch = (E*)cs.parts;
  g.tickets = sh.tickets ? cs.tickets : nullptr;
  g.status = w->dstatus();
  g.groups = sh.G;
  g.phases = phases;
  pipeline_fault(&g.stop_after, &g.wait_polls);
  GemvMaps maps{};
  const bool direct = rows_direct || cols_direct;
  if (!direct && !gemv_maps(&maps, dA, (size_t)es, Rs, Cs, q.lda, phases, nt, sh.G))
    return false;
  count_launch(sh.records && !sh.tickets ? 2 : 1);
  if (!cuda_ok(o->gemv(g, direct ? nullptr : &maps, nt, sh.grid, s), "gemv launch")) return false;
  if (y_host) {
    int* hs = w->hstatus();
    if (!cuda_ok(cudaMemcpyAsync(q.Y, dY, y_bytes, cudaMemcpyDeviceToHost, s), "copy y") ||
        !cuda_ok(cudaMemcpyAsync(hs, w->dstatus(), 4, cudaMemcpyDeviceToHost, s), "copy status") ||
        !cuda_ok(cudaStreamSynchronize(s), "cudaStreamSynchronize"))
      return false;
    if (*hs != 0) {
      w->reset_after_abort();
      set_error(RB_ERR_CUDA, "gemv: a pipeline wait timed out (affected entries are NaN)");
      return false;
    }
  }
  return true;
}

template <typename E, bool CX>
struct XGemmReq {
  int fold;
  char order, ta, tb;
  int M, N, K;
  Scalar<E, CX> alpha;
  const void* A;
  int lda;
  const void* B;
  int ldb;
  Scalar<E, CX> beta;
  void* C;          // values or binned states
  int ldc;
  int mode;
};

template <typename E, bool CX>
bool run_xgemm(const XGemmReq<E, CX>& q) {
  constexpr int NC = CX ? 2 : 1;
  if (q.M == 0 || q.N == 0) return true;   // r[szc]gemm.c: early return
  const int maxf = sizeof(E) == 8 ? kMaxFoldD : kMaxFoldS;
  if (q.fold < 2 || q.fold > maxf) {
    set_error(RB_ERR_INVALID_ARG, "fold must be in [2, " + std::to_string(maxf) + "]");
    return false;
  }
  const XOps<E>* o = xops_for<E, CX>(q.fold);
  if (q.M < 0 || q.N < 0 || q.K < 0 || q.lda < 1 || q.ldb < 1 || q.ldc < 1) {
    set_error(RB_ERR_INVALID_ARG, "gemm: negative size or leading dimension < 1");
    return false;
  }
  const bool row = xrow(q.order), ta = !xnt(q.ta), tb = !xnt(q.tb);
  XGemmArgs<E> g{};
  g.M = q.M;
  g.N = q.N;
  const bool alpha_zero = q.alpha.r == E(0) && q.alpha.i == E(0);
  g.K = alpha_zero ? 0 : q.K;   // [szc]b[szc]gemm: alpha == 0 deposits nothing
  if (row) {
    g.sai = ta ? 1 : q.lda;  g.sak = ta ? q.lda : 1;
    g.sbk = tb ? 1 : q.ldb;  g.sbj = tb ? q.ldb : 1;
    g.sci = q.ldc;           g.scj = 1;
  } else {
    g.sai = ta ? q.lda : 1;  g.sak = ta ? 1 : q.lda;
    g.sbk = tb ? q.ldb : 1;  g.sbj = tb ? 1 : q.ldb;
    g.sci = 1;               g.scj = q.ldc;
  }
  g.ar = q.alpha.r;
  g.ai = q.alpha.i;
  g.br = q.beta.r;
  g.bi = q.beta.i;
  g.alpha_one = q.alpha.r == E(1) && q.alpha.i == E(0);
  g.conja = (CX && ta && !xplain_t(q.ta)) ? 1 : 0;
  g.conjb = (CX && tb && !xplain_t(q.tb)) ? 1 : 0;
  g.mode = q.mode;
  if (q.mode == kOutBinned && g.K == 0) return true;   // binned form touches nothing
  if (!o) {
    // folds above the register-resident kernels: one thread per entry (rb_foldn.cu)
    EntryReq<E> e{};
    e.fold = q.fold;
    e.mode = q.mode;
    e.M = g.M; e.N = g.N; e.K = g.K;
    e.A = q.A; e.sai = g.sai; e.sak = g.sak;
    e.B = q.B; e.sbk = g.sbk; e.sbj = g.sbj;
    e.ar = g.ar; e.ai = g.ai; e.br = g.br; e.bi = g.bi;
    e.conja = g.conja != 0;
    e.conjb = g.conjb != 0;
    e.C = q.C; e.sci = g.sci; e.scj = g.scj;
    return run_entries_n<E, CX>(e);
  }

  std::unique_lock<std::mutex> lock;
  Workspace* w = acquire_workspace(&lock);
  if (!w) return false;
  cudaStream_t s = w->stream;
  const size_t es = sizeof(E) * NC;
  const size_t per = q.mode == kOutValue ? es : (size_t)2 * q.fold * es;
  const size_t a_bytes = g.K ? ((size_t)(g.M - 1) * g.sai + (size_t)(g.K - 1) * g.sak + 1) * es : 0;
  const size_t b_bytes = g.K ? ((size_t)(g.K - 1) * g.sbk + (size_t)(g.N - 1) * g.sbj + 1) * es : 0;
  const size_t c_bytes = ((size_t)(g.M - 1) * g.sci + (size_t)(g.N - 1) * g.scj + 1) * per;
  const bool a_host = a_bytes && !on_device(q.A), b_host = b_bytes && !on_device(q.B);
  const bool c_host = !on_device(q.C);
  const size_t need = (a_host ? a_bytes : 0) + (b_host ? b_bytes : 0) + (c_host ? c_bytes : 0) + 3 * 256;
  if (need > 3 * 256 && !w->ensure_big(need)) return false;
  Bump bm{w->big};
  bool ok = true;
  g.A = (const E*)to_device(q.A, a_bytes, &bm, s, &ok);
  g.B = (const E*)to_device(q.B, b_bytes, &bm, s, &ok);
  E* dC = (E*)to_device(q.C, c_bytes, &bm, s, &ok);
  if (!ok) return false;
  g.C = q.mode == kOutValue ? dC : nullptr;
  g.Cbin = q.mode == kOutBinned ? dC : nullptr;
  GemmPlan plan;
  if (!gemm_decompose(o->gemm_plan, w, g.M, g.N, g.K, &plan)) return false;
  count_launch();
  if (!cuda_ok(o->gemm(g, plan, s), "gemm launch")) return false;
  if (c_host) {
    if (!cuda_ok(cudaMemcpyAsync(q.C, dC, c_bytes, cudaMemcpyDeviceToHost, s), "copy C") ||
        !cuda_ok(cudaStreamSynchronize(s), "cudaStreamSynchronize"))
      return false;
  }
  return true;
}

template <typename E, bool CX, typename S>
void gemv_entry(int fold, char Order, char TransA, int M, int N, S alpha, const void* A, int lda,
                const void* X, int incX, S beta, void* Y, int incY, int mode) {
  XGemvReq<E, CX> q{fold, Order, TransA, M, N, read_scalar<E, CX>(alpha), A, lda, X, incX,
                    read_scalar<E, CX>(beta), Y, incY, mode};
  run_xgemv<E, CX>(q);
}

template <typename E, bool CX, typename S>
void gemm_entry(int fold, char Order, char TransA, char TransB, int M, int N, int K, S alpha,
                const void* A, int lda, const void* B, int ldb, S beta, void* C, int ldc,
                int mode) {
  XGemmReq<E, CX> q{fold, Order, TransA, TransB, M, N, K, read_scalar<E, CX>(alpha), A, lda, B,
                    ldb, read_scalar<E, CX>(beta), C, ldc, mode};
  run_xgemm<E, CX>(q);
}

// beta of the binned forms: 1 (merge into the caller's states; unused in that mode)
template <typename E, bool CX>
const void* one_scalar() {
  static const E one[2] = {E(1), E(0)};
  return one;
}

}  // namespace
}  // namespace rb

extern "C" {

// ---- FP64 real -------------------------------------------------------------------------------
void reproBLAS_rdgemv(const int fold, const char Order, const char TransA, const int M,
                      const int N, const double alpha, const double* A, const int lda,
                      const double* X, const int incX, const double beta, double* Y,
                      const int incY) {
  rb::gemv_entry<double, false, double>(fold, Order, TransA, M, N, alpha, A, lda, X, incX, beta, Y,
                                        incY, rb::kOutValue);
}
void reproBLAS_dgemv(const char Order, const char TransA, const int M, const int N,
                     const double alpha, const double* A, const int lda, const double* X,
                     const int incX, const double beta, double* Y, const int incY) {
  reproBLAS_rdgemv(3, Order, TransA, M, N, alpha, A, lda, X, incX, beta, Y, incY);
}
void binnedBLAS_dbdgemv(const int fold, const char Order, const char TransA, const int M,
                        const int N, const double alpha, const double* A, const int lda,
                        const double* X, const int incX, double_binned* Y, const int incY) {
  rb::gemv_entry<double, false, double>(fold, Order, TransA, M, N, alpha, A, lda, X, incX, 1.0, Y,
                                        incY, rb::kOutBinned);
}
void reproBLAS_rdgemm(const int fold, const char Order, const char TransA, const char TransB,
                      const int M, const int N, const int K, const double alpha, const double* A,
                      const int lda, const double* B, const int ldb, const double beta,
                      double* C, const int ldc) {
  rb::gemm_entry<double, false, double>(fold, Order, TransA, TransB, M, N, K, alpha, A, lda, B, ldb,
                                        beta, C, ldc, rb::kOutValue);
}
void reproBLAS_dgemm(const char Order, const char TransA, const char TransB, const int M,
                     const int N, const int K, const double alpha, const double* A,
                     const int lda, const double* B, const int ldb, const double beta,
                     double* C, const int ldc) {
  reproBLAS_rdgemm(3, Order, TransA, TransB, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
}
void binnedBLAS_dbdgemm(const int fold, const char Order, const char TransA, const char TransB,
                        const int M, const int N, const int K, const double alpha,
                        const double* A, const int lda, const double* B, const int ldb,
                        double_binned* C, const int ldc) {
  rb::gemm_entry<double, false, double>(fold, Order, TransA, TransB, M, N, K, alpha, A, lda, B, ldb,
                                        1.0, C, ldc, rb::kOutBinned);
}

// ---- FP32 real -------------------------------------------------------------------------------
void reproBLAS_rsgemv(const int fold, const char Order, const char TransA, const int M,
                      const int N, const float alpha, const float* A, const int lda,
                      const float* X, const int incX, const float beta, float* Y,
                      const int incY) {
  rb::gemv_entry<float, false, float>(fold, Order, TransA, M, N, alpha, A, lda, X, incX, beta, Y,
                                      incY, rb::kOutValue);
}
void reproBLAS_sgemv(const char Order, const char TransA, const int M, const int N,
                     const float alpha, const float* A, const int lda, const float* X,
                     const int incX, const float beta, float* Y, const int incY) {
  reproBLAS_rsgemv(3, Order, TransA, M, N, alpha, A, lda, X, incX, beta, Y, incY);
}
void binnedBLAS_sbsgemv(const int fold, const char Order, const char TransA, const int M,
                        const int N, const float alpha, const float* A, const int lda,
                        const float* X, const int incX, float_binned* Y, const int incY) {
  rb::gemv_entry<float, false, float>(fold, Order, TransA, M, N, alpha, A, lda, X, incX, 1.0f, Y,
                                      incY, rb::kOutBinned);
}
void reproBLAS_rsgemm(const int fold, const char Order, const char TransA, const char TransB,
                      const int M, const int N, const int K, const float alpha, const float* A,
                      const int lda, const float* B, const int ldb, const float beta, float* C,
                      const int ldc) {
  rb::gemm_entry<float, false, float>(fold, Order, TransA, TransB, M, N, K, alpha, A, lda, B, ldb,
                                      beta, C, ldc, rb::kOutValue);
}
void reproBLAS_sgemm(const char Order, const char TransA, const char TransB, const int M,
                     const int N, const int K, const float alpha, const float* A, const int lda,
                     const float* B, const int ldb, const float beta, float* C, const int ldc) {
  reproBLAS_rsgemm(3, Order, TransA, TransB, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
}
void binnedBLAS_sbsgemm(const int fold, const char Order, const char TransA, const char TransB,
                        const int M, const int N, const int K, const float alpha, const float* A,
                        const int lda, const float* B, const int ldb, float_binned* C,
                        const int ldc) {
  rb::gemm_entry<float, false, float>(fold, Order, TransA, TransB, M, N, K, alpha, A, lda, B, ldb,
                                      1.0f, C, ldc, rb::kOutBinned);
}

// ---- FP64 complex ------------------------------------------------------------------------------
void reproBLAS_rzgemv(const int fold, const char Order, const char TransA, const int M,
                      const int N, const void* alpha, const void* A, const int lda,
                      const void* X, const int incX, const void* beta, void* Y, const int incY) {
  rb::gemv_entry<double, true, const void*>(fold, Order, TransA, M, N, alpha, A, lda, X, incX,
                                            beta, Y, incY, rb::kOutValue);
}
void reproBLAS_zgemv(const char Order, const char TransA, const int M, const int N,
                     const void* alpha, const void* A, const int lda, const void* X,
                     const int incX, const void* beta, void* Y, const int incY) {
  reproBLAS_rzgemv(3, Order, TransA, M, N, alpha, A, lda, X, incX, beta, Y, incY);
}
void binnedBLAS_zbzgemv(const int fold, const char Order, const char TransA, const int M,
                        const int N, const void* alpha, const void* A, const int lda,
                        const void* X, const int incX, double_complex_binned* Y,
                        const int incY) {
  rb::gemv_entry<double, true, const void*>(fold, Order, TransA, M, N, alpha, A, lda, X, incX,
                                            rb::one_scalar<double, true>(), Y, incY,
                                            rb::kOutBinned);
}
void reproBLAS_rzgemm(const int fold, const char Order, const char TransA, const char TransB,
                      const int M, const int N, const int K, const void* alpha, const void* A,
                      const int lda, const void* B, const int ldb, const void* beta, void* C,
                      const int ldc) {
  rb::gemm_entry<double, true, const void*>(fold, Order, TransA, TransB, M, N, K, alpha, A, lda,
                                            B, ldb, beta, C, ldc, rb::kOutValue);
}
void reproBLAS_zgemm(const char Order, const char TransA, const char TransB, const int M,
                     const int N, const int K, const void* alpha, const void* A, const int lda,
                     const void* B, const int ldb, const void* beta, void* C, const int ldc) {
  reproBLAS_rzgemm(3, Order, TransA, TransB, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
}
void binnedBLAS_zbzgemm(const int fold, const char Order, const char TransA, const char TransB,
                        const int M, const int N, const int K, const void* alpha, const void* A,
                        const int lda, const void* B, const int ldb, double_complex_binned* C,
                        const int ldc) {
  rb::gemm_entry<double, true, const void*>(fold, Order, TransA, TransB, M, N, K, alpha, A, lda,
                                            B, ldb, rb::one_scalar<double, true>(), C, ldc,
                                            rb::kOutBinned);
}

// ---- FP32 complex ------------------------------------------------------------------------------
void reproBLAS_rcgemv(const int fold, const char Order, const char TransA, const int M,
                      const int N, const void* alpha, const void* A, const int lda,
                      const void* X, const int incX, const void* beta, void* Y, const int incY) {
  rb::gemv_entry<float, true, const void*>(fold, Order, TransA, M, N, alpha, A, lda, X, incX,
                                           beta, Y, incY, rb::kOutValue);
}
void reproBLAS_cgemv(const char Order, const char TransA, const int M, const int N,
                     const void* alpha, const void* A, const int lda, const void* X,
                     const int incX, const void* beta, void* Y, const int incY) {
  reproBLAS_rcgemv(3, Order, TransA, M, N, alpha, A, lda, X, incX, beta, Y, incY);
}
void binnedBLAS_cbcgemv(const int fold, const char Order, const char TransA, const int M,
                        const int N, const void* alpha, const void* A, const int lda,
                        const void* X, const int incX, float_complex_binned* Y, const int incY) {
  rb::gemv_entry<float, true, const void*>(fold, Order, TransA, M, N, alpha, A, lda, X, incX,
                                           rb::one_scalar<float, true>(), Y, incY,
                                           rb::kOutBinned);
}
void reproBLAS_rcgemm(const int fold, const char Order, const char TransA, const char TransB,
                      const int M, const int N, const int K, const void* alpha, const void* A,
                      const int lda, const void* B, const int ldb, const void* beta, void* C,
                      const int ldc) {
  rb::gemm_entry<float, true, const void*>(fold, Order, TransA, TransB, M, N, K, alpha, A, lda,
                                           B, ldb, beta, C, ldc, rb::kOutValue);
}
void reproBLAS_cgemm(const char Order, const char TransA, const char TransB, const int M,
                     const int N, const int K, const void* alpha, const void* A, const int lda,
                     const void* B, const int ldb, const void* beta, void* C, const int ldc) {
  reproBLAS_rcgemm(3, Order, TransA, TransB, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
}
void binnedBLAS_cbcgemm(const int fold, const char Order, const char TransA, const char TransB,
                        const int M, const int N, const int K, const void* alpha, const void* A,
                        const int lda, const void* B, const int ldb, float_complex_binned* C,
                        const int ldc) {
  rb::gemm_entry<float, true, const void*>(fold, Order, TransA, TransB, M, N, K, alpha, A, lda,
                                           B, ldb, rb::one_scalar<float, true>(), C, ldc,
                                           rb::kOutBinned);
}

}  // extern "C"
