// rb_gemv_stream.cuh -- binned gemv of every element type (FP64 / FP32, real and complex): A
// streams through a ring of shared-memory stages filled by bulk copies, so the bytes in
// flight per SM are set by the ring's size rather than by the consumers' registers.
//
//   y_i <- conv( binned(beta*y_i) + sum_j products of op(A)_ij and bx_j ),  bx_j = fl(alpha*x_j)
// (src/reproBLAS/r[dszc]gemv.c, src/binnedBLAS/[dszc]b[dszc]gemv.ccog; the deposited values are
// listed in rb_entry.cuh). A is row-major R x C (leading dimension lda); the rows kernel
// reduces along rows (R outputs), the columns kernel along columns (C outputs).
//
// What bounds it: HBM (A is read once), as long as the deposits keep up. One SM receives a
// 64 KB stage in ~1.5 us = 2900 cycles, in which each of its four sub-partitions has 128 rows
// of 128 bytes to deposit; a fold-3 FP64 element costs ~25 issue cycles, an FP32 one ~14, so
// real types need 50-60 % of the stage's time and complex types, with four deposits per
// element, about all of it. Per-element checks are therefore left out as in the gemm tile
// (rb_gemm_tile.cuh): per stage a thread bounds its products by max|A| * max|bx| and deposits
// them unchecked when the bound stays below its accumulator's cap.
//
// CTA = 16 consumer warps, a copy warp and an x warp, one CTA per SM, each streaming an equal
// share of A's stages. Every consumer thread owns whole outputs (a row of a band, or a column
// of a block). A stage is brought in by TMA box loads. TMA wants 16-byte aligned rows, which
// an odd leading dimension does not give, so the rows are taken in NPH phases (1, 2 or 4):
// phase h holds rows h, h + NPH, ..., whose pitch NPH*lda is a multiple of 16 bytes, behind a
// tensor map of its own that starts at the 16-byte boundary at or before row h. A row then
// lands `shift` bytes (0 to 15, its phase's distance from that boundary) into its slot; slots
// are 16 bytes longer than a row's elements, which also keeps a thread-per-row access free of
// bank conflicts. Any leading dimension and alignment streams at the same rate (row-by-row
// cp.async.bulk copies did not: ~80 issue cycles each, 82 us against 40 at 4096^2). The x
// warp reads x at any stride, forms fl(alpha*x) and the stage's largest key. Every wait is
// bounded: a wait that gives up sets the CTA's abort flag, the affected entries come out NaN
// (their states get the NaN class), *status is set to 2, and the copy warp lets its copies
// in flight land (bounded) before the CTA exits.
#pragma once
#include "rb_entry.cuh"
#include "rb_gemm_tile.cuh"
#include "rb_ptx.cuh"

namespace rb {
namespace gs {

using xb::Val;

constexpr int kConsumers = 512;                 // 16 consumer warps
constexpr int kStages = 3;
// FP64 complex consumers need 97-104 registers (without them fold 3 spilled: 297 us at 8192^2,
// 266 with, rows kernel); 18 warps leave each thread 96. Their CTA therefore
// has a whole warpgroup of producers (two warps of it idle), launches at 96 registers a thread
// and moves 32 from each producer to the four consumer warpgroups: 512 * 104 + 128 * 64 =
// 640 * 96, all that the launch owns (gemv_streams checks that it was built so).
template <typename E, bool CX>
__host__ __device__ constexpr bool moves_regs() { return CX && sizeof(E) == 8; }
template <typename E, bool CX>
__host__ __device__ constexpr int threads() { return kConsumers + (moves_regs<E, CX>() ? 128 : 64); }
constexpr int kMoveLaunch = 96, kMoveConsumer = 104, kMoveProducer = 64;
static_assert(kConsumers * kMoveConsumer + 128 * kMoveProducer <= (kConsumers + 128) * kMoveLaunch,
              "registers moved must be registers launched with");
constexpr uint32_t kThreadBytes = 128;          // of A per consumer thread and stage

// The 512 consumer threads own P = 512/G outputs (G = g.groups in {2, 4, 8}, chosen by the
// host), G threads each: lane l of a warp is group l / (32/G) of the warp's output l mod
// (32/G). Units are bands of P rows (rows kernel) or blocks of P columns (columns kernel); a
// stage covers SC = PE*G elements of the reduction, PE = 128 bytes / element. Rows kernel:
// group q deposits columns q*PE .. q*PE + PE - 1 of the stage; columns kernel: rows q, q + G,
// q + 2G, ... (so that a thread's rows belong to one phase). At the end of a unit's run the G partial states of an output
// meet by shuffles within their warp: no warp waits for another from the first stage to the
// finished entries. A larger G makes units narrower, hence more of them, and fewer CTAs share
// a unit, which shortens the merge of the cut units' parts.
// Bytes per row slot of a stage in phases (shifted rows): 16 more than the row's elements. A stage
// of unshifted rows (one phase) has no slack -- boxes wider than their rows cost bandwidth (2 %
// per 16 bytes at 528, 11 % for 64 bytes at 1088): the rows kernel takes G boxes of 128 bytes x P
// rows with the 128-byte swizzle (16-byte chunk c of box row r sits at c ^ (r & 7), so lanes on
// neighbouring rows read different banks), the columns kernel one box, whose groups' reads
// conflict on banks (2-way for 8-byte elements, 4-way for 4-byte ones) within what the
// shared memory has to spare.
template <bool ROWS>
__host__ __device__ constexpr uint32_t slot_bytes(int G, int es, int phases) {
  return (ROWS ? kThreadBytes * (uint32_t)G : (uint32_t)(kConsumers / G) * (uint32_t)es) + (phases > 1 ? 16u : 0u);
}
constexpr uint32_t kStageA = kConsumers * kThreadBytes + 4096;   // rows in slots (at most 256 rows)
constexpr uint32_t kStageX = 1024;                               // PE*G elements of bx
constexpr uint32_t kStageBytes = kStageA + kStageX;              // a multiple of 1024
constexpr size_t kSmemBytes = (size_t)kStages * kStageBytes + 1024;
static_assert(kSmemBytes + 256 <= 227 * 1024, "shared memory of the gemv kernel");

// Work split. The stages are numbered unit-major, x = u * nb + j (unit u = band of rows or
// block of columns; j = its j-th stage), and every CTA streams a contiguous range of them: with
// `parts` = 0, q or q + 1 stages each, whatever the shape; with parts = p > 0, the p-th part of a
// unit (p > 1) or q whole units (p = 1), so that a CTA has one run, or no unit is cut. A unit
// whose stages all fall in one CTA is finished there; a unit cut between CTAs leaves one
// partial state per CTA, and the last of those CTAs to finish (ticket) merges them.
struct Split {
  int q, rem, parts, nb, x0, x1;
  template <typename E>
  __device__ __forceinline__ explicit Split(const XGemvArgs<E>& g)
      : q(g.q), rem(g.rem), parts(g.parts), nb(g.nb) {
    x0 = start((int)blockIdx.x);
    x1 = start((int)blockIdx.x + 1);
  }
  __device__ __forceinline__ int start(int b) const {
    if (parts == 0) return b * q + (b < rem ? b : rem);
    if (parts == 1) return (b * q < rem ? b * q : rem) * nb;   // rem: units in all
    return b / parts * nb + (int)((long long)(b % parts) * nb / parts);
  }
  // CTA whose range holds stage x
  __device__ __forceinline__ int owner(int x) const {
    if (parts == 0) {
      const int big = rem * (q + 1);
      return x < big ? x / (q + 1) : rem + (x - big) / q;
    }
    const int u = x / nb;
    if (parts == 1) return u / q;
    return u * parts + (int)(((long long)(x - u * nb + 1) * parts - 1) / nb);
  }
};

// Ring position: stage index and the parity of its current phase.
struct Ring {
  int st = 0;
  unsigned ph = 0;
  __device__ __forceinline__ void next() {
    if (++st == kStages) { st = 0; ph ^= 1u; }
  }
};

// Geometry of a launch, the same for every role.
template <typename E, bool CX, bool ROWS>
struct Geom {
  static constexpr int NC = CX ? 2 : 1;
  static constexpr int ES = NC * (int)sizeof(E);          // bytes per element
  static constexpr int PE = (int)kThreadBytes / ES;       // elements per thread and stage
  int G, lgG, P, lgP, SC; // SC = PE*G elements of the reduction per stage
  int lgN;                // log2 of the phases
  uint32_t pitch;         // bytes per row slot
  uint32_t phase_bytes;   // of one phase's slots in a stage
  long long nout, nred;
  __device__ __forceinline__ explicit Geom(const XGemvArgs<E>& g) {
    G = g.groups;
    lgG = __ffs(G) - 1;
    P = kConsumers >> lgG;
    lgP = __ffs(kConsumers) - 1 - lgG;
    SC = PE << lgG;
    lgN = __ffs(g.phases) - 1;
    pitch = slot_bytes<ROWS>(G, ES, g.phases);
    phase_bytes = ((uint32_t)(ROWS ? P : SC) >> lgN) * pitch;
    nout = ROWS ? g.R : g.C;
    nred = ROWS ? g.C : g.R;
  }
};

// mbarriers and small words shared by the roles
struct Sync {
  unsigned long long full[kStages];     // A of the stage has landed
  unsigned long long xfull[kStages];    // bx of the stage is written
  unsigned long long empty[kStages];    // the consumers are done with the stage
  unsigned xkey[kStages];
  int abort_flag;
};

// Copy warp (its lane 0): the boxes of each stage, all completing on the stage's `full` mbarrier.
// Rows and columns outside A are zero-filled. Before returning it waits (bounded) until every
// copy it issued has landed, so that none is still writing shared memory when the CTA exits.
template <typename E, bool CX, bool ROWS>
__device__ __forceinline__ void copy_stages(const XGemvArgs<E>& g, const Geom<E, CX, ROWS>& m,
                                            const GemvMaps& maps, const Split& sp, unsigned char* ring,
                                            Sync& sy) {
  using Gm = Geom<E, CX, ROWS>;
  const int nph = 1 << m.lgN;
  const int boxes = ROWS && nph == 1 ? m.G : nph;
  const uint32_t box_bytes = ROWS && nph == 1 ? (uint32_t)m.P * kThreadBytes : m.phase_bytes;
  Ring r;
  int u = sp.x0 / g.nb, j = sp.x0 - u * g.nb;
  long long issued = 0;
  for (int x = sp.x0; x < sp.x1; x++, issued++) {
    if (g.stop_after >= 0 && issued >= g.stop_after) break;   // test hook: stop feeding the ring
    if (issued >= kStages && !mbar_wait_bounded(smem_u32(&sy.empty[r.st]), r.ph ^ 1u)) {
      atomicExch(&sy.abort_flag, 1);
      break;
    }
    if (*(volatile int*)&sy.abort_flag) break;
    const uint32_t fb = smem_u32(&sy.full[r.st]);
    mbar_expect_tx(fb, (uint32_t)boxes * box_bytes);
    const uint32_t dst = smem_u32(ring + (size_t)r.st * kStageBytes);
    // coordinates in 8-byte words (a multiple of 16 bytes) and rows of the phase
    const int c = (int)((ROWS ? (long long)j * m.SC : (long long)u * m.P) * Gm::ES / 8);
    const int row = (int)((ROWS ? (long long)u * m.P : (long long)j * m.SC) >> m.lgN);
    for (int h = 0; h < boxes; h++)
      tma_load_2d(dst + (uint32_t)h * box_bytes, &maps.m[nph == 1 ? 0 : h],
                  ROWS && nph == 1 ? c + h * (int)(kThreadBytes / 8) : c, row, fb);
    r.next();
    if (++j == g.nb) { j = 0; u++; }
  }
  // the last phase of each slot it used belongs to one of the last kStages stages it issued
  const long long first = issued > kStages ? issued - kStages : 0;
  for (long long k = first; k < issued; k++)
    mbar_wait_bounded(smem_u32(&sy.full[k % kStages]), (unsigned)((k / kStages) & 1));
}

// x warp: bx = fl(alpha*x) of each stage and its largest key, into the stage's x area; one
// arrival on the stage's `xfull` mbarrier.
template <typename E, bool CX, bool ROWS>
__device__ __forceinline__ void scale_stages(const XGemvArgs<E>& g, const Geom<E, CX, ROWS>& m,
                                             const Split& sp, unsigned char* ring, Sync& sy) {
  constexpr int NC = Geom<E, CX, ROWS>::NC;
  const int lane = threadIdx.x & 31;
  Ring r;
  int j = sp.x0 % g.nb;
  for (int x = sp.x0; x < sp.x1; x++) {
    bool go = x - sp.x0 < kStages || mbar_wait_bounded(smem_u32(&sy.empty[r.st]), r.ph ^ 1u);
    if (!go) atomicExch(&sy.abort_flag, 1);
    go = go && *(volatile int*)&sy.abort_flag == 0;
    if (!__all_sync(0xffffffffu, go)) break;
    E* xs = (E*)(ring + (size_t)r.st * kStageBytes + kStageA);
    unsigned key = 0;
    for (int i = lane; i < m.SC; i += 32) {
      const long long e = (long long)j * m.SC + i;
      Val<E, CX> v{E(0), E(0)};
      if (e < m.nred) {
        v = xb::ldv<E, CX>(g.x, e * g.incx);
        if (!g.alpha_one) v = xb::scale<E, CX>(v, g.ar, g.ai);
      }
      // in the order the groups read it (columns kernel: element e of group q is row e*G + q)
      const int pos = ROWS ? i : (i & (m.G - 1)) * Geom<E, CX, ROWS>::PE + (i >> m.lgG);
      xs[pos * NC] = v.r;
      unsigned k = BT<E>::key(v.r);
      if constexpr (CX) {
        xs[pos * NC + 1] = v.i;
        const unsigned ki = BT<E>::key(v.i);
        k = ki > k ? ki : k;
      }
      key = k > key ? k : key;
    }
    key = __reduce_max_sync(0xffffffffu, key);
    if (lane == 0) sy.xkey[r.st] = key;
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&sy.xfull[r.st]));
    r.next();
    if (++j == g.nb) j = 0;
  }
}

// Consumer side of one stage: wait for its A and x (unless aborted); false when the data is
// not there (abort), in which case the caller skips its deposits.
__device__ __forceinline__ bool stage_ready(Sync& sy, const Ring& r, long long polls) {
  if (*(volatile int*)&sy.abort_flag) return false;
  if (!mbar_wait_bounded(smem_u32(&sy.full[r.st]), r.ph, polls) ||
      !mbar_wait_bounded(smem_u32(&sy.xfull[r.st]), r.ph, polls)) {
    atomicExch(&sy.abort_flag, 1);
    return false;
  }
  return true;
}

// The PE elements of this thread in one stage, and their deposit into its accumulators.
template <typename E, bool CX, int F, bool ROWS>
struct Consumer {
  using Gm = Geom<E, CX, ROWS>;
  using B = BT<E>;
  static constexpr int NC = Gm::NC, PE = Gm::PE, ES = Gm::ES, D = CX ? 2 : 1;
  // a stage's elements are taken in STEPS steps of PS: FP64 complex would spill with all 128
  // bytes in registers
  static constexpr int STEPS = (CX && sizeof(E) == 8) ? 2 : 1;
  static constexpr int PS = PE / STEPS, ND = PS * D;
  static constexpr int NR = PS * NC;   // reals per thread and step

  Acc<E, F> a[NC];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int c = 0; c < NC; c++) a[c].zero();
  }

  // Where this thread's elements are in a stage: element e at base + e*stride + shift; or, rows
  // kernel with unshifted rows (vec), in 16-byte chunks c at base + ((c ^ swz) << 4).
  struct Place {
    uint32_t stride, shift, swz;
    bool vec;
  };

  // the elements of step h
  __device__ __forceinline__ void load(const unsigned char* base, const Place& pl, int h, E (&v)[NR]) const {
    if (pl.vec) {
      if constexpr (ROWS) {
        constexpr int PER = 16 / (int)sizeof(E), CH = NR / PER;
#pragma unroll
        for (int c = 0; c < CH; c++) {
          E t[PER];
          gt::lds_vec<E, PER>((const E*)(base + (((uint32_t)(h * CH + c) ^ pl.swz) << 4)), t);
#pragma unroll
          for (int i = 0; i < PER; i++) v[c * PER + i] = t[i];
        }
      } else {
        const unsigned char* p = base + (uint32_t)(h * PS) * pl.stride;
#pragma unroll
        for (int e = 0; e < PS; e++) {
          E t[NC];
          gt::lds_vec<E, NC>((const E*)(p + (uint32_t)e * pl.stride), t);
#pragma unroll
          for (int c = 0; c < NC; c++) v[e * NC + c] = t[c];
        }
      }
    } else {
      const uint32_t stride = ROWS ? (uint32_t)ES : pl.stride;
      const unsigned char* p = base + pl.shift + (uint32_t)(h * PS) * stride;
#pragma unroll
      for (int e = 0; e < PS; e++)
#pragma unroll
        for (int c = 0; c < NC; c++) v[e * NC + c] = ((const E*)(p + (uint32_t)e * stride))[c];
    }
  }
  // real i of element e, the same way
  __device__ __forceinline__ static const E* at(const unsigned char* base, const Place& pl, int e) {
    const uint32_t o = (uint32_t)e * pl.stride;
    return (const E*)(base + (ROWS && pl.vec ? o ^ (pl.swz << 4) : o + pl.shift));
  }

  // the D products of component c of (ar, ai) * (xr, xi)
  static __device__ __forceinline__ void prods(const E* av, const E* xv, int c, E (&p)[D]) {
    if constexpr (CX) {
      p[0] = c == 0 ? B::mul(av[0], xv[0]) : B::mul(av[0], xv[1]);
      p[1] = c == 0 ? B::mul(-av[1], xv[1]) : B::mul(av[1], xv[0]);
    } else {
      p[0] = B::mul(av[0], xv[0]);
    }
  }

  // one by one: elements [e0, e1), with every check (Acc::tile)
  __device__ __forceinline__ void deposit_careful(const unsigned char* base, const Place& pl, const E* xs,
                                                  int e0, int e1, bool conj) {
#pragma unroll 1
    for (int e = e0; e < e1; e++) {
      const E* p = at(base, pl, e);
      E av[NC], xv[NC];
#pragma unroll
      for (int c = 0; c < NC; c++) {
        av[c] = p[c];
        xv[c] = xs[e * NC + c];
      }
      if (CX && conj) av[NC - 1] = -av[NC - 1];
#pragma unroll
      for (int c = 0; c < NC; c++) {
        E v[D];
        prods(av, xv, c, v);
        a[c].template tile<D>(v, D);
      }
    }
  }

  __device__ __forceinline__ void stage(const unsigned char* base, const Place& pl, const E* xs,
                                        unsigned xkey, int nval, bool conj) {
    if constexpr (STEPS > 1) {
      if (nval < PE) {
        if (nval > 0) deposit_careful(base, pl, xs, 0, nval, conj);
        return;
      }
#pragma unroll 1
      for (int h = 0; h < STEPS; h++) step(base, pl, h, xs + h * NR, xs, xkey, conj);
      return;
    }
    if (nval <= 0) return;
    bool careful = nval < PE;
    E v[NR];
    if (!careful) {
      load(base, pl, 0, v);
      float m = 0.0f;
#pragma unroll
      for (int i = 0; i < NR; i += 2) m = max_abs3(m, key_word(v[i]), key_word(v[i + 1]));
      const unsigned bound =
          B::key(B::mul(key_ceiling<E>(__float_as_uint(m)), key_ceiling<E>(xkey)));
      bool fast = true;
#pragma unroll
      for (int c = 0; c < NC; c++) fast = fast && a[c].fast(bound, ND);
      if (CX && conj) {
#pragma unroll
        for (int e = 0; e < PE; e++) v[e * NC + NC - 1] = -v[e * NC + NC - 1];
      }
      if (fast) {
#pragma unroll
        for (int c = 0; c < NC; c++) a[c].deposits += ND;
      } else if (bound >= B::kInfKey) {
        careful = true;
      } else {
        // the exact largest key of each component's products, then the index that needs
        unsigned mk[NC];
#pragma unroll
        for (int c = 0; c < NC; c++) mk[c] = 0u;
#pragma unroll
        for (int e = 0; e < PE; e++)
#pragma unroll
          for (int c = 0; c < NC; c++) {
            E p[D], xv[NC];
#pragma unroll
            for (int q = 0; q < NC; q++) xv[q] = xs[e * NC + q];
            prods(v + e * NC, xv, c, p);
#pragma unroll
            for (int d = 0; d < D; d++) {
              const unsigned kk = B::key(p[d]);
              mk[c] = kk > mk[c] ? kk : mk[c];
            }
          }
#pragma unroll
        for (int c = 0; c < NC; c++) {
          a[c].prepare(mk[c], ND);
          if (a[c].idx == 0) careful = true;
        }
      }
    }
    if (careful) {
      deposit_careful(base, pl, xs, 0, nval, conj);
      return;
    }
#pragma unroll
    for (int e = 0; e < PE; e += 16 / ES) {
      constexpr int XR = 16 / (int)sizeof(E);   // reals of one 16-byte vector of bx
      E xv[XR];
      gt::lds_vec<E, XR>(xs + e * NC, xv);
#pragma unroll
      for (int q = 0; q < 16 / ES; q++)
#pragma unroll
        for (int c = 0; c < NC; c++) {
          E p[D];
          prods(v + (e + q) * NC, xv + q * NC, c, p);
#pragma unroll
          for (int d = 0; d < D; d++) a[c].deposit(p[d]);
        }
    }
  }
  // step h of a whole stage (xh: its bx)
  __device__ __forceinline__ void step(const unsigned char* base, const Place& pl, int h, const E* xh,
                                       const E* xs, unsigned xkey, bool conj) {
    E v[NR];
    load(base, pl, h, v);
    float m = 0.0f;
#pragma unroll
    for (int i = 0; i < NR; i += 2) m = max_abs3(m, key_word(v[i]), key_word(v[i + 1]));
    const unsigned bound = B::key(B::mul(key_ceiling<E>(__float_as_uint(m)), key_ceiling<E>(xkey)));
    bool fast = true;
#pragma unroll
    for (int c = 0; c < NC; c++) fast = fast && a[c].fast(bound, ND);
    if (CX && conj) {
#pragma unroll
      for (int e = 0; e < PS; e++) v[e * NC + NC - 1] = -v[e * NC + NC - 1];
    }
    if (fast) {
#pragma unroll
      for (int c = 0; c < NC; c++) a[c].deposits += ND;
    } else {
      bool careful = bound >= B::kInfKey;
      if (!careful) {
        // the exact largest key of each component's products, then the index that needs
        unsigned mk[NC];
#pragma unroll
        for (int c = 0; c < NC; c++) mk[c] = 0u;
#pragma unroll
        for (int e = 0; e < PS; e++)
#pragma unroll
          for (int c = 0; c < NC; c++) {
            E p[D], xv[NC];
#pragma unroll
            for (int q = 0; q < NC; q++) xv[q] = xh[e * NC + q];
            prods(v + e * NC, xv, c, p);
#pragma unroll
            for (int d = 0; d < D; d++) {
              const unsigned kk = B::key(p[d]);
              mk[c] = kk > mk[c] ? kk : mk[c];
            }
          }
#pragma unroll
        for (int c = 0; c < NC; c++) {
          a[c].prepare(mk[c], ND);
          if (a[c].idx == 0) careful = true;
        }
      }
      if (careful) {
        deposit_careful(base, pl, xs, h * PS, (h + 1) * PS, conj);
        return;
      }
    }
    constexpr int XR = 16 / (int)sizeof(E);   // reals of one 16-byte vector of bx
#pragma unroll
    for (int e = 0; e < PS; e += XR / NC) {
      E xv[XR];
      gt::lds_vec<E, XR>(xh + e * NC, xv);
#pragma unroll
      for (int q = 0; q < XR / NC; q++)
#pragma unroll
        for (int c = 0; c < NC; c++) {
          E p[D];
          prods(v + (e + q) * NC, xv + q * NC, c, p);
#pragma unroll
          for (int d = 0; d < D; d++) a[c].deposit(p[d]);
        }
    }
  }
};

// Partial states of units cut between CTAs: a CTA holds at most two, that of the unit its range
// begins inside (slot 2*cta) and that of the unit that begins in its range and goes on in the next
// CTA's (slot 2*cta + 1), whatever the number of outputs. Structure of arrays: field i
// (< NC*(2F+1): pri, car, flags per component) of slot s for the unit's output pp at
// scratch[(i*2*grid + s)*P + pp]. A cut unit's tickets, one per warp, are those of the CTA it
// begins in. Units that many CTAs share are summed by a kernel of their own (gemv_sum_parts_kernel).
//
// A CTA's range of stages holds whole units in its middle and possibly cut units at its two
// ends. Ends::close() ends the run of unit u in this CTA for the warp's outputs: the groups
// merge; a whole unit's entry is finished at once, a cut unit's part is saved and the unit is
// recorded as pending (at most two per CTA). Ends::settle() then, after the CTA's last stage,
// takes the tickets of the pending units (one per unit and warp: warps settle by themselves);
// the warp of the last CTA to arrive merges the parts (group q takes parts q, q+G, ...) and
// finishes its entries. Deferring the tickets keeps their atomics out of the stream.
template <typename E, bool CX, int F>
struct Ends {
  static constexpr int NC = CX ? 2 : 1, REC = 2 * F + 1;
  const XGemvArgs<E>& g;
  int P, lgG, grp, pp, out;   // group of this lane, its output's offset in a unit, lanes per group
  long long nout;
  int fs;                     // distance of a record's fields
  int n, u0, u1;              // pending units

  __device__ __forceinline__ void finish(long long o, Acc<E, F> (&a)[NC], const E (&y)[NC]) const {
    xb::finish_from<E, CX, F>(a, g.mode, y, g.y + o * g.incy * NC, g.br, g.bi,
                              g.ybin + o * g.incy * 2 * F * NC);
  }
  __device__ __forceinline__ void read_y(long long o, bool want, E (&y)[NC]) const {
#pragma unroll
    for (int c = 0; c < NC; c++) y[c] = want && g.mode == kOutValue ? g.y[o * g.incy * NC + c] : E(0);
  }
  // this lane's output in the partial state of CTA i; begins: of the unit that begins in its range
  __device__ __forceinline__ int slot(int i, bool begins) const { return (2 * i + (begins ? 1 : 0)) * P + pp; }
  __device__ __forceinline__ void close(const Split& sp, int u, Acc<E, F> (&a)[NC]) {
    const long long o = (long long)u * P + pp;
    const bool mine = grp == 0 && o < nout;
    const bool begins = u * g.nb >= sp.x0, whole = begins && u * g.nb + g.nb <= sp.x1;
    E y[NC];   // the entry's current value, loaded early
    read_y(o, mine && whole, y);
    lanes_merge<E, F, NC>(a, out);
    if (whole) {
      if (mine) finish(o, a, y);
      return;
    }
    if (mine) {
      E* rec = g.scratch + slot((int)blockIdx.x, begins);
#pragma unroll
      for (int c = 0; c < NC; c++) xb::put_rec<E, F>(a[c], rec + c * REC * fs, fs);
    }
    if (n == 0) u0 = u;
    else u1 = u;
    n += g.tickets != nullptr;   // without tickets gemv_sum_parts_kernel sums the parts
  }
  __device__ __forceinline__ void settle(const Split& sp) {
    if (n == 0) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // release this warp's parts, then take its tickets (lanes 0 and 1, one each)
    __threadfence();
    __syncwarp();
    bool last = false;
    if (lane < n) {
      const int b = (lane == 0 ? u0 : u1) * g.nb, first = sp.owner(b);
      unsigned* t = g.tickets + first * (kConsumers / 32) + warp;
      last = atomicAdd(t, 1u) == (unsigned)(sp.owner(b + g.nb - 1) - first);
      if (last) *t = 0u;
    }
    const unsigned mask = __ballot_sync(0xffffffffu, last);
    if (mask == 0) return;
    __threadfence();
#pragma unroll 1
    for (int k = 0; k < n; k++) {
      if (!(mask & (1u << k))) continue;
      const int u = k == 0 ? u0 : u1, first = sp.owner(u * g.nb);
      const int count = sp.owner(u * g.nb + g.nb - 1) - first + 1;
      const long long o = (long long)u * P + pp;
      E y[NC];
      read_y(o, grp == 0 && o < nout, y);
      Acc<E, F> a[NC];
#pragma unroll
      for (int c = 0; c < NC; c++) {
        SumAcc<E, F> sum;
        sum.zero();
        if (o < nout) {
#pragma unroll 2
          for (int q = grp; q < count; q += 1 << lgG) {
            Acc<E, F> part;
            xb::read_rec<E, F>(part, g.scratch + slot(first + q, q == 0) + c * REC * fs, fs);
            sum.add(part);
          }
        }
        sum.get(a[c]);
      }
      lanes_merge<E, F, NC>(a, out);
      if (grp == 0 && o < nout) finish(o, a, y);
    }
  }
};

template <typename E, bool CX, int F, bool ROWS>
__global__ void __launch_bounds__((threads<E, CX>()), 1)
gemv_stream_kernel(const __grid_constant__ XGemvArgs<E> g, const __grid_constant__ GemvMaps maps) {
  using Gm = Geom<E, CX, ROWS>;
  constexpr int NC = Gm::NC, PE = Gm::PE, ES = Gm::ES;
  extern __shared__ unsigned char smem_raw[];
  __shared__ Sync sy;
  unsigned char* ring = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, lane = tid & 31;
  const Gm m(g);
  const Split sp(g);

  if (tid == kConsumers) {
    for (int h = 0; h < g.phases; h++)
      asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.m[h]) : "memory");
    for (int i = 0; i < kStages; i++) {
      mbar_init(smem_u32(&sy.full[i]), 1);
      mbar_init(smem_u32(&sy.xfull[i]), 1);
      mbar_init(smem_u32(&sy.empty[i]), kConsumers / 32);
    }
    sy.abort_flag = 0;
    fence_barrier_init();
  }
  __syncthreads();

  if (tid >= kConsumers) {
    if constexpr (moves_regs<E, CX>()) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kMoveProducer));
    const int w = tid >> 5;
    if (w == kConsumers / 32 + 1) scale_stages<E, CX, ROWS>(g, m, sp, ring, sy);
    else if (w == kConsumers / 32 && lane == 0) copy_stages<E, CX, ROWS>(g, m, maps, sp, ring, sy);
  } else {
    if constexpr (moves_regs<E, CX>()) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kMoveConsumer));
    const long long polls = g.wait_polls > 0 ? g.wait_polls : kWaitPolls;
    const bool conj = CX && g.conj;
    const int lgN = m.lgN, nph = 1 << lgN;
    Ends<E, CX, F> ends{g, m.P, m.lgG, 0, 0, 32 >> m.lgG, m.nout, 2 * (int)gridDim.x * m.P, 0, 0, 0};
    const int grp = lane >> (5 - m.lgG);
    // rows kernel: thread p takes slot p, i.e. row (p mod P/NPH)*NPH + p / (P/NPH) of the band,
    // so that neighbouring lanes read neighbouring slots; columns kernel: column p
    const int p = (tid >> 5) * ends.out + (lane & (ends.out - 1));
    const int pp = ROWS ? ((p & ((m.P >> lgN) - 1)) << lgN) + (p >> (m.lgP - lgN)) : p;
    ends.grp = grp;
    ends.pp = pp;
    // phase of its row(s): columns kernel rows grp, grp + G, ... with G a multiple of NPH
    const int ph = (ROWS ? pp : grp) & (nph - 1);
    typename Consumer<E, CX, F, ROWS>::Place pl;
    pl.vec = lgN == 0;
    pl.stride = ROWS ? (uint32_t)ES : (uint32_t)(m.G >> lgN) * m.pitch;
    pl.shift = (uint32_t)((uintptr_t)g.A + (unsigned long long)ph * g.lda * ES) & 15u;
    pl.swz = (uint32_t)p & 7u;
    const uint32_t off =
        ROWS ? (pl.vec ? (uint32_t)(grp * m.P + p) * kThreadBytes : (uint32_t)p * m.pitch + (uint32_t)grp * kThreadBytes)
             : (uint32_t)ph * m.phase_bytes + (uint32_t)(grp >> lgN) * m.pitch + (uint32_t)p * ES;
    Ring r;
    int u = sp.x0 / g.nb, j = sp.x0 - u * g.nb;
    Consumer<E, CX, F, ROWS> con;
    con.zero();
    bool lost = false;
#pragma unroll 1
    for (int x = sp.x0; x < sp.x1;) {
      // the run of unit u in this CTA (a loop of its own: with the run's end inside the stage loop the
      // compiler lengthens the stage; FP32 complex rows, 8192^2, 164 us against 152)
      const int xe = sp.x1 - x < g.nb - j ? sp.x1 : x + (g.nb - j);
#pragma unroll 1
      for (; x < xe; x++) {
        if (stage_ready(sy, r, polls)) {
          const unsigned char* st = ring + (size_t)r.st * kStageBytes;
          // elements of this thread that exist; the columns kernel takes a partial last stage
          // whole (rows outside A arrive as zeros, and so do their x) unless A has fewer rows
          // than phases
          const long long k0 = (long long)j * m.SC;
          const long long rem = ROWS ? m.nred - k0 - grp * PE : (m.nred - k0 - grp + m.G - 1) >> m.lgG;
          const bool whole = rem >= PE || (!ROWS && m.nred >= 4);
          const int nval = (long long)u * m.P + pp >= m.nout || rem <= 0 ? 0 : whole ? PE : (int)rem;
          con.stage(st + off, pl, (const E*)(st + kStageA) + grp * PE * NC, sy.xkey[r.st], nval, conj);
        } else {
          lost = true;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&sy.empty[r.st]));
        r.next();
        j++;
      }
#pragma unroll
      for (int c = 0; c < NC; c++) {
        con.a[c].renorm();
        if (lost) con.a[c].flags |= kNaN;
      }
      ends.close(sp, u, con.a);
      con.zero();
      lost = false;
      j = 0;
      u++;
    }
    ends.settle(sp);
  }
  __syncthreads();
  if (tid == 0 && sy.abort_flag) atomicExch(g.status, 2);
}

// Sum of the parts of cut units, after a streaming kernel that took no tickets: where units are shared
// by more than kWide CTAs the last of them would sum all their parts alone (FP64 complex, 64 rows of
// 400,000: 148 parts, 1 MB, 139 us a call against 121 with this launch behind the stream). A CTA takes
// kSumOutputs outputs of a unit; thread (group, output) sums parts group, group + 32, ...; the groups
// of a warp meet by shuffles, the warps in shared memory.
constexpr int kWide = 12, kSumOutputs = 8;
template <typename E, bool CX, int F, bool ROWS>
__global__ void __launch_bounds__(256) gemv_sum_parts_kernel(const __grid_constant__ XGemvArgs<E> g, int grid) {
  constexpr int NC = CX ? 2 : 1, REC = 2 * F + 1;
  __shared__ E sm[8][kSumOutputs][NC * REC];
  const Split sp(g);
  const int P = kConsumers / g.groups, per = P / kSumOutputs;
  const int u = (int)blockIdx.x / per, t = threadIdx.x % kSumOutputs, warp = threadIdx.x >> 5;
  const int pp = (int)blockIdx.x % per * kSumOutputs + t, group = threadIdx.x / kSumOutputs;
  const int first = sp.owner(u * g.nb), count = sp.owner(u * g.nb + g.nb - 1) - first + 1;
  if (count == 1) return;   // finished by the streaming kernel
  const long long o = (long long)u * P + pp;
  const bool some = o < (ROWS ? g.R : g.C);
  const int fs = 2 * grid * P;
  Acc<E, F> a[NC];
#pragma unroll
  for (int c = 0; c < NC; c++) {
    SumAcc<E, F> sum;
    sum.zero();
    if (some) {
#pragma unroll 2
      for (int q = group; q < count; q += 256 / kSumOutputs) {
        Acc<E, F> part;
        xb::read_rec<E, F>(part, g.scratch + (2 * (first + q) + (q == 0 ? 1 : 0)) * P + pp + c * REC * fs, fs);
        sum.add(part);
      }
    }
    sum.get(a[c]);
  }
  lanes_merge<E, F, NC>(a, kSumOutputs);
  if ((threadIdx.x & 31) < kSumOutputs) {
#pragma unroll
    for (int c = 0; c < NC; c++) xb::put_rec<E, F>(a[c], &sm[warp][t][c * REC], 1);
  }
  __syncthreads();
  if (threadIdx.x >= kSumOutputs || !some) return;
#pragma unroll
  for (int c = 0; c < NC; c++) {
    SumAcc<E, F> sum;
    sum.zero();
#pragma unroll 1
    for (int w = 0; w < 8; w++) {
      Acc<E, F> part;
      part.zero();
#pragma unroll
      for (int i = 0; i < F; i++) {
        part.pri[i] = sm[w][t][c * REC + i];
        part.car[i] = sm[w][t][c * REC + F + i];
      }
      part.flags = xb::flags_from<E>(sm[w][t][c * REC + 2 * F]);
      part.set_idx_from_pri();
      sum.add(part);
    }
    sum.get(a[c]);
  }
  xb::finish<E, CX, F>(a, g.mode, g.y + o * g.incy * NC, g.br, g.bi, g.ybin + o * g.incy * 2 * F * NC);
}

// ---------------------------------------------------------------------------------------
// Rows kernel straight from global memory, for small matrices and for few rows. A CTA of 8 warps
// takes 8/S rows, S = g.groups warps to a row (S = 1, 2, 4, 8). No pipeline to fill and no unit to
// merge across CTAs: 7-8 us a call where the streaming kernel takes 10-12. Few long rows are cut
// between gridDim.y CTAs each (S = 8): every CTA leaves a partial state, record `part` of the row,
// and the last one to arrive (ticket) sums them. Field i of the record is at
// scratch[(i*R + row)*parts + part].
// ---------------------------------------------------------------------------------------
// Sum of the states of the S warps of a row (each the same in all its lanes), into the first of
// them. All threads of the CTA call it.
template <typename E, int F, int NC>
__device__ __forceinline__ void sum_warps(Acc<E, F> (&a)[NC], E (*sm)[NC * (2 * F + 1)], int S) {
  constexpr int REC = 2 * F + 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
#pragma unroll
    for (int c = 0; c < NC; c++) xb::put_rec<E, F>(a[c], &sm[warp][c * REC], 1);
  }
  __syncthreads();
  if ((warp & (S - 1)) == 0 && lane == 0) {
#pragma unroll
    for (int c = 0; c < NC; c++) {
      SumAcc<E, F> sum;
      sum.zero();
      sum.add(a[c]);
#pragma unroll 1
      for (int q = 1; q < S; q++) {
        Acc<E, F> o;
        o.zero();
#pragma unroll
        for (int i = 0; i < F; i++) {
          o.pri[i] = sm[warp + q][c * REC + i];
          o.car[i] = sm[warp + q][c * REC + F + i];
        }
        o.flags = xb::flags_from<E>(sm[warp + q][c * REC + 2 * F]);
        o.set_idx_from_pri();
        sum.add(o);
      }
      sum.get(a[c]);
    }
  }
}

// CTAs per SM it is built for: as many as hold its accumulators without spilling much (FP64 500x6291:
// 14.4 us with four against 18.5 with three).
template <typename E, bool CX>
constexpr int rows_direct_ctas(int fold) {
  if (sizeof(E) == 8) return CX ? (fold <= 2 ? 3 : 2) : fold <= 4 ? 4 : fold <= 6 ? 3 : 2;
  return CX ? (fold <= 3 ? 4 : fold <= 5 ? 3 : 2) : 4;
}

template <typename E, bool CX, int F>
__global__ void __launch_bounds__(256, (rows_direct_ctas<E, CX>(F))) gemv_rows_direct_kernel(const __grid_constant__ XGemvArgs<E> g) {
  constexpr int NC = CX ? 2 : 1, D = CX ? 2 : 1, REC = 2 * F + 1;
  constexpr int K = 4;   // elements per lane and step
  __shared__ E sm[8][NC * REC];
  __shared__ unsigned s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, S = g.groups;
  const int rows = 8 / S, parts = gridDim.y;
  const long long r = (long long)blockIdx.x * rows + warp / S;
  // this CTA's columns of the row: whole steps of the S warps
  const long long stride = (long long)K * 32 * S;
  const long long per = ((g.C + parts - 1) / parts + stride - 1) / stride * stride;
  const long long c0 = blockIdx.y * per, c1 = c0 + per < g.C ? c0 + per : g.C;
  Acc<E, F> a[NC];
#pragma unroll
  for (int c = 0; c < NC; c++) a[c].zero();
  if (r < g.R) {
    const E* row = g.A + r * g.lda * NC;
    // K elements from b (which exists) on, 32*S apart; WHOLE: all of them exist; PAIR: whole pairs are
    // loaded. All loads before the math and without branches: an absent element loads element b
    auto step = [&](long long b, auto whole, auto pair) {
      constexpr bool WHOLE = decltype(whole)::value != 0, PAIR = decltype(pair)::value != 0;
      Val<E, CX> av[K], xv[K];
#pragma unroll
      for (int k = 0; k < K; k++) {
        long long e = b + (long long)k * 32 * S;
        if (!WHOLE) e = e < c1 ? e : b;
        av[k] = xb::ldv<E, CX, PAIR>(row, e);
        xv[k] = xb::ldv<E, CX, PAIR>(g.x, e * g.incx);
      }
      int n = K;   // elements that exist
      if (!WHOLE) {
#pragma unroll
        for (int k = 1; k < K; k++)
          if (b + (long long)k * 32 * S >= c1) {
            av[k] = xv[k] = Val<E, CX>{E(0), E(0)};
            n = n < k ? n : k;
          }
      }
      E v[NC][K * D];
#pragma unroll
      for (int k = 0; k < K; k++) {
        if (!g.alpha_one && (WHOLE || k < n)) xv[k] = xb::scale<E, CX>(xv[k], g.ar, g.ai);
        if (CX && g.conj) av[k].i = -av[k].i;
        xb::products<E, CX, K * D>(av[k], xv[k], v, k);
      }
#pragma unroll
      for (int c = 0; c < NC; c++) a[c].template tile<K * D>(v[c], n * D);
    };
    auto steps = [&](auto pair) {
      long long w = c0 + (warp & (S - 1)) * 32;   // the warp's first element: it takes one of the two together
#pragma unroll 1
      for (; w + (long long)(K - 1) * 32 * S + 31 < c1; w += stride) step(w + lane, gt::Const<1>{}, pair);
      if (w + lane < c1) step(w + lane, gt::Const<0>{}, pair);
    };
    if (CX && ((uintptr_t)g.A | (uintptr_t)g.x) % (2 * sizeof(E)) == 0) steps(gt::Const<1>{});
    else steps(gt::Const<0>{});
  }
#pragma unroll
  for (int c = 0; c < NC; c++) a[c].renorm();
  warp_merge_all<E, F, NC>(a);
  if (S > 1) sum_warps<E, F, NC>(a, sm, S);
  if (parts > 1) {   // S = 8: one row per CTA
    const long long fs = g.R * parts;
    if (threadIdx.x == 0) {
      E* rec = g.scratch + r * parts + blockIdx.y;
#pragma unroll
      for (int c = 0; c < NC; c++) xb::put_rec<E, F>(a[c], rec + c * REC * fs, fs);
      __threadfence();
      s_last = atomicAdd(g.tickets + blockIdx.x, 1u) == (unsigned)parts - 1 ? 1u : 0u;
      if (s_last) g.tickets[blockIdx.x] = 0u;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
#pragma unroll
    for (int c = 0; c < NC; c++) {
      SumAcc<E, F> sum;
      sum.zero();
#pragma unroll 1
      for (int q = threadIdx.x; q < parts; q += 256) {
        Acc<E, F> o;
        xb::read_rec<E, F>(o, g.scratch + r * parts + q + c * REC * fs, fs);
        sum.add(o);
      }
      sum.get(a[c]);
    }
    warp_merge_all<E, F, NC>(a);
    sum_warps<E, F, NC>(a, sm, S);
  }
  if ((warp & (S - 1)) == 0 && lane == 0 && r < g.R)
    xb::finish<E, CX, F>(a, g.mode, g.y + r * g.incy * NC, g.br, g.bi, g.ybin + r * g.incy * 2 * F * NC);
}

// ---------------------------------------------------------------------------------------
// Columns kernel straight from global memory, for small matrices, which pay for filling the
// streaming kernel's pipeline and for its ends (us a call, this kernel / the streaming one:
// FP64 500x2000 10.7 / 13.5, 2048x1024 14.5 / 16.6, FP32 1000x500 10.4 / 13.7; even at
// 32 MB, and slower for short reductions: FP32 100x5000 10.4 / 8.3), and for FP64 complex up to
// 192 MB, where four deposits per element leave the stream little to hide (fold 3: 2048^2
// 35.0 / 37.7, 20000x500 66.0 / 68.9, but 4096^2 91.0 / 85.0 and 8192^2 307 / 270; fold 6: 2048^2
// 48.6 / 58.4, 5000^2 210 / 202), or of any size from fold 7, whose two accumulators spill in
// the streaming kernel (fold 8, 5000^2: 254 / 329).
// Short reductions of many columns come here too: a unit of the streaming kernel is 128/es*G rows deep,
// whatever the number of rows, and its ends cost as much as a stage (FP64 8x4000000 109 / 270, 100x500000
// 96 / 115, but 160x200000 72 / 55; FP32 8x4000000 106 / 304, 40x2000000 141 / 156, but 64x1000000 106 / 84;
// FP64 complex 8x4000000 273 / 1004, 300x100000 148 / 168, but 500x40000 117 / 105; FP32 complex 8x4000000
// 189 / 488, 128x300000 115 / 125, but 160x200000 107 / 95; and fewer columns: FP64 100x50000 24.6 / 20.6).
// A CTA of 256 threads is G = g.groups row groups of 256/G threads, one column each; grid =
// (column blocks, row chunks), inside a chunk group q takes rows q, q + G, ..., four per step.
// fl(alpha*x) of 256 rows at a time is formed in shared memory. The groups' states merge
// through shared memory; with several chunks each leaves a partial state (structure of
// arrays), and the last CTA of a column block to arrive sums them and finishes.
// ---------------------------------------------------------------------------------------
template <typename E, bool CX>
__host__ __device__ constexpr bool stream_cols(int fold) { return !(CX && sizeof(E) == 8 && fold > 6); }
template <typename E, bool CX>
constexpr bool direct_cols(long long nout, long long nred) {
  constexpr int es = (CX ? 2 : 1) * (int)sizeof(E);
  if (nout >= 80000 && nred <= (es == 16 ? 384 : es == 4 ? 48 : 128)) return true;
  return es == 16 ? nout * nred * es <= (192ll << 20) : nred >= 256 && nout * nred * es <= (16ll << 20);
}

// Sum of the G row groups' states (renormalised) through sm[i * 256 + thread]: group 0 ends with
// the merged state. All 256 threads call it.
template <typename E, int F>
__device__ __forceinline__ void sum_groups(Acc<E, F>& a, E* sm, int grp, int t, int G, int T) {
  if (G == 1) return;
  __syncthreads();
  if (grp > 0) xb::put_rec<E, F>(a, sm + threadIdx.x, 256);
  __syncthreads();
  if (grp == 0) {
    SumAcc<E, F> sum;
    sum.zero();
    sum.add(a);
#pragma unroll 1
    for (int q = 1; q < G; q++) {
      const E* rec = sm + q * T + t;
      Acc<E, F> o;
      o.zero();
#pragma unroll
      for (int i = 0; i < F; i++) {
        o.pri[i] = rec[i * 256];
        o.car[i] = rec[(F + i) * 256];
      }
      o.flags = xb::flags_from<E>(rec[2 * F * 256]);
      o.set_idx_from_pri();
      sum.add(o);
    }
    sum.get(a);
  }
}

template <typename E, bool CX>
constexpr int cols_direct_ctas(int fold) {
  return CX ? (sizeof(E) == 4 && fold <= 3 ? 3 : 2) : fold <= 4 ? 4 : fold <= 6 || sizeof(E) == 4 ? 3 : 2;
}

template <typename E, bool CX, int F>
__global__ void __launch_bounds__(256, (cols_direct_ctas<E, CX>(F))) gemv_cols_direct_kernel(const __grid_constant__ XGemvArgs<E> g) {
  constexpr int NC = CX ? 2 : 1, D = CX ? 2 : 1, K = 4, REC = 2 * F + 1;
  __shared__ E sm[REC * 256];
  __shared__ E xs[256 * NC];
  __shared__ unsigned s_last;
  const int G = g.groups, T = 256 / G;
  const int grp = threadIdx.x / T, t = threadIdx.x % T;
  const long long col = (long long)blockIdx.x * T + t;
  const int chunk = blockIdx.y, nchunks = gridDim.y;
  const long long per = (g.R + nchunks - 1) / nchunks;
  const long long r0 = (long long)chunk * per < g.R ? (long long)chunk * per : g.R;
  const long long r1 = r0 + per < g.R ? r0 + per : g.R;
  Acc<E, F> a[NC];
#pragma unroll
  for (int c = 0; c < NC; c++) a[c].zero();
  const E* A = g.A + col * NC;
#pragma unroll 1
  for (long long base = r0; base < r1; base += 256) {
    const int n = r1 - base < 256 ? (int)(r1 - base) : 256;
    __syncthreads();
    if ((int)threadIdx.x < n) {
      Val<E, CX> v = xb::ldv<E, CX>(g.x, (base + threadIdx.x) * g.incx);
      if (!g.alpha_one) v = xb::scale<E, CX>(v, g.ar, g.ai);
      xs[threadIdx.x * NC] = v.r;
      if constexpr (CX) xs[threadIdx.x * NC + 1] = v.i;
    }
    __syncthreads();
    if (col >= g.C) continue;
    // K rows from b (which exists) on, G apart; WHOLE: all of them exist; PAIR: whole pairs are loaded.
    // All loads before the math and without branches: an absent row loads row b
    auto step = [&](int b, auto whole, auto pair) {
      constexpr bool WHOLE = decltype(whole)::value != 0, PAIR = decltype(pair)::value != 0;
      Val<E, CX> av[K];
#pragma unroll
      for (int k = 0; k < K; k++) {
        const int i = WHOLE || b + k * G < n ? b + k * G : b;
        av[k] = xb::ldv<E, CX, PAIR>(A + (base + i) * g.lda * NC, 0);
      }
      int m = K;   // rows that exist; the others multiply zeros
      E v[NC][K * D];
#pragma unroll
      for (int k = 0; k < K; k++) {
        Val<E, CX> xv{E(0), E(0)};
        if (WHOLE || b + k * G < n) {
          const int i = b + k * G;
          xv = Val<E, CX>{xs[i * NC], CX ? xs[i * NC + NC - 1] : E(0)};
        } else {
          av[k] = Val<E, CX>{E(0), E(0)};
          m = m < k ? m : k;
        }
        if (CX && g.conj) av[k].i = -av[k].i;
        xb::products<E, CX, K * D>(av[k], xv, v, k);
      }
      if constexpr (CX) tile2<E, F, K * D>(a[0], v[0], a[1], v[1]);
      else a[0].template tile<K * D>(v[0], m * D);
    };
    auto steps = [&](auto pair) {
      int b = grp;
      if constexpr (CX && sizeof(E) == 8 && F > 4) {   // whole steps of their own would spill
#pragma unroll 1
        for (; b < n; b += K * G) step(b, gt::Const<0>{}, pair);
      } else {
#pragma unroll 1
        for (; b + (K - 1) * G < n; b += K * G) step(b, gt::Const<1>{}, pair);
        if (b < n) step(b, gt::Const<0>{}, pair);
      }
    };
    if (CX && (uintptr_t)g.A % (2 * sizeof(E)) == 0) steps(gt::Const<1>{});
    else steps(gt::Const<0>{});
  }
  E* part = g.scratch + (long long)chunk * NC * REC * g.C + col;   // field i at part[i * C]
#pragma unroll
  for (int c = 0; c < NC; c++) {
    a[c].renorm();
    sum_groups<E, F>(a[c], sm, grp, t, G, T);
    if (nchunks > 1 && grp == 0 && col < g.C) xb::put_rec<E, F>(a[c], part + c * REC * g.C, g.C);
  }
  if (nchunks > 1) {
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
      s_last = atomicAdd(g.tickets + blockIdx.x, 1u) == (unsigned)nchunks - 1 ? 1u : 0u;
      if (s_last) g.tickets[blockIdx.x] = 0u;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
#pragma unroll
    for (int c = 0; c < NC; c++) {
      SumAcc<E, F> sum;
      sum.zero();
      if (col < g.C) {
#pragma unroll 2
        for (int ch = grp; ch < nchunks; ch += G) {
          Acc<E, F> o;
          xb::read_rec<E, F>(o, g.scratch + ((long long)ch * NC + c) * REC * g.C + col, g.C);
          sum.add(o);
        }
      }
      sum.get(a[c]);
      sum_groups<E, F>(a[c], sm, grp, t, G, T);
    }
  }
  if (grp == 0 && col < g.C)
    xb::finish<E, CX, F>(a, g.mode, g.y + col * g.incy * NC, g.br, g.bi, g.ybin + col * g.incy * 2 * F * NC);
}

// Whether the streaming kernel of rows (columns) can run on the current device; the first query
// opts it in to its shared memory there. It cannot where the compiler built it with other than the
// registers that moves_regs() deals out (its setmaxnreg would wait for ever): the direct kernel serves
// then.
template <typename E, bool CX, int F>
cudaError_t gemv_streams(bool rows, bool* can) {
  if (!rows && !stream_cols<E, CX>(F)) {
    *can = false;
    return cudaSuccess;
  }
  constexpr int kMaxDevices = 64;
  static std::atomic<int> known[kMaxDevices][2];   // 0: not yet, 1: no, 2: yes
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  int k = dev < kMaxDevices ? known[dev][rows].load(std::memory_order_relaxed) : 0;
  if (k == 0) {
    const auto f = rows ? gemv_stream_kernel<E, CX, F, true> : gemv_stream_kernel<E, CX, F, !stream_cols<E, CX>(F)>;
    k = 2;
    if constexpr (moves_regs<E, CX>()) {
      cudaFuncAttributes at;
      if ((e = cudaFuncGetAttributes(&at, f)) != cudaSuccess) return e;
      if (at.numRegs != kMoveLaunch) k = 1;
    }
    e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
    if (e != cudaSuccess) return e;
    if (dev < kMaxDevices) known[dev][rows].store(k, std::memory_order_relaxed);
  }
  *can = k == 2;
  return cudaSuccess;
}

template <typename E, bool CX, int F>
cudaError_t launch_gemv(const XGemvArgs<E>& g, const GemvMaps* maps, bool rows, int grid, cudaStream_t s) {
  if (!maps) {
    if (rows) {
      gemv_rows_direct_kernel<E, CX, F><<<dim3(grid, g.parts), 256, 0, s>>>(g);
    } else {
      gemv_cols_direct_kernel<E, CX, F><<<dim3(grid, g.parts), 256, 0, s>>>(g);
    }
    return cudaGetLastError();
  }
  const auto f = rows ? gemv_stream_kernel<E, CX, F, true> : gemv_stream_kernel<E, CX, F, !stream_cols<E, CX>(F)>;
  f<<<grid, threads<E, CX>(), kSmemBytes, s>>>(g, *maps);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || !g.scratch || g.tickets) return e;
  // parts without tickets: their sum
  const long long nout = rows ? g.R : g.C;
  const int P = kConsumers / g.groups;
  const unsigned blocks = (unsigned)((nout + P - 1) / P * (P / kSumOutputs));
  if (rows) gemv_sum_parts_kernel<E, CX, F, true><<<blocks, 256, 0, s>>>(g, grid);
  else gemv_sum_parts_kernel<E, CX, F, false><<<blocks, 256, 0, s>>>(g, grid);
  return cudaGetLastError();
}

}  // namespace gs
}  // namespace rb
