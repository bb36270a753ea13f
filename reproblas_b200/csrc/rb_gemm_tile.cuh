// rb_gemm_tile.cuh -- the plain binned gemm of every element type (FP64 / FP32, real and
// complex) on sm_100a: one kernel over tiles of C and blocks of K.
//
// C_ij <- conv( binned(beta*C_ij) + sum_k products of fl(alpha*op(A)_ik) and op(B)_kj )
// (src/reproBLAS/r[dszc]gemm.c, src/binnedBLAS/[dszc]b[dszc]gemm.ccog; the deposited values are
// listed in rb_entry.cuh). Operands use general strides in elements,
//   op(A)_ik = A[i*sai + k*sak], op(B)_kj = B[k*sbk + j*sbj], C_ij = C[i*sci + j*scj],
// which cover both orders and all transposes.
//
// What bounds it: instruction issue. Measured with register-resident deposits fed from shared
// memory, a warp instruction on the FP64 pipe takes two issue cycles of its SM sub-partition
// and every other instruction one, so a fold-3 FP64 product (1 multiply, 7 adds, 3 sticky-bit
// ORs, 2 copies of a high word) cannot take less than ~21.5 cycles: 1.70 T products/s =
// 3.4 TFLOP/s on 148 SMs. FP32 products (8 FP32 instructions, 3 ORs) take 12.2 cycles at best
// (packed f32x2 adds issue at half rate and save nothing: 11.6). So everything here serves the
// deposit loop: no per-product checks, operands read as 16-byte shared-memory vectors, tiles
// copied by cp.async (no registers and no address arithmetic per element), and only the
// primaries in registers -- carries and non-finite classes, touched every few thousand
// deposits, live in shared memory.
//
// Tile check: per K block the largest magnitude key of every tile row of op(A) and column of
// op(B) is found (alpha and conjugation are applied in the same pass). When the product of
// two bounds stays below an entry's cap (rounding is monotone, so every product of the block
// is at most that bound), no product of the block can need a coarser index or be non-finite,
// and the block's products are deposited without further checks. Otherwise the exact largest
// magnitude of each entry's products is found first (dmdupdate), then the same loop runs;
// only blocks with non-finite products or index-0 entries take a per-product loop.
#pragma once
#include <atomic>

#include "rb_entry.cuh"
#include "rb_ptx.cuh"

namespace rb {
namespace gt {

using xb::Val;

// N adjacent reals of shared memory, as the widest vectors their total size allows.
template <typename E, int N>
__device__ __forceinline__ void lds_vec(const E* p, E (&v)[N]) {
  constexpr int B = N * (int)sizeof(E);
  if constexpr (B % 16 == 0) {
    constexpr int PER = 16 / (int)sizeof(E);
#pragma unroll
    for (int t = 0; t < N / PER; t++) {
      if constexpr (sizeof(E) == 8) {
        const double2 w = *(const double2*)(p + t * PER);
        v[t * PER] = w.x;
        v[t * PER + 1] = w.y;
      } else {
        const float4 w = *(const float4*)(p + t * PER);
        v[t * PER] = w.x;
        v[t * PER + 1] = w.y;
        v[t * PER + 2] = w.z;
        v[t * PER + 3] = w.w;
      }
    }
  } else if constexpr (B == 8 && sizeof(E) == 4) {
    const float2 w = *(const float2*)p;
    v[0] = w.x;
    v[1] = w.y;
  } else {
#pragma unroll
    for (int t = 0; t < N; t++) v[t] = p[t];
  }
}

// cp.async of BYTES (4, 8 or 16; both addresses so aligned), zero-filled when !ok (the source is
// not read then).
template <int BYTES>
__device__ __forceinline__ void cp_async_zfill(uint32_t dst, const void* src, bool ok) {
  const int n = ok ? BYTES : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(BYTES), "r"(n)
               : "memory");
}

constexpr int kThreads = 256;   // 16 x 16

template <int V> struct Const { static constexpr int value = V; };

// Tile geometry: thread (tx, ty) owns the TM x TN entries at rows ty*TM.., columns tx*TN...
template <typename E, bool CX, int F, int TM, int TN>
struct Geo {
  static constexpr int NC = CX ? 2 : 1, D = CX ? 2 : 1;   // components; deposits per product
  static constexpr int BM = 16 * TM, BN = 16 * TN, BK = 32;
  static constexpr int PAD = 16 / (int)sizeof(E);         // keeps the k rows 16-byte aligned
  static constexpr int LDA = BM * NC + PAD, LDB = BN * NC + PAD;   // reals per k row
  static constexpr int NA = TM * TN * NC;                 // accumulators per thread
  static constexpr int STAGE = BK * (LDA + LDB);          // reals per stage (two stages)
  static constexpr size_t CAR_OFF = (size_t)2 * STAGE * sizeof(E);
  static constexpr size_t KEY_OFF = CAR_OFF + (size_t)NA * F * kThreads * 4;
  static constexpr size_t FLAG_OFF = KEY_OFF + (size_t)3 * (BM + BN) * 4;
  static constexpr size_t SMEM = FLAG_OFF + (size_t)NA * kThreads;
  static constexpr int REC = 2 * F + 1;                   // reals of one partial record
  // partial state of one tile, reals
  static constexpr size_t PART = (size_t)NA * REC * kThreads;
};

template <typename E, bool CX, int F, int TM, int TN>
struct Tile {
  using G = Geo<E, CX, F, TM, TN>;
  using B = BT<E>;
  static constexpr int NC = G::NC, D = G::D, BM = G::BM, BN = G::BN, BK = G::BK, NA = G::NA;
  static constexpr int LDA = G::LDA, LDB = G::LDB;
  // k steps per trip of the deposit loop (a longer body moves fewer registers at its end, until
  // it leaves the instruction cache)
  static constexpr int UK = (sizeof(E) == 8 || CX) ? 8 : 4;

  E pri[NA][F];    // entry (i, j), component c at (i*TN + j)*NC + c
  unsigned cap;    // smallest cap of this thread's entries (BT::cap_of; 0: some entry is empty)
  int dep;         // deposits since the last renormalisation (the same for the whole CTA)
  E* stages;
  int* car;        // carries, [NA][F][256] (every carry is an integer below 2^31)
  unsigned* keys;  // three buffers of [BM] rows of op(A), [BN] columns of op(B)
  unsigned char* flg;   // non-finite classes, [NA][256]

  __device__ __forceinline__ void attach(unsigned char* smem) {
    stages = (E*)smem;
    car = (int*)(smem + G::CAR_OFF) + threadIdx.x;
    keys = (unsigned*)(smem + G::KEY_OFF);
    flg = smem + G::FLAG_OFF + threadIdx.x;
  }
  // Empty states for the tile at (m0, n0). Entries outside C (whose products are zeros and which
  // are never written) start at index 1, above any bound, so that they take no thread of an
  // edge tile off the unchecked path.
  __device__ __forceinline__ void zero(const XGemmArgs<E>& g, long long m0, long long n0) {
    const int ra = (threadIdx.x >> 4) * TM, cb = (threadIdx.x & 15) * TN;
#pragma unroll
    for (int e = 0; e < NA; e++) {
      const int i = e / (TN * NC), j = e / NC % TN;
      const bool in = m0 + ra + i < g.M && n0 + cb + j < g.N;
#pragma unroll
      for (int q = 0; q < F; q++) {
        pri[e][q] = in ? E(0) : B::bin(1 + q);
        car[(e * F + q) * kThreads] = 0;
      }
      flg[e * kThreads] = 0;
    }
    cap = 0u;
    dep = 0;
  }

  // accumulator e as a whole (e is a compile-time constant where this is used)
  __device__ __forceinline__ void get(int e, Acc<E, F>& a) const {
#pragma unroll
    for (int i = 0; i < F; i++) {
      a.pri[i] = pri[e][i];
      a.car[i] = (E)car[(e * F + i) * kThreads];
    }
    a.flags = flg[e * kThreads];
    a.deposits = 0;
    a.set_idx_from_pri();
    a.renorm();
  }

  static __device__ __forceinline__ unsigned cap_of_pri(E p0) {
    return p0 == E(0) ? 0u : B::cap_of(B::mindex(p0));
  }

  // binned_dmrenorm (src/binned/dmrenorm.c:70-86) of every accumulator
  __device__ __forceinline__ void renorm_all() {
#pragma unroll
    for (int e = 0; e < NA; e++) {
      if (pri[e][0] == E(0)) continue;
#pragma unroll
      for (int i = 0; i < F; i++) {
        typename B::U u = B::bits(pri[e][i]);
        car[(e * F + i) * kThreads] += (int)((u >> (B::kMant - 3)) & 3) - 2;
        u &= ~((typename B::U)1 << (B::kMant - 3));
        u |= (typename B::U)1 << (B::kMant - 2);
        pri[e][i] = B::from(u);
      }
    }
    dep = 0;
  }

  __device__ __forceinline__ void load_ab(const E* sa, const E* sb, int k, E (&a)[TM * NC],
                                          E (&b)[TN * NC]) const {
    lds_vec<E, TM * NC>(sa + k * LDA, a);
    lds_vec<E, TN * NC>(sb + k * LDB, b);
  }
  // the D products of entry (i, j), component c
  static __device__ __forceinline__ void prods(const E (&a)[TM * NC], const E (&b)[TN * NC], int i,
                                               int j, int c, E (&p)[D]) {
    if constexpr (CX) {
      const E ar = a[2 * i], ai = a[2 * i + 1], br = b[2 * j], bi = b[2 * j + 1];
      p[0] = c == 0 ? B::mul(ar, br) : B::mul(ar, bi);
      p[1] = c == 0 ? B::mul(-ai, bi) : B::mul(ai, br);
    } else {
      p[0] = B::mul(a[i], b[j]);
    }
  }
  // binned_dmddeposit (src/binned/dmddeposit.c:57-70), index != 0
  __device__ __forceinline__ void deposit(int e, E x) {
#pragma unroll
    for (int i = 0; i < F - 1; i++) {
      const E q = B::add(odd(x), pri[e][i]);
      x = B::add(x, B::sub(pri[e][i], q));
      pri[e][i] = q;
    }
    pri[e][F - 1] = B::add(pri[e][F - 1], odd(x));
  }

  // Some entry's bound reaches its cap: find the largest finite magnitude of every entry's
  // products in the block and move the entries that need it to a coarser index. Returns true
  // when the block must be deposited product by product (a product may be non-finite, or an
  // entry is at index 0).
  __device__ __noinline__ static unsigned raise_entry(E* p, int* c, unsigned m) {
    Acc<E, F> a;
#pragma unroll
    for (int i = 0; i < F; i++) {
      a.pri[i] = p[i];
      a.car[i] = (E)c[i * kThreads];
    }
    a.flags = 0;
    a.deposits = 0;
    a.set_idx_from_pri();
    const int ni = B::index_of_key(m);
    if (ni < a.idx) {
      a.raise_to(ni);
#pragma unroll
      for (int i = 0; i < F; i++) {
        p[i] = a.pri[i];
        c[i * kThreads] = (int)a.car[i];
      }
    }
    return a.cap | (a.idx == 0 ? 1u : 0u);   // caps are multiples of 2^20 (2^23 in FP32)
  }
  // Largest key of each accumulator's products; FINITE: none of them is Inf or NaN (a float maximum
  // then does: one three-input instruction for two products), else only the finite ones count.
  template <bool FINITE>
  __device__ __forceinline__ void max_keys(const E* sa, const E* sb, int kend, unsigned (&mk)[NA]) const {
    // FP64 products of 2^1017 and more, whose high words are a float's NaN, give a key of index 0,
    // which is theirs
    float top[NA];
#pragma unroll
    for (int e = 0; e < NA; e++) {
      mk[e] = 0u;
      top[e] = 0.0f;
    }
#pragma unroll 1
    for (int k = 0; k < kend; k += 2) {   // kend is even
      E a[2][TM * NC], b[2][TN * NC];
#pragma unroll
      for (int q = 0; q < 2; q++) load_ab(sa, sb, k + q, a[q], b[q]);
#pragma unroll
      for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN; j++)
#pragma unroll
          for (int c = 0; c < NC; c++) {
            E p[2][D];
#pragma unroll
            for (int q = 0; q < 2; q++) prods(a[q], b[q], i, j, c, p[q]);
            const int e = (i * TN + j) * NC + c;
            if constexpr (FINITE) {
#pragma unroll
              for (int d = 0; d < D; d++) top[e] = max_abs3(top[e], key_word(p[0][d]), key_word(p[1][d]));
            } else {
#pragma unroll
              for (int q = 0; q < 2; q++)
#pragma unroll
                for (int d = 0; d < D; d++) {
                  const unsigned kk = B::key(p[q][d]);
                  mk[e] = kk > mk[e] && kk < B::kInfKey ? kk : mk[e];
                }
            }
          }
    }
    if constexpr (FINITE) {
#pragma unroll
      for (int e = 0; e < NA; e++) mk[e] = __float_as_uint(top[e]);
    }
  }
  __device__ __forceinline__ bool prepare(const E* sa, const E* sb, int kend, bool finite,
                                          const unsigned* kra, const unsigned* kcb) {
    unsigned mk[NA];
    bool careful = !finite;
    bool exact = false;
    if (finite) {
      // The index wanted is that of the largest product. Where that of the bound and that of the
      // largest of the first four products agree, as they nearly always do in FP64 (an index spans 40
      // binades), it lies between the two and is known. In FP32 (13 binades) some entry of a warp
      // nearly always needs the whole block.
      if constexpr (sizeof(E) == 8) {
        max_keys<true>(sa, sb, 4, mk);
        exact = true;
#pragma unroll
        for (int i = 0; i < TM; i++)
#pragma unroll
          for (int j = 0; j < TN; j++) {
            const int ib = B::index_of_key(B::key(B::mul(key_ceiling<E>(kra[i]), key_ceiling<E>(kcb[j]))));
#pragma unroll
            for (int c = 0; c < NC; c++) exact = exact && B::index_of_key(mk[(i * TN + j) * NC + c]) == ib;
          }
      }
      if (!exact) max_keys<true>(sa, sb, kend, mk);
    } else {
      max_keys<false>(sa, sb, kend, mk);
    }
    cap = 0xffffffffu;
#pragma unroll
    for (int e = 0; e < NA; e++) {
      unsigned c;
      if (pri[e][0] == E(0)) {
        // empty: straight to the index (its carries are zero)
        const int ni = B::index_of_key(mk[e]);
#pragma unroll
        for (int i = 0; i < F; i++) pri[e][i] = B::bin(ni + i);
        c = B::cap_of(ni) | (ni == 0 ? 1u : 0u);
      } else {
        // through a copy: the call takes an address, and pri must stay in registers
        E t[F];
#pragma unroll
        for (int i = 0; i < F; i++) t[i] = pri[e][i];
        c = raise_entry(t, car + e * F * kThreads, mk[e]);
#pragma unroll
        for (int i = 0; i < F; i++) pri[e][i] = t[i];
      }
      careful = careful || (c & 1u);
      cap = (c & ~1u) < cap ? (c & ~1u) : cap;
    }
    return careful;
  }
  // product by product: non-finite values only record their class, index-0 entries take the
  // compressed first slice
  __device__ __forceinline__ void deposit_careful(const E* sa, const E* sb, int kend) {
#pragma unroll 1
    for (int k = 0; k < kend; k++) {
      E a[TM * NC], b[TN * NC];
      load_ab(sa, sb, k, a, b);
#pragma unroll
      for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN; j++)
#pragma unroll
          for (int c = 0; c < NC; c++) {
            E p[D];
            prods(a, b, i, j, c, p);
            const int e = (i * TN + j) * NC + c;
#pragma unroll
            for (int d = 0; d < D; d++) {
              if (B::key(p[d]) >= B::kInfKey) {
                flg[e * kThreads] |= (unsigned char)classify_nonfinite(p[d]);
              } else if (B::mindex0(pri[e][0])) {
                Acc<E, F> t;
#pragma unroll
                for (int q = 0; q < F; q++) t.pri[q] = pri[e][q];
                t.deposit0(p[d]);
#pragma unroll
                for (int q = 0; q < F; q++) pri[e][q] = t.pri[q];
              } else {
                deposit(e, p[d]);
              }
            }
          }
    }
  }

  // Deposit the products of K blocks [kb0, kb1) of the tile at (m0, n0). All 256 threads of the
  // CTA call it together.
  __device__ __forceinline__ void reduce(const XGemmArgs<E>& g, long long m0, long long n0,
                                         long long kb0, long long kb1) {
    const int tid = threadIdx.x, lane = tid & 31;
    const int ra = (tid >> 4) * TM, cb = (tid & 15) * TN;
    // element copies of a stage: thread t copies AEL elements of op(A) and BEL of op(B), at a
    // fixed distance, along the operand's unit stride
    constexpr int AEL = BM * BK / kThreads, BEL = BN * BK / kThreads;
    const bool a_k = g.sak == 1, b_j = g.sbj == 1;
    const int ai = a_k ? tid / BK : tid % BM, ak = a_k ? tid % BK : tid / BM;
    const int bj = b_j ? tid % BN : tid / BK, bk = b_j ? tid / BN : tid % BK;
    constexpr int UA_I = kThreads / BK, UA_K = kThreads / BM, UB_J = kThreads / BK, UB_K = kThreads / BN;
    const long long a_step = a_k ? UA_I * g.sai : UA_K * g.sak;
    const long long b_step = b_j ? UB_K * g.sbk : UB_J * g.sbj;
    const E* pa = g.A + ((m0 + ai) * g.sai + (kb0 * BK + ak) * g.sak) * NC;
    const E* pb = g.B + ((kb0 * BK + bk) * g.sbk + (n0 + bj) * g.sbj) * NC;
    // a complex element is copied whole when the array is aligned to it
    const bool a_whole = CX && ((uintptr_t)g.A % (2 * sizeof(E))) == 0;
    const bool b_whole = CX && ((uintptr_t)g.B % (2 * sizeof(E))) == 0;

    const int a_off = ak * LDA + ai * NC, b_off = BK * LDA + bk * LDB + bj * NC;
    const int a_doff = a_k ? UA_I * NC : UA_K * LDA, b_doff = b_j ? UB_K * LDB : UB_J * NC;
    const bool mn_whole = m0 + BM <= g.M && n0 + BN <= g.N;

    // copies of one operand's elements; WHOLE: all of them exist
    auto copy = [&](auto whole, auto cnt, const E* p, long long step, uint32_t d, uint32_t dstep,
                    bool vec, auto exists, const E* base) {
#pragma unroll
      for (int u = 0; u < decltype(cnt)::value; u++) {
        const bool ok = decltype(whole)::value || exists(u);
        const E* s = ok ? p : base;
        if constexpr (CX) {
          if (vec) cp_async_zfill<2 * sizeof(E)>(d, s, ok);
          else {
            cp_async_zfill<sizeof(E)>(d, s, ok);
            cp_async_zfill<sizeof(E)>(d + sizeof(E), s + 1, ok);
          }
        } else {
          cp_async_zfill<sizeof(E)>(d, s, ok);
        }
        p += step;
        d += dstep;
      }
    };
    using Yes = Const<1>;
    using No = Const<0>;
    auto issue = [&](long long kb, int st) {
      const long long k0 = kb * BK;
      const uint32_t so = smem_u32(stages) + (uint32_t)(st * G::STAGE * sizeof(E));
      const uint32_t da = so + a_off * (uint32_t)sizeof(E), db = so + b_off * (uint32_t)sizeof(E);
      const uint32_t sda = a_doff * (uint32_t)sizeof(E), sdb = b_doff * (uint32_t)sizeof(E);
      if (mn_whole && k0 + BK <= g.K) {
        auto all = [](int) { return true; };
        copy(Yes{}, Const<AEL>{}, pa, a_step * NC, da, sda, a_whole, all, g.A);
        copy(Yes{}, Const<BEL>{}, pb, b_step * NC, db, sdb, b_whole, all, g.B);
      } else {
        copy(No{}, Const<AEL>{}, pa, a_step * NC, da, sda, a_whole, [&](int u) {
          return m0 + ai + (a_k ? UA_I * u : 0) < g.M && k0 + ak + (a_k ? 0 : UA_K * u) < g.K;
        }, g.A);
        copy(No{}, Const<BEL>{}, pb, b_step * NC, db, sdb, b_whole, [&](int u) {
          return n0 + bj + (b_j ? 0 : UB_J * u) < g.N && k0 + bk + (b_j ? UB_K * u : 0) < g.K;
        }, g.B);
      }
      pa += BK * g.sak * NC;
      pb += BK * g.sbk * NC;
      cp_async_commit();
    };
    // Largest key of the elements this thread copied, element u at p + u*step; alpha and the
    // conjugation are applied to them first (UPD). Along k (lane = k) a warp holds whole rows,
    // else the thread holds one row and the warps meet in shared memory.
    auto scan = [&](auto cnt, E* p, int step, bool along_k, int row, int row_step, unsigned* kr,
                    bool conj, bool mul, int kfirst, int kstep, int krem) {
      unsigned top = 0;
#pragma unroll
      for (int u = 0; u < decltype(cnt)::value; u++) {
        unsigned m;
        if constexpr (CX) {
          Val<E, CX> v{p[0], p[1]};
          if (conj || mul) {
            if (conj) v.i = -v.i;
            if (mul && kfirst + u * kstep < krem) v = xb::scale<E, CX>(v, g.ar, g.ai);
            p[0] = v.r;
            p[1] = v.i;
          }
          const unsigned mr = B::key(v.r), mi = B::key(v.i);
          m = mr > mi ? mr : mi;
        } else {
          E v = p[0];
          if (mul) {
            if (kfirst + u * kstep < krem) v = B::mul(v, g.ar);   // padding stays zero
            p[0] = v;
          }
          m = B::key(v);
        }
        p += step;
        if (along_k) {
          m = __reduce_max_sync(0xffffffffu, m);
          if (lane == 0) kr[row + u * row_step] = m;
        } else {
          top = m > top ? m : top;
        }
      }
      if (!along_k) atomicMax(kr + row, top);
    };

    __syncthreads();   // the stages and keys may still be read by the previous call's last block
    for (int r = tid; r < 2 * (BM + BN); r += kThreads) keys[r] = 0u;
    issue(kb0, 0);
    __syncthreads();
    int kc = 0;        // key buffer of block kb (three in turn)
#pragma unroll 1
    for (long long kb = kb0; kb < kb1; kb++) {
      const int st = (int)(kb - kb0) & 1;
      E* sa = stages + st * G::STAGE;
      E* sb = sa + BK * LDA;
      const long long krem = g.K - kb * BK;
      const int kr = krem < BK ? (int)krem : BK;
      unsigned* kcur = keys + kc * (BM + BN);
      cp_async_wait<0>();   // this thread's copies of block kb have landed
      scan(Const<AEL>{}, sa + a_off, a_doff, a_k, ai, UA_I, kcur, g.conja, !g.alpha_one, ak,
           a_k ? 0 : UA_K, kr);
      scan(Const<BEL>{}, sa + b_off, b_doff, !b_j, bj, UB_J, kcur + BM, g.conjb, false, 0, 0, kr);
      __syncthreads();      // block kb and its keys are complete; block kb - 1 is done with
      if (kb + 1 < kb1) issue(kb + 1, st ^ 1);
      kc = kc == 2 ? 0 : kc + 1;
      // clear the buffer of block kb + 2, last read for block kb - 1
      unsigned* kclr = keys + (kc == 2 ? 0 : kc + 1) * (BM + BN);
      if (tid < BM + BN) kclr[tid] = 0u;
      if (krem <= 0) continue;   // K == 0: no products
      // past K both operands hold zeros, whose products deposit nothing
      const int kend = (kr + UK - 1) & ~(UK - 1);
      if (dep + kend * D > B::kEndurance) renorm_all();
      const E* ta = sa + ra * NC;
      const E* tb = sb + cb * NC;
      // bound of the thread's entries together, then entry by entry
      unsigned ka = 0, kbm = 0;
#pragma unroll
      for (int i = 0; i < TM; i++) ka = kcur[ra + i] > ka ? kcur[ra + i] : ka;
#pragma unroll
      for (int j = 0; j < TN; j++) kbm = kcur[BM + cb + j] > kbm ? kcur[BM + cb + j] : kbm;
      const unsigned all = B::key(B::mul(key_ceiling<E>(ka), key_ceiling<E>(kbm)));
      bool ok = all < cap;
      if (!ok) {
        ok = true;
#pragma unroll
        for (int i = 0; i < TM; i++)
#pragma unroll
          for (int j = 0; j < TN; j++) {
            const unsigned bound = B::key(
                B::mul(key_ceiling<E>(kcur[ra + i]), key_ceiling<E>(kcur[BM + cb + j])));
#pragma unroll
            for (int c = 0; c < NC; c++) {
              const E p0 = pri[(i * TN + j) * NC + c][0];
              // zeros deposit nothing into a state that is not empty
              ok = ok && (bound < cap_of_pri(p0) || (bound == 0u && p0 != E(0)));
            }
          }
      }
      bool careful = false;
      if (!ok) careful = prepare(ta, tb, kend, all < B::kInfKey, kcur + ra, kcur + BM + cb);
      dep += kend * D;
      if (careful) {
        deposit_careful(ta, tb, kend);
        continue;
      }
#pragma unroll 1
      for (int k = 0; k < kend; k += UK) {
#pragma unroll
        for (int q = 0; q < UK; q++) {
          E a[TM * NC], b[TN * NC];
          load_ab(ta, tb, k + q, a, b);
#pragma unroll
          for (int i = 0; i < TM; i++)
#pragma unroll
            for (int j = 0; j < TN; j++)
#pragma unroll
              for (int c = 0; c < NC; c++) {
                E p[D];
                prods(a, b, i, j, c, p);
#pragma unroll
                for (int d = 0; d < D; d++) deposit((i * TN + j) * NC + c, p[d]);
              }
        }
      }
    }
  }

  // Finish the entries of the whole tile at (m0, n0). With first < last the tile was cut: the
  // partial states of the other CTAs of [first, last] (in slot(v) of the scratch) are merged first.
  template <class Slot>
  __device__ __forceinline__ void finish(const XGemmArgs<E>& g, long long m0, long long n0,
                                         const E* scratch, long long first, long long last,
                                         long long self, Slot slot) {
    const int ra = (threadIdx.x >> 4) * TM, cb = (threadIdx.x & 15) * TN;
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
      for (int j = 0; j < TN; j++) {
        const long long gi = m0 + ra + i, gj = n0 + cb + j;
        if (gi < g.M && gj < g.N) {
          Acc<E, F> a[NC];
#pragma unroll
          for (int c = 0; c < NC; c++) get((i * TN + j) * NC + c, a[c]);
          if (first < last) {
#pragma unroll
            for (int c = 0; c < NC; c++) {
              SumAcc<E, F> sum;
              sum.zero();
              sum.add(a[c]);
#pragma unroll 2
              for (long long v = first; v <= last; v++) {
                if (v == self) continue;
                const E* rec = scratch + slot(v) * (long long)G::PART + threadIdx.x;
                Acc<E, F> o;
                xb::read_rec<E, F>(o, rec + (size_t)((i * TN + j) * NC + c) * G::REC * kThreads, kThreads);
                sum.add(o);
              }
              sum.get(a[c]);
            }
          }
          const long long off = gi * g.sci + gj * g.scj;
          xb::finish<E, CX, F>(a, g.mode, g.C + off * NC, g.br, g.bi, g.Cbin + off * 2 * F * NC);
        }
      }
  }

  // Save the tile's partial state (records of 2F+1 reals per accumulator, thread-minor).
  __device__ __forceinline__ void save(E* rec) {
#pragma unroll
    for (int e = 0; e < NA; e++) {
      Acc<E, F> a;
      get(e, a);
      xb::put_rec<E, F>(a, rec + (size_t)e * G::REC * kThreads + threadIdx.x, kThreads);
    }
  }
};

// One CTA per share of the units (see GemmPlan): its range of units meets whole tiles, which it
// finishes, and at most two cut ones, which leave a partial state in slot 2*cta (the first
// tile of its range) or 2*cta + 1 (its last); the last CTA to arrive at a cut tile merges
// the others' states into its own and finishes the tile.
template <typename E, bool CX, int F, int TM, int TN>
__global__ void __launch_bounds__(kThreads, 2)
gemm_kernel(const __grid_constant__ XGemmArgs<E> g, const __grid_constant__ GemmPlan pl) {
  using T = Tile<E, CX, F, TM, TN>;
  using G = typename T::G;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ unsigned s_last;
  T t;
  t.attach(smem);
  auto start = [&](long long v) { return v * pl.units / pl.grid; };
  const long long cta = blockIdx.x, x1 = start(cta + 1);
  long long x = start(cta);
  const long long x0 = x;
#pragma unroll 1
  while (x < x1) {
    const long long tile = x / pl.nkb, kb0 = x - tile * pl.nkb;
    const long long kb1 = pl.nkb - kb0 < x1 - x ? pl.nkb : kb0 + (x1 - x);
    const long long m0 = tile / pl.ntn * T::BM, n0 = tile % pl.ntn * T::BN;
    t.zero(g, m0, n0);
    t.reduce(g, m0, n0, kb0, kb1);
    bool last = true;
    long long fc = cta, lc = cta;
    const long long u0 = tile * pl.nkb;
    if (kb0 != 0 || kb1 != pl.nkb) {
      t.save((E*)pl.scratch + (2 * cta + (x == x0 ? 0 : 1)) * (long long)G::PART);
      // CTAs that hold the tile's first and last unit
      fc = ((u0 + 1) * pl.grid - 1) / pl.units;
      lc = ((u0 + pl.nkb) * pl.grid - 1) / pl.units;
      __threadfence();
      __syncthreads();
      if (threadIdx.x == 0) {
        const unsigned tk = atomicAdd(pl.tickets + tile, 1u);
        s_last = tk == (unsigned)(lc - fc) ? 1u : 0u;
        if (s_last) pl.tickets[tile] = 0u;
      }
      __syncthreads();
      last = s_last != 0;
      if (last) __threadfence();
      __syncthreads();   // s_last is reused by the next cut tile
    }
    if (last)
      t.finish(g, m0, n0, (const E*)pl.scratch, fc, lc, cta,
               [&](long long v) { return 2 * v + (start(v) >= u0 ? 0 : 1); });
    x += kb1 - kb0;
  }
}

// CTAs of a kernel that fit the device at once (queried once per device; the query also opts
// the kernel in to its shared memory).
template <typename E, bool CX, int F, int TM, int TN>
cudaError_t resident_ctas(int sms, int* out) {
  constexpr int kMaxDevices = 64;
  static std::atomic<int> cache[kMaxDevices];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  int per = dev < kMaxDevices ? cache[dev].load(std::memory_order_relaxed) : 0;
  if (per == 0) {
    const size_t smem = Geo<E, CX, F, TM, TN>::SMEM;
    e = cudaFuncSetAttribute(gemm_kernel<E, CX, F, TM, TN>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, gemm_kernel<E, CX, F, TM, TN>, kThreads,
                                                        smem);
    if (e != cudaSuccess) return e;
    if (per < 1) per = 1;
    if (dev < kMaxDevices) cache[dev].store(per, std::memory_order_relaxed);
  }
  *out = per * sms;
  return cudaSuccess;
}

// Tile shapes per element type and fold: as many accumulators as 128 registers hold beside the
// operands, without spills at folds 2 and 3 (FP64 complex 1x2 spills 20 bytes at fold 4). Issue cycles
// per fold-3 product at 2048^3 (real) / 1024^3
// (complex): FP64 2x2 24.3, 4x2 24.8 (spills); FP32 2x4 14.8, 4x2 15.2, 4x4 15.3 (spills), 2x2
// 16.5; FP64 complex 1x2 22.7, 1x1 24.2, 2x2 24.5 (spills); FP32 complex 2x2 13.9, 2x4 14.3, and at
// fold 8, 700^3, 2x2 2204 us (596 bytes spilled), 1x2 1481. Three
// CTAs per SM (80 registers) spill: FP64 2x2 29.7. The small shape serves sizes that fill the
// large tile badly; `ratio` is its cost per product against the large one's.
template <typename E, bool CX, int F>
struct Shapes {
  static constexpr bool f32 = sizeof(E) == 4;
  static constexpr int TM = CX ? (f32 && F <= 6 ? 2 : 1) : f32 ? 2 : (F <= 6 ? 2 : 1);
  static constexpr int TN = CX ? (f32 || F <= 5 ? 2 : 1) : f32 ? 4 : 2;
  static constexpr int SM = TM > 1 && TN <= 2 ? TM / 2 : TM, SN = TM > 1 && TN <= 2 ? TN : TN > 1 ? TN / 2 : 1;
  static constexpr double ratio = 1.12;
};

// Decomposition for one tile shape; returns its cost estimate in K-block units of the large
// tile's work per CTA slot.
template <typename E, bool CX, int F, int TM, int TN>
cudaError_t plan_shape(long long M, long long N, long long K, int sms, bool whole, GemmPlan* p,
                       double* cost) {
  using G = Geo<E, CX, F, TM, TN>;
  int slots = 0;
  cudaError_t e = resident_ctas<E, CX, F, TM, TN>(sms, &slots);
  if (e != cudaSuccess) return e;
  const long long ntm = (M + G::BM - 1) / G::BM;
  p->ntn = (N + G::BN - 1) / G::BN;
  p->tiles = ntm * p->ntn;
  p->nkb = K > 0 ? (K + G::BK - 1) / G::BK : 1;
  p->units = p->tiles * p->nkb;
  // Whole tiles: waves of CTAs. Cut tiles: an even share of the units, plus (in units) one for
  // the partial states and the tickets -- more where whole tiles would not even take one CTA per
  // SM, whose units are short -- and about a quarter per state merged.
  const double over = p->tiles <= sms ? 2.5 : 1.0;
  double best = (double)((p->tiles + slots - 1) / slots) * p->nkb;
  long long grid = p->tiles;
  if (!whole) {
    auto consider = [&](long long gr) {
      if (gr <= 0 || gr > slots || gr >= p->units) return;
      if (p->units % gr == 0 && (p->units / gr) % p->nkb == 0) return;   // whole tiles
      const double share = (double)((p->units + gr - 1) / gr);
      const double c = share + over + 0.25 * (p->nkb / share + 1.0);
      if (c < 0.97 * best) {
        best = c;
        grid = gr;
      }
    };
    if (p->tiles < slots)
      for (long long parts = slots / p->tiles; parts >= 2; parts = parts * 3 / 4) consider(p->tiles * parts);
    consider(slots);
  }
  p->grid = (int)grid;
  p->cut = grid != p->tiles;
  p->scratch_bytes = p->cut ? (size_t)2 * grid * G::PART * sizeof(E) : 0;
  *cost = best * TM * TN;
  return cudaSuccess;
}

template <typename E, bool CX, int F>
cudaError_t plan_gemm(long long M, long long N, long long K, int sms, bool whole, GemmPlan* p) {
  using Sh = Shapes<E, CX, F>;
  *p = GemmPlan{};
  double c0 = 0;
  cudaError_t e = plan_shape<E, CX, F, Sh::TM, Sh::TN>(M, N, K, sms, whole, p, &c0);
  if (e != cudaSuccess) return e;
  p->shape = 0;
  GemmPlan q{};
  double c1 = 0;
  e = plan_shape<E, CX, F, Sh::SM, Sh::SN>(M, N, K, sms, whole, &q, &c1);
  if (e != cudaSuccess) return e;
  if (Sh::ratio * c1 < c0) {
    *p = q;
    p->shape = 1;
  }
  return cudaSuccess;
}

template <typename E, bool CX, int F>
cudaError_t launch_gemm(const XGemmArgs<E>& g, const GemmPlan& p, cudaStream_t s) {
  using Sh = Shapes<E, CX, F>;
  if (p.shape == 1)
    gemm_kernel<E, CX, F, Sh::SM, Sh::SN><<<p.grid, kThreads, Geo<E, CX, F, Sh::SM, Sh::SN>::SMEM, s>>>(g, p);
  else
    gemm_kernel<E, CX, F, Sh::TM, Sh::TN><<<p.grid, kThreads, Geo<E, CX, F, Sh::TM, Sh::TN>::SMEM, s>>>(g, p);
  return cudaGetLastError();
}

}  // namespace gt
}  // namespace rb
