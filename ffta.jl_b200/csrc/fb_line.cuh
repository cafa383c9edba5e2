// fb_line.cuh -- the generic line kernel: any length with prime factors up to
// 71, its radix program read at run time.
//
// A "line" is one 1-D transform of length L.  A block holds G lines; each line
// is processed by T threads.  The kernel
//   1. has its first stage read the line straight from global memory (gathering
//      strided elements, zero-filling absent ones, multiplying by an optional
//      per-element table -- the Bluestein chirp -- or the four-step twiddle); a
//      first stage of a prime of 17 or more finds the line in shared memory,
//   2. runs a Stockham stage program (radix 2/3/4/5/7/8/9/11/13/16 butterflies in
//      registers, primes of 17 to 71 shared by the line's threads) that exchanges
//      its values through shared memory, in place: every stage reads its
//      butterflies into registers, synchronises, then writes,
//   3. optionally multiplies by a pointwise table and runs a second program in
//      the opposite direction (the Bluestein convolution in one kernel),
//   4. has its last stage store straight to global memory (a prime of 17 or more:
//      from shared memory), fusing the four-step twiddle, an optional per-element
//      table and a scale factor.
// The same kernel serves batched 1-D columns, strided N-D axes, both passes
// of the four-step and all three passes of the multi-pass Bluestein.
//
// The reference computes all of this on the CPU with recursive radix-4 /
// radix-3 / DFT / Bluestein functions (FFTA src/algos.jl:51-424) and a
// Singleton twiddle recurrence (src/singleton_twiddle.jl:25-39); here every
// twiddle comes from a table computed in FP64 and rounded once.
#pragma once
#include <cuda_runtime.h>

#include "fb_device.cuh"
#include "fb_internal.h"

namespace fb {

// Elements of a line that are present: i*ves + voff < vn, i.e. i < count.
__device__ __forceinline__ int present_count(int64_t vn, int64_t ves, int64_t voff, bool ok) {
  if (!ok || voff >= vn) return 0;
  if (ves == 0 || vn == INT64_MAX) return INT32_MAX;
  const int64_t c = (vn - voff + ves - 1) / ves;
  return c > INT32_MAX ? INT32_MAX : (int)c;
}
// Batch levels of line l (LineIO): l = q0 + m0*(q1 + m1*q2).  Launches of
// fewer than 2^31 lines divide by 32-bit reciprocals made on the host
// (LineArgs::d0, d1); the 64-bit divisions they replace took about a
// thousand cycles before a block could issue its first load.
__device__ __forceinline__ void split_line(const LineArgs& a, int64_t l, int64_t* q0, int64_t* q1,
                                           int64_t* q2) {
  if (a.d0.mul) {
    const uint32_t x = (uint32_t)l, t = a.d0.quot(x), w = a.d1.quot(t);
    *q0 = x - t * (uint32_t)a.m0;
    *q1 = t - w * (uint32_t)a.m1;
    *q2 = w;
  } else {
    const int64_t t = l / a.m0;
    *q0 = l % a.m0;
    *q1 = t % a.m1;
    *q2 = t / a.m1;
  }
}
// compile-time offsets (must match prime_table_offset)
template <int P> struct POff;
#define FB_POFF(p, o) \
  template <> struct POff<p> { static constexpr int v = o; };
FB_POFF(7, 0)
FB_POFF(11, 7)
FB_POFF(13, 18)
FB_POFF(17, 31)
FB_POFF(19, 48)
FB_POFF(23, 67)
FB_POFF(29, 90)
FB_POFF(31, 119)
FB_POFF(37, 150)
FB_POFF(41, 187)
FB_POFF(43, 228)
FB_POFF(47, 271)
FB_POFF(53, 318)
FB_POFF(59, 371)
FB_POFF(61, 430)
FB_POFF(67, 491)
FB_POFF(71, 558)
#undef FB_POFF

// ---------------------------------------------------------------- stages
template <typename R, int RAD, int DIR>
__device__ __forceinline__ void butterfly(cplx<R>* v, const R* pcs) {
  if constexpr (RAD == 2) {
    bf2<R, DIR>(v[0], v[1]);
  } else if constexpr (RAD == 3) {
    dft3<R, DIR>(v);
  } else if constexpr (RAD == 4) {
    dft4<R, DIR>(v);
  } else if constexpr (RAD == 5) {
    dft5<R, DIR>(v);
  } else if constexpr (RAD == 8) {
    dft8<R, DIR>(v);
  } else if constexpr (RAD == 9) {
    dft9<R, DIR>(v);
  } else if constexpr (RAD == 16) {
    dft16<R, DIR>(v);
  } else {
    dftp<R, DIR, RAD>(v, pcs + 2 * POff<RAD>::v);
  }
}

// ------------------------------------------------------------ I/O
// One line's input or output in global memory.  `cnt` elements are present
// (absent ones load as zero and are not stored); `mul` (the chirp) is read
// at mul + i*ves, the four-step twiddle at tab + i*tab_es, the line's offset
// included in both.  LEAN (LineArgs::plain_io): every element present, no
// chirp and no root tables, 32-bit steps between a butterfly's elements; a twiddle on the loads is
// tw_elem's product instead of the entry itself.  What a pass rarely has is
// applied to the registers in loops of its own, so the straight code between
// loads and stores stays short: with the tests inside the unrolled loops a
// quarter of the kernel's stalls were instruction fetches (no_instruction 3.5
// of 14 cycles per issue).  One B200, before -> after: 6240 x 6 ComplexF32 14.9
// -> 10.6 us, 231 x 3000 11.4 -> 8.8, 176 x 1728 x 5 ComplexF64 40.9 -> 34.9.
template <typename C> __device__ __forceinline__ C* step_ptr(C* p, int step, int r) {
  // p + r*step elements: a 32 x 32 -> 64 bit product added to the address
  return (C*)((uintptr_t)p + (uint64_t)((int64_t)step * (int64_t)(r * (int)sizeof(C))));
}
template <bool LEAN, typename C>
__device__ __forceinline__ C* row_ptr(C* p, int64_t step, int r) {
  if constexpr (LEAN)
    return step_ptr(p, (int)step, r);
  else
    return p + step * r;
}
template <typename R, bool LEAN> struct GenIn {
  const cplx<R>* __restrict__ base;
  int64_t es;
  int cnt;
  const cplx<R>* __restrict__ mul;
  int64_t ves;
  const cplx<R>* __restrict__ tab;  // twiddle on load, or null
  int64_t tab_es;
  int tw_dir;

  // inputs j + r*nb of a butterfly: every data load is issued before any
  // table load
  template <int RAD> __device__ __forceinline__ void load(int j, int nb, cplx<R>* v) const {
    const cplx<R>* p = base + j * es;
#pragma unroll
    for (int r = 0; r < RAD; ++r)
      v[r] = LEAN || j + r * nb < cnt ? __ldcs(row_ptr<LEAN>(p, nb * es, r))
                                      : Sc<R>::mk(R(0), R(0));
  }
  template <int RAD> __device__ __forceinline__ void finish(int j, int nb, cplx<R>* v) const {
    if (!LEAN && mul) {
      const cplx<R>* p = mul + j * ves;
#pragma unroll
      for (int r = 0; r < RAD; ++r)
        if (j + r * nb < cnt) v[r] = cmul<R>(v[r], __ldg(p + r * (nb * ves)));
    }
    if (!tab) return;
    const int64_t ts = nb * tab_es;
    const cplx<R>* p = tab + j * tab_es;
    auto apply = [&](int r, cplx<R> w) {
      if (LEAN || j + r * nb < cnt) v[r] = tw_dir < 0 ? cmul<R>(v[r], w) : cmulc<R>(v[r], w);
    };
    if constexpr (LEAN && RAD >= 4) {
      cplx<R> s[4];
#pragma unroll
      for (int c = 1; c < 4; ++c) s[c] = __ldg(row_ptr<LEAN>(tab, ts, c));
#pragma unroll
      for (int a = 0; a < RAD; a += 4) {
        const cplx<R> b = __ldg(row_ptr<LEAN>(p, ts, a));
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (a + c < RAD) apply(a + c, c == 0 ? b : cmul<R>(b, s[c]));
      }
    } else {
#pragma unroll
      for (int r = 0; r < RAD; ++r)
        if (LEAN || j + r * nb < cnt) apply(r, __ldg(row_ptr<LEAN>(p, ts, r)));
    }
  }
  // element i alone (loads staged through shared memory); nb and rad of the
  // program's first stage
  __device__ __forceinline__ cplx<R> one(int i, int nb, int rad) const {
    if (!LEAN && i >= cnt) return Sc<R>::mk(R(0), R(0));
    cplx<R> v = __ldcs(base + i * es);
    if (!LEAN && mul) v = cmul<R>(v, __ldg(mul + i * ves));
    if (tab) {
      auto at = [&](int k) { return __ldg(tab + k * tab_es); };
      const cplx<R> w = LEAN ? tw_elem<R>(at, i, nb, rad) : at(i);
      v = tw_dir < 0 ? cmul<R>(v, w) : cmulc<R>(v, w);
    }
    return v;
  }
};

template <typename R, bool LEAN> struct GenOut {
  cplx<R>* __restrict__ base;
  int64_t es;
  int cnt;
  const cplx<R>* __restrict__ mul;
  int64_t ves;
  const cplx<R>* __restrict__ tab;
  int64_t tab_es;
  const cplx<R>* __restrict__ tw_hi;  // root tables, or null
  const cplx<R>* __restrict__ tw_lo;
  int64_t lt;  // the line's twiddle index
  int tw_shift, tw_dir;
  R scale;
  bool ok, cs;

  // outputs e0 + r*st of a butterfly
  template <int RAD> __device__ __forceinline__ void store(int e0, int st, cplx<R>* v) const {
    if (LEAN && !ok) return;
    auto here = [&](int r) { return LEAN || e0 + r * st < cnt; };
    auto twiddle = [&](int r, cplx<R> w) {
      v[r] = tw_dir < 0 ? cmul<R>(v[r], w) : cmulc<R>(v[r], w);
    };
    if (!LEAN && mul) {
#pragma unroll
      for (int r = 0; r < RAD; ++r)
        if (here(r)) v[r] = cmul<R>(v[r], __ldg(mul + (e0 + r * st) * ves));
    }
    if (tab) {
      const cplx<R>* p = tab + e0 * tab_es;
#pragma unroll
      for (int r = 0; r < RAD; ++r)
        if (here(r)) twiddle(r, __ldg(row_ptr<LEAN>(p, st * tab_es, r)));
    } else if (!LEAN && tw_hi) {
#pragma unroll
      for (int r = 0; r < RAD; ++r)
        if (here(r)) twiddle(r, root(e0 + r * st));
    }
    if (scale != R(1)) {
#pragma unroll
      for (int r = 0; r < RAD; ++r) v[r] = cscale<R>(v[r], scale);
    }
    cplx<R>* p = base + e0 * es;
#pragma unroll
    for (int r = 0; r < RAD; ++r)
      if (here(r)) write(row_ptr<LEAN>(p, st * es, r), v[r]);
  }
  __device__ __forceinline__ void one(int i, cplx<R> v) const {
    if (LEAN ? !ok : i >= cnt) return;
    if (!LEAN && mul) v = cmul<R>(v, __ldg(mul + i * ves));
    if (tab || (!LEAN && tw_hi)) {
      const cplx<R> w = tab ? __ldg(tab + i * tab_es) : root(i);
      v = tw_dir < 0 ? cmul<R>(v, w) : cmulc<R>(v, w);
    }
    if (scale != R(1)) v = cscale<R>(v, scale);
    write(base + i * es, v);
  }
  __device__ __forceinline__ cplx<R> root(int i) const {
    const int64_t e = lt * (int64_t)i;
    return cmul<R>(__ldg(tw_hi + (e >> tw_shift)),
                   __ldg(tw_lo + (e & ((int64_t(1) << tw_shift) - 1))));
  }
  __device__ __forceinline__ void write(cplx<R>* p, cplx<R> v) const {
    if (cs)
      __stcs(p, v);
    else
      *p = v;
  }
};

// A line's I/O made from the launch's arguments and the block's per-line
// values in shared memory when a stage needs it (held across the stages it
// would take 35 registers): lb holds five arrays of G -- offsets of the input
// and output, first batch level, twiddle index, elements present on load and
// (upper half) on store.
template <typename R, bool LEAN> struct LineCtx {
  const LineArgs& a;
  const int64_t* lb;
  __device__ __forceinline__ GenIn<R, LEAN> input(int g) const {
    typedef cplx<R> C;
    const int G = a.G;
    const bool tw = a.tw_on_load && a.tw_tab;
    return GenIn<R, LEAN>{(const C*)a.in + lb[g], a.ld.es, (int)lb[4 * G + g],
                          !LEAN && a.ld.mul ? (const C*)a.ld.mul + lb[2 * G + g] * a.ld.vls
                                            : nullptr,
                          a.ld.ves, tw ? (const C*)a.tw_tab + lb[3 * G + g] * a.tw_ls : nullptr,
                          a.tw_es, a.tw_dir};
  }
  __device__ __forceinline__ GenOut<R, LEAN> output(int g) const {
    typedef cplx<R> C;
    const int G = a.G;
    const int64_t lt = lb[3 * G + g];
    const bool tab = a.tw_tab && !a.tw_on_load;
    const int cnt = (int)(lb[4 * G + g] >> 32);
    return GenOut<R, LEAN>{(C*)a.out + lb[G + g], a.st.es, cnt,
                           !LEAN && a.st.mul ? (const C*)a.st.mul + lb[2 * G + g] * a.st.vls
                                             : nullptr,
                           a.st.ves, tab ? (const C*)a.tw_tab + lt * a.tw_ls : nullptr, a.tw_es,
                           !LEAN && a.tw_N ? (const C*)a.tw_hi : nullptr, (const C*)a.tw_lo, lt,
                           a.tw_shift, a.tw_dir, (R)a.scale, cnt > 0, a.st_stream != 0};
  }
};

// ---------------------------------------------------------------- stages
// k = j mod Ns through the stage's reciprocal.
__device__ __forceinline__ int mod_ns(int j, int Ns, Divisor d) {
  return j - (int)d.quot((uint32_t)j) * Ns;
}

// One Stockham stage of radix RAD on a line of length L.  Ns is the product
// of the radices already applied.  Butterfly j (k = j mod Ns) reads
// x[j + r*L/RAD], twiddles input r by w_{Ns*RAD}^(r k), and writes
// y[(j-k)*RAD + k + r*Ns].  The line is held in `buf` (padded layout),
// updated in place; the first stage may read the line's input and the last
// one write its output instead (ld, st), which saves one trip through shared memory each.
// What bounds it: instruction issue and the barriers between stages.  The
// values now stay in registers (see v below); before, every stage of every
// program ran through 2.3 KB of local memory per thread, 2.6 times the
// algorithmic traffic at 7168 points.  One B200, before -> after, same bits:
// 23100 x 256 ComplexF32 (100 x 231) 178.6 -> 116.9 us (78.0 with the lean
// form below), 176 x 1728 x 5
// ComplexF64 158.1 -> 47.2, 6240 x 6 22.5 -> 16.4, irfft 648 x 189 x 46
// 295.6 -> 224.2.
template <typename R, int RAD, int DIR, int CAP, bool LEAN>
__device__ __forceinline__ void stage(cplx<R>* buf, int L, int Ns, Divisor nsd,
                                      const cplx<R>* __restrict__ tw, const R* pcs, int u, int T,
                                      bool ld, bool st, const LineCtx<R, LEAN>& io, int g) {
  constexpr int UM = (RAD >= CAP) ? 1 : CAP / RAD;
  const int nb = L / RAD;
  // Defined for every butterfly, present or not: inside the loop over the
  // stages the values of all switch cases would otherwise count as carried
  // over from the previous iteration, all of them alive at once (2.2 KB of
  // spills per thread).
  cplx<R> v[UM][RAD];
#pragma unroll
  for (int q = 0; q < UM; ++q)
#pragma unroll
    for (int r = 0; r < RAD; ++r) v[q][r] = Sc<R>::mk(R(0), R(0));
  if (st && !ld) grid_release();
  if (ld) {
    const GenIn<R, LEAN> in = io.input(g);
#pragma unroll
    for (int q = 0; q < UM; ++q) {
      const int j = u + q * T;
      if (j < nb) in.template load<RAD>(j, nb, v[q]);
    }
#pragma unroll
    for (int q = 0; q < UM; ++q) {
      const int j = u + q * T;
      if (j < nb) in.template finish<RAD>(j, nb, v[q]);
    }
    if (st) grid_release();
  } else {
#pragma unroll
    for (int q = 0; q < UM; ++q) {
      const int j = u + q * T;
      if (j < nb) {
        const GenSlots sl(j, nb);
#pragma unroll
        for (int r = 0; r < RAD; ++r) v[q][r] = buf[sl[r]];
      }
    }
    // in place: all reads of the line finish before any write
    if (!st) __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < UM; ++q) {
    const int j = u + q * T;
    if (j < nb) {
      int k = 0;
      if (Ns > 1) {
        k = mod_ns(j, Ns, nsd);
        const cplx<R>* w = tw + k;  // entry (r-1)*Ns + k
#pragma unroll
        for (int r = 1; r < RAD; ++r) v[q][r] = ctw<R, DIR>(v[q][r], __ldg(w + (r - 1) * Ns));
      }
      butterfly<R, RAD, DIR>(v[q], pcs);
      const int base = (j - k) * RAD + k;
      if (st) {
        io.output(g).template store<RAD>(base, Ns, v[q]);
      } else {
        const GenSlots sl(base, Ns);
#pragma unroll
        for (int r = 0; r < RAD; ++r) buf[sl[r]] = v[q][r];
      }
    }
  }
  if (!st) __syncthreads();
}

// A stage of odd prime radix P >= 17: too many values for one thread, so the
// T threads of the line share each butterfly.  First the twiddled inputs are
// replaced in place by a_k = x_k + x_{P-k} and b_k = x_k - x_{P-k}; then
// thread (j, ml) computes the output pairs m = ml, ml + T/nb, ... of butterfly
// j, X_{m, P-m} = (x_0 + sum_k a_k cos(2 pi m k / P)) +- i dir (sum_k b_k sin),
// reading each a_k, b_k once for all its pairs.  A thread holds at most PAIRS
// pairs: T/nb * PAIRS > H (line_threads sees to it for kPrimePairs).  The sums
// run in the order of dftp, with the same operations.  The one-thread form
// indexed its values in a loop and so kept them in local memory: a
// 59-point transform took 97 us.
template <typename R, int DIR, int PAIRS>
__device__ __forceinline__ void stage_prime(cplx<R>* buf, int L, int P, int Ns, Divisor nsd,
                                            const cplx<R>* __restrict__ tw,
                                            const R* __restrict__ cs, int u, int T) {
  typedef Sc<R> S;
  typedef cplx<R> C;
  const int nb = L / P, H = (P - 1) / 2;
  for (int t = u; t < nb * H; t += T) {
    const int j = t % nb, k = t / nb + 1;
    const int s0 = padi(j + k * nb), s1 = padi(j + (P - k) * nb);
    C x = buf[s0], y = buf[s1];
    if (Ns > 1) {
      const C* w = tw + mod_ns(j, Ns, nsd);
      x = ctw<R, DIR>(x, __ldg(w + (k - 1) * Ns));
      y = ctw<R, DIR>(y, __ldg(w + (P - k - 1) * Ns));
    }
    buf[s0] = cadd<R>(x, y);
    buf[s1] = csub<R>(x, y);
  }
  __syncthreads();
  const int ML = T / nb, j = u % nb, ml = u / nb;
  const bool mine = ml < ML && ml <= H;
  C A[PAIRS], B[PAIRS];
  int idx[PAIRS];
#pragma unroll
  for (int q = 0; q < PAIRS; ++q) A[q] = B[q] = S::mk(R(0), R(0));  // as in stage
  if (mine) {
    const C x0 = buf[padi(j)];
#pragma unroll
    for (int q = 0; q < PAIRS; ++q) {
      A[q] = x0;
      B[q] = S::mk(R(0), R(0));
      idx[q] = 0;
    }
#pragma unroll 1
    for (int k = 1; k <= H; ++k) {
      const C a = buf[padi(j + k * nb)], b = buf[padi(j + (P - k) * nb)];
#pragma unroll
      for (int q = 0; q < PAIRS; ++q) {
        const int m = ml + q * ML;
        if (m <= H) {
          idx[q] += m;
          if (idx[q] >= P) idx[q] -= P;
          const C w = __ldg((const C*)cs + idx[q]);  // (cos, sin) of 2 pi idx / P
          A[q] = S::mk(S::fma(w.x, a.x, A[q].x), S::fma(w.x, a.y, A[q].y));
          B[q] = S::mk(S::fma(w.y, b.x, B[q].x), S::fma(w.y, b.y, B[q].y));
        }
      }
    }
  }
  __syncthreads();  // every read of the line is done
  if (mine) {
    const int k = Ns > 1 ? mod_ns(j, Ns, nsd) : 0;
    const int base = (j - k) * P + k;
#pragma unroll
    for (int q = 0; q < PAIRS; ++q) {
      const int m = ml + q * ML;
      if (m == 0) {
        buf[padi(base)] = A[q];
      } else if (m <= H) {
        const C rb = rot<R, DIR>(B[q]);
        buf[padi(base + m * Ns)] = cadd<R>(A[q], rb);
        buf[padi(base + (P - m) * Ns)] = csub<R>(A[q], rb);
      }
    }
  }
  __syncthreads();
}

// (cos, sin) table of prime P inside prime_cs, or -1 for no prime 17..71.
__device__ __forceinline__ int big_prime_offset(int P) {
  switch (P) {
    case 17: return POff<17>::v;
    case 19: return POff<19>::v;
    case 23: return POff<23>::v;
    case 29: return POff<29>::v;
    case 31: return POff<31>::v;
    case 37: return POff<37>::v;
    case 41: return POff<41>::v;
    case 43: return POff<43>::v;
    case 47: return POff<47>::v;
    case 53: return POff<53>::v;
    case 59: return POff<59>::v;
    case 61: return POff<61>::v;
    case 67: return POff<67>::v;
    case 71: return POff<71>::v;
    default: return -1;
  }
}

// The stages of program p.  ld: the first stage reads the line's input; st:
// the last one writes its output; else the line is in `buf` before and after.
template <typename R, int DIR, int CAP, bool BIG, bool LEAN>
__device__ __forceinline__ void run_prog(cplx<R>* buf, const StageProg& p, const R* pcs, int u,
                                         int T, int* err, bool ld, bool st,
                                         const LineCtx<R, LEAN>& io, int g) {
  const cplx<R>* twb = (const cplx<R>*)p.tw;
  int Ns = 1, L = p.L;
#pragma unroll 1
  for (int s = 0; s < p.nst; ++s) {
    const int rad = p.radix[s];
    const cplx<R>* tw = twb + p.tw_off[s];
    const Divisor d = p.nsd[s];
    const bool l = ld && s == 0, t = st && s == p.nst - 1;
    // The slots a stage reads depend on (u, T, L, radix) alone; left visible
    // as loop invariants, those of every radix are computed before the loop
    // and spilled (2.2 KB per thread).  The empty statement makes u and L
    // values of this iteration.
    asm volatile("" : "+r"(u), "+r"(L));
    switch (rad) {
      case 2: stage<R, 2, DIR, CAP, LEAN>(buf, L, Ns, d, tw, pcs, u, T, l, t, io, g); break;
      case 3: stage<R, 3, DIR, CAP, LEAN>(buf, L, Ns, d, tw, pcs, u, T, l, t, io, g); break;
      case 4: stage<R, 4, DIR, CAP, LEAN>(buf, L, Ns, d, tw, pcs, u, T, l, t, io, g); break;
      case 5: stage<R, 5, DIR, CAP, LEAN>(buf, L, Ns, d, tw, pcs, u, T, l, t, io, g); break;
      case 7: stage<R, 7, DIR, CAP, LEAN>(buf, L, Ns, d, tw, pcs, u, T, l, t, io, g); break;
      case 8: stage<R, 8, DIR, CAP, LEAN>(buf, L, Ns, d, tw, pcs, u, T, l, t, io, g); break;
      case 9: stage<R, 9, DIR, CAP, LEAN>(buf, L, Ns, d, tw, pcs, u, T, l, t, io, g); break;
      case 11: stage<R, 11, DIR, CAP, LEAN>(buf, L, Ns, d, tw, pcs, u, T, l, t, io, g); break;
      case 13: stage<R, 13, DIR, CAP, LEAN>(buf, L, Ns, d, tw, pcs, u, T, l, t, io, g); break;
      case 16: stage<R, 16, DIR, CAP, LEAN>(buf, L, Ns, d, tw, pcs, u, T, l, t, io, g); break;
      default: {
        const int off = BIG ? big_prime_offset(rad) : -1;
        if (off >= 0) {
          if constexpr (BIG) {
            if (T / (L / rad) * 8 > rad / 2)
              stage_prime<R, DIR, 8>(buf, L, rad, Ns, d, tw, pcs + 2 * off, u, T);
            else
              stage_prime<R, DIR, kPrimePairs>(buf, L, rad, Ns, d, tw, pcs + 2 * off, u, T);
          }
        } else if (threadIdx.x == 0 && threadIdx.y == 0 && err) {
          atomicExch(err, rad);
        }
      }
    }
    Ns *= rad;
  }
}

// ----------------------------------------------------------------- kernel
// One block's work: lines block*G .. block*G + G-1 of `a`.  Thread (u, g) is
// butterfly lane u of line g; tid = g*T + u.  Threads of a block beyond T*G
// pass u = kIdle (no butterflies, no elements) and tid = T*G, and only take
// part in the barriers.
//
// Where a pass's lines are neighbours in memory (element-major: ld.mode or
// st.mode 1; G is a power of two) the lines run fastest across the threads,
// g = tid mod G, and the line pitch spreads them over the banks.  The first
// stage reads and the last stage writes global memory directly.  Where one
// side's lines are contiguous (the rows of a four-step's second pass) an
// element-major block holds G lines such that a warp still covers whole
// 32-byte sectors of each (pick_G); staging those loads through shared memory
// instead formed the four-step twiddle element by element, 80 instructions
// each: 23100 x 256 ComplexF32 116.9 -> 102.8 us.
//
// OVERLAPPED: launched by launch_overlapped.
constexpr int kIdle = 1 << 29;

template <typename R, int CAP, bool BIG, bool LEAN, bool OVERLAPPED>
__device__ __forceinline__ void line_body(const LineArgs& a, int64_t block, int u, int g, int tid,
                                          unsigned char* smraw) {
  typedef cplx<R> C;
  C* sm = (C*)smraw;
  const int T = a.T, G = a.G, L = a.prog.L;
  const int nthr = G * T;
  const int64_t line0 = block * G;
  const int Lp = line_pitch(a, (int)sizeof(C));
  const bool em = elem_major(a);
  if (em && tid < nthr) {
    g = tid & (G - 1);
    u = tid >> (__ffs(G) - 1);
  }
  int64_t* lb = (int64_t*)(sm + (size_t)G * Lp);
  if (tid < G) {
    const int64_t l = line0 + tid;
    const bool ok = l < a.nlines;
    int64_t l0, l1, l2;
    split_line(a, ok ? l : 0, &l0, &l1, &l2);
    lb[tid] = l0 * a.ld.s0 + l1 * a.ld.s1 + l2 * a.ld.s2;
    lb[G + tid] = l0 * a.st.s0 + l1 * a.st.s1 + l2 * a.st.s2;
    lb[2 * G + tid] = l0;
    lb[3 * G + tid] = a.tw_level ? l1 : l0;
    lb[4 * G + tid] =
        (int64_t)min(present_count(a.ld.vn, a.ld.ves, l0 * a.ld.vls, ok), ok ? a.ld.count : 0) |
        (int64_t)min(present_count(a.st.vn, a.st.ves, l0 * a.st.vls, ok), ok ? a.st.count : 0) << 32;
  }
  if constexpr (OVERLAPPED) grid_wait();
  __syncthreads();
  const LineCtx<R, LEAN> io{a, lb};
  // direct I/O: not for the prime stages, which work in shared memory, nor
  // for an empty program (a copy)
  const bool direct = a.prog.nst > 0;
  const bool ld = direct && a.prog.radix[0] <= 16;
  const bool st = direct && a.prog.radix[a.prog.nst - 1] <= 16;
  C* buf = sm + g * Lp;
  const R* pcs = (const R*)a.prime_cs;
  const int rad0 = direct ? a.prog.radix[0] : 1, nb0 = L / rad0;
  if (!ld) {
    if (a.ld.mode == 1) {  // (em) line fastest
      const GenIn<R, LEAN> src = io.input(g);
      for (int i = u; i < L; i += T) buf[padi(i)] = src.one(i, nb0, rad0);
    } else {               // element fastest, whatever the thread order
      const int gg = tid / T, uu = tid - gg * T;
      if (gg < G) {
        const GenIn<R, LEAN> src = io.input(gg);
        C* d = sm + gg * Lp;
        for (int i = uu; i < L; i += T) d[padi(i)] = src.one(i, nb0, rad0);
      }
    }
    __syncthreads();
  }
  // One program, or (Bluestein) program -> pointwise multiply -> program in
  // the other direction.  The loop keeps one inlined copy per direction.
  const int npass = !LEAN && a.mid ? 2 : 1;
#pragma unroll 1
  for (int ps = 0; ps < npass; ++ps) {
    const bool l = ld && ps == 0, t = st && ps == npass - 1;
    if ((ps == 0 ? a.dir1 : a.dir2) < 0)
      run_prog<R, -1, CAP, BIG, LEAN>(buf, a.prog, pcs, u, T, a.err, l, t, io, g);
    else
      run_prog<R, 1, CAP, BIG, LEAN>(buf, a.prog, pcs, u, T, a.err, l, t, io, g);
    if (!LEAN && ps == 0 && a.mid) {
      const C* __restrict__ mid = (const C*)a.mid;
      const int64_t l0 = lb[2 * G + g];
      for (int k = u; k < L; k += T)
        buf[padi(k)] = cmul<R>(buf[padi(k)], __ldg(mid + l0 * a.mid_ls + (int64_t)k * a.mid_es));
      __syncthreads();
    }
  }
  if (!st) {
    grid_release();
    if (a.st.mode == 1 || !em) {
      const GenOut<R, LEAN> dst = io.output(g);
      for (int i = u; i < L; i += T) dst.one(i, buf[padi(i)]);
    } else {
      const int gg = tid / T, uu = tid - gg * T;
      if (gg < G) {
        const GenOut<R, LEAN> dst = io.output(gg);
        const C* d = sm + gg * Lp;
        for (int i = uu; i < L; i += T) dst.one(i, d[padi(i)]);
      }
    }
  }
}

// Two blocks of 512 threads per SM for ComplexF32 with 16 values per thread.
template <typename R, int CAP, bool BIG> struct LineBounds {
  static constexpr int min_blocks = sizeof(R) == 4 && CAP == 16 && !BIG ? 2 : 1;
};
template <typename R, int CAP, bool BIG, bool LEAN>
__global__ void __launch_bounds__(512, LineBounds<R, CAP, BIG>::min_blocks) line_kernel(const __grid_constant__ LineArgs a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int u = threadIdx.x, g = threadIdx.y;
  line_body<R, CAP, BIG, LEAN, true>(a, blockIdx.x, u, g, g * a.T + u, smraw);
}

// Work-descriptor launch: many line transforms -- different lengths,
// directions, pointers -- in one grid.  Descriptor r owns blocks
// bstart[r] .. bstart[r+1]-1 and is run by the generic body with its own
// T x G shape inside the launch's one-dimensional block.
template <typename R, int CAP, bool BIG>
__global__ void __launch_bounds__(512, LineBounds<R, CAP, BIG>::min_blocks)
    line_kernel_desc(const LineArgs* __restrict__ descs, const int64_t* __restrict__ bstart,
                     int ndesc) {
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ LineArgs sa;
  __shared__ int64_t sblock;
  if (threadIdx.x == 0) {
    int lo = 0, hi = ndesc - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (__ldg(bstart + mid) <= (int64_t)blockIdx.x)
        lo = mid;
      else
        hi = mid - 1;
    }
    sa = descs[lo];
    sblock = (int64_t)blockIdx.x - __ldg(bstart + lo);
  }
  __syncthreads();
  const int nthr = sa.T * sa.G;
  const bool active = (int)threadIdx.x < nthr;
  const int u = active ? (int)threadIdx.x % sa.T : kIdle;
  const int g = active ? (int)threadIdx.x / sa.T : 0;
  line_body<R, CAP, BIG, false, false>(sa, sblock, u, g, active ? (int)threadIdx.x : nthr, smraw);
}

}  // namespace fb
