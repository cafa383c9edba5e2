// fb_kernels.cu -- line-kernel dispatch and the FP64 table generators.
//
// A "line" is one 1-D transform of length L held in shared memory.  A block
// holds G lines; each line is processed by T threads.  The kernel
//   1. loads its lines (gathering strided elements, zero-filling absent ones,
//      multiplying by an optional per-element table -- the Bluestein chirp),
//   2. runs a Stockham stage program in shared memory (radix 2/3/4/5/8/16
//      and odd-prime butterflies up to 71), in place: every stage reads its
//      butterflies into registers, synchronises, then writes,
//   3. optionally multiplies by a pointwise table and runs a second program in
//      the opposite direction (the Bluestein convolution in one kernel),
//   4. stores, fusing the four-step twiddle, an optional per-element table
//      and a scale factor.
// The same kernel serves batched 1-D columns, strided N-D axes, both passes
// of the four-step and all three passes of the multi-pass Bluestein.
//
// The reference computes all of this on the CPU with recursive radix-4 /
// radix-3 / DFT / Bluestein functions (FFTA src/algos.jl:51-424) and a
// Singleton twiddle recurrence (src/singleton_twiddle.jl:25-39); here every
// twiddle comes from a table computed in FP64 and rounded once.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>

#include "fb_device.cuh"
#include "fb_internal.h"

namespace fb {

// ------------------------------------------------------------ prime tables
static const int kPrimes[] = {7, 11, 13, 17, 19, 23, 29, 31, 37, 41, 43, 47, 53, 59, 61, 67, 71};
static const int kNumPrimes = sizeof(kPrimes) / sizeof(kPrimes[0]);

int prime_table_offset(int p) {
  int off = 0;
  for (int i = 0; i < kNumPrimes; ++i) {
    if (kPrimes[i] == p) return off;
    off += kPrimes[i];
  }
  return -1;
}
int prime_table_total() {
  int off = 0;
  for (int i = 0; i < kNumPrimes; ++i) off += kPrimes[i];
  return off;
}

const FastFn* fast_table_f32_0(int*);
const FastFn* fast_table_f32_1(int*);
const FastFn* fast_table_f32_2(int*);
const FastFn* fast_table_f32_3(int*);
const FastFn* fast_table_f64_0(int*);
const FastFn* fast_table_f64_1(int*);
const FastFn* fast_table_f64_2(int*);
const FastFn* fast_table_f64_3(int*);

int fast_table_parts() { return 4; }
const FastFn* fast_table(int dtype, int part, int* count) {
  typedef const FastFn* (*Get)(int*);
  static const Get f32[4] = {fast_table_f32_0, fast_table_f32_1, fast_table_f32_2,
                             fast_table_f32_3};
  static const Get f64[4] = {fast_table_f64_0, fast_table_f64_1, fast_table_f64_2,
                             fast_table_f64_3};
  if (part < 0 || part >= 4) {
    *count = 0;
    return nullptr;
  }
  return (dtype == 0 ? f32 : f64)[part](count);
}

#define FB_DESC_DECL(tag)                                                                 \
  cudaError_t launch_desc_##tag(const LineArgs*, const int64_t*, int, int64_t, int, size_t, \
                                cudaStream_t);
FB_DESC_DECL(f32_c16)
FB_DESC_DECL(f32_c32)
FB_DESC_DECL(f32_big)
FB_DESC_DECL(f64_c16)
FB_DESC_DECL(f64_c32)
FB_DESC_DECL(f64_big)
#undef FB_DESC_DECL

cudaError_t launch_desc(int dtype, int variant, const LineArgs* descs, const int64_t* bstart,
                        int ndesc, int64_t nblocks, int threads, size_t smem, cudaStream_t s) {
  const bool cap32 = variant & 1, big = variant & 2;
  if (dtype == 0) {
    if (big) return launch_desc_f32_big(descs, bstart, ndesc, nblocks, threads, smem, s);
    return cap32 ? launch_desc_f32_c32(descs, bstart, ndesc, nblocks, threads, smem, s)
                 : launch_desc_f32_c16(descs, bstart, ndesc, nblocks, threads, smem, s);
  }
  if (big) return launch_desc_f64_big(descs, bstart, ndesc, nblocks, threads, smem, s);
  return cap32 ? launch_desc_f64_c32(descs, bstart, ndesc, nblocks, threads, smem, s)
               : launch_desc_f64_c16(descs, bstart, ndesc, nblocks, threads, smem, s);
}

cudaError_t launch_line_f32_c16(const LineArgs&, size_t, cudaStream_t);
cudaError_t launch_line_f32_c32(const LineArgs&, size_t, cudaStream_t);
cudaError_t launch_line_f32_big(const LineArgs&, size_t, cudaStream_t);
cudaError_t launch_line_f64_c16(const LineArgs&, size_t, cudaStream_t);
cudaError_t launch_line_f64_c32(const LineArgs&, size_t, cudaStream_t);
cudaError_t launch_line_f64_big(const LineArgs&, size_t, cudaStream_t);

thread_local char g_launch_msg[512] = {0};
const char* last_launch_message() { return g_launch_msg; }

size_t line_smem_bytes(int dtype, const LineArgs& a) {
  const size_t es = dtype == 0 ? 8 : 16;
  return (size_t)a.G * line_pitch(a, (int)es) * es + (size_t)5 * a.G * sizeof(int64_t);
}
int line_max_threads() { return 512; }

cudaError_t launch_line(int dtype, int variant, const LineArgs& a, cudaStream_t s) {
  const size_t smem = line_smem_bytes(dtype, a);
  const bool cap32 = variant & 1, big = variant & 2;
  if (dtype == 0) {
    if (big) return launch_line_f32_big(a, smem, s);
    return cap32 ? launch_line_f32_c32(a, smem, s) : launch_line_f32_c16(a, smem, s);
  }
  if (big) return launch_line_f64_big(a, smem, s);
  return cap32 ? launch_line_f64_c32(a, smem, s) : launch_line_f64_c16(a, smem, s);
}

// ------------------------------------------------------------ FP64 tables
// exp(-2 pi i m / N) for integer m, computed in FP64: the index is reduced
// exactly to a quadrant and a fraction <= 1/2 of it, then CUDA's sincospi.
__device__ double2 root_fp64(int64_t m, int64_t N) {
  m %= N;
  if (m < 0) m += N;
  const int64_t m4 = 4 * m;
  const int q = (int)(m4 / N);
  const int64_t rem = m4 - (int64_t)q * N;  // theta = (pi/2)(q + rem/N)
  const bool flip = 2 * rem > N;
  const int64_t rr = flip ? N - rem : rem;
  const double x = (double)rr / (double)N;  // in [0, 1/2]
  double s, c;
  sincospi(0.5 * x, &s, &c);
  const double cq = flip ? s : c, sq = flip ? c : s;  // cos, sin of (pi/2) rem/N
  double ct, st;
  switch (q) {
    case 0: ct = cq; st = sq; break;
    case 1: ct = -sq; st = cq; break;
    case 2: ct = -cq; st = -sq; break;
    default: ct = sq; st = -cq; break;
  }
  return make_double2(ct, -st);
}

template <typename C> __device__ __forceinline__ C from_d2(double2 v);
template <> __device__ __forceinline__ float2 from_d2<float2>(double2 v) {
  return make_float2((float)v.x, (float)v.y);
}
template <> __device__ __forceinline__ double2 from_d2<double2>(double2 v) { return v; }

template <typename C>
__global__ void k_stage_tw(C* out, int R, int64_t Ns, int64_t count) {
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < count;
       idx += (int64_t)gridDim.x * blockDim.x) {
    // r-major: the R-1 twiddles of butterfly k sit Ns apart, so the threads
    // of a warp (consecutive k) read consecutive entries
    const int64_t r = idx / Ns + 1;
    const int64_t k = idx % Ns;
    out[idx] = from_d2<C>(root_fp64(r * k, Ns * R));
  }
}

// out[i*n_ln + l] = exp(-2 pi i (i*l mod N) / N) for i < n_el, l < n_ln.
template <typename C>
__global__ void k_tw_table(C* out, int64_t N, int64_t n_el, int64_t n_ln) {
  const int64_t count = n_el * n_ln;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < count;
       q += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = q / n_ln, l = q % n_ln;
    const unsigned __int128 e = (unsigned __int128)i * (unsigned __int128)l;
    out[q] = from_d2<C>(root_fp64((int64_t)(e % (unsigned __int128)N), N));
  }
}

template <typename C>
__global__ void k_roots(C* out, int64_t N, int64_t step, int64_t count) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < count;
       q += (int64_t)gridDim.x * blockDim.x) {
    const unsigned __int128 e = (unsigned __int128)q * (unsigned __int128)step;
    out[q] = from_d2<C>(root_fp64((int64_t)(e % (unsigned __int128)N), N));
  }
}

// b[n] = exp(i pi sgn p / N), p = n^2 mod 2N (exact), sgn = -dir.
// exp(-i pi p / N) = root(p, 2N); sgn > 0 takes the conjugate.
__device__ double2 chirp_b(int64_t n, int64_t N, int dir) {
  const unsigned __int128 p = ((unsigned __int128)n * (unsigned __int128)n) % (unsigned __int128)(2 * N);
  double2 r = root_fp64((int64_t)p, 2 * N);
  if (-dir > 0) r.y = -r.y;
  return r;
}

template <typename C>
__global__ void k_chirp(C* pre, C* post, double2* bext, int64_t N, int64_t M, int dir) {
  const double invM = 1.0 / (double)M;
  for (int64_t m = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; m < M;
       m += (int64_t)gridDim.x * blockDim.x) {
    if (m < N) {
      const double2 b = chirp_b(m, N, dir);
      if (pre) pre[m] = from_d2<C>(make_double2(b.x, -b.y));
      if (post) post[m] = from_d2<C>(make_double2(b.x * invM, -b.y * invM));
    }
    if (bext) {
      double2 v = make_double2(0.0, 0.0);
      if (m < N)
        v = chirp_b(m, N, dir);
      else if (M - m < N)
        v = chirp_b(M - m, N, dir);
      bext[m] = v;
    }
  }
}

template <typename C>
__global__ void k_convert(C* dst, const double2* src, int64_t n, double scale) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double2 v = src[i];
    dst[i] = from_d2<C>(make_double2(v.x * scale, v.y * scale));
  }
}

__global__ void k_prime_tables(float* f32, double* f64, int total) {
  // walk the prime list: entry e belongs to prime p at offset off
  const int primes[] = {7, 11, 13, 17, 19, 23, 29, 31, 37, 41, 43, 47, 53, 59, 61, 67, 71};
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
    int off = 0, p = 0;
    for (int i = 0; i < 17; ++i) {
      if (e < off + primes[i]) { p = primes[i]; break; }
      off += primes[i];
    }
    const int m = e - off;
    const double2 r = root_fp64(m, p);  // (cos, -sin)
    f64[2 * e] = r.x;
    f64[2 * e + 1] = -r.y;
    f32[2 * e] = (float)r.x;
    f32[2 * e + 1] = (float)(-r.y);
  }
}

static unsigned grid_for(int64_t n) {
  int64_t b = (n + 255) / 256;
  if (b < 1) b = 1;
  if (b > 65535) b = 65535;
  return (unsigned)b;
}

cudaError_t gen_stage_twiddles(int dtype, void* out, int R, int64_t Ns, cudaStream_t s) {
  const int64_t count = (int64_t)(R - 1) * Ns;
  if (count <= 0) return cudaSuccess;
  if (dtype == 0)
    k_stage_tw<float2><<<grid_for(count), 256, 0, s>>>((float2*)out, R, Ns, count);
  else
    k_stage_tw<double2><<<grid_for(count), 256, 0, s>>>((double2*)out, R, Ns, count);
  return cudaGetLastError();
}

cudaError_t gen_roots(int dtype, void* out, int64_t N, int64_t step, int64_t count,
                      cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  if (dtype == 0)
    k_roots<float2><<<grid_for(count), 256, 0, s>>>((float2*)out, N, step, count);
  else
    k_roots<double2><<<grid_for(count), 256, 0, s>>>((double2*)out, N, step, count);
  return cudaGetLastError();
}

cudaError_t gen_tw_table(int dtype, void* out, int64_t N, int64_t n_el, int64_t n_ln,
                         cudaStream_t s) {
  const int64_t count = n_el * n_ln;
  if (count <= 0) return cudaSuccess;
  if (dtype == 0)
    k_tw_table<float2><<<grid_for(count), 256, 0, s>>>((float2*)out, N, n_el, n_ln);
  else
    k_tw_table<double2><<<grid_for(count), 256, 0, s>>>((double2*)out, N, n_el, n_ln);
  return cudaGetLastError();
}

cudaError_t gen_chirp(int dtype, void* pre, void* post, void* bext_c64, int64_t N, int64_t M,
                      int dir, cudaStream_t s) {
  if (dtype == 0)
    k_chirp<float2><<<grid_for(M), 256, 0, s>>>((float2*)pre, (float2*)post, (double2*)bext_c64,
                                                N, M, dir);
  else
    k_chirp<double2><<<grid_for(M), 256, 0, s>>>((double2*)pre, (double2*)post,
                                                 (double2*)bext_c64, N, M, dir);
  return cudaGetLastError();
}

cudaError_t convert_c64(int dtype, void* dst, const void* src_c64, int64_t n, double scale,
                        cudaStream_t s) {
  if (dtype == 0)
    k_convert<float2><<<grid_for(n), 256, 0, s>>>((float2*)dst, (const double2*)src_c64, n, scale);
  else
    k_convert<double2><<<grid_for(n), 256, 0, s>>>((double2*)dst, (const double2*)src_c64, n,
                                                   scale);
  return cudaGetLastError();
}

// ------------------------------------------------------ real transforms
// The helpers of the real transforms on column-major arrays (rank <= 8).
// Their index splits divide by 32-bit reciprocals (Divisor) for arrays of
// fewer than 2^31 elements, in 64 bits beyond: with 64-bit divisions the
// Hermitian extension of 648 x 189 x 46 ran at a seventh of memory speed (92
// us); irfft 231 x 819 x 5 Float32 64.4 -> 53.3 us.
// They are launched early (launch_overlapped): `in` is read by __ldcs alone, or by
// __ldca where a sector or an element is read again (a strided copy, the mirror
// image).
struct Dims {
  int rank;
  int64_t n[8];
  Divisor d[8];  // mul 0: divide in 64 bits
};
static Dims make_dims(int rank, const int64_t* n) {
  Dims g;
  memset(&g, 0, sizeof(g));
  g.rank = rank;
  int64_t total = 1;
  for (int i = 0; i < rank; ++i) {
    g.n[i] = n[i];
    total *= n[i];
  }
  if (total > 0 && total < (int64_t(1) << 31))
    for (int i = 0; i < rank; ++i) g.d[i] = Divisor((uint32_t)n[i]);
  return g;
}
// t = t / n[i]; returns t mod n[i]
__device__ __forceinline__ int64_t take_dim(const Dims& g, int i, int64_t& t) {
  if (g.d[i].mul) {
    const uint32_t x = (uint32_t)t, q = g.d[i].quot(x);
    t = q;
    return x - q * (uint32_t)g.n[i];
  }
  const int64_t k = t % g.n[i];
  t /= g.n[i];
  return k;
}
struct RealGeom {
  Dims dims;        // the full (complex) dims
  int64_t xs[8];    // strides of the half spectra
  int r0;
  int64_t h;        // n/2 + 1 along r0
  uint32_t region;  // bit d: dim d is transformed
};

template <typename R>
__global__ void k_real_to_complex(const R* in, cplx<R>* out, int64_t count) {
  grid_release();
  grid_wait();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < count;
       i += (int64_t)gridDim.x * blockDim.x)
    out[i] = Sc<R>::mk(__ldcs(in + i), R(0));
}

template <typename R>
__global__ void k_complex_to_real(const cplx<R>* in, R* out, int64_t count) {
  grid_release();
  grid_wait();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < count;
       i += (int64_t)gridDim.x * blockDim.x)
    out[i] = __ldcs(in + i).x;
}

// out[sum_d k_d * os[d]] = the real part of in, contiguous in the order of dims
template <typename R>
__global__ void k_real_part(const cplx<R>* in, R* out, PermCopy p, Dims dims) {
  grid_release();
  grid_wait();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < p.count;
       i += (int64_t)gridDim.x * blockDim.x) {
    int64_t t = i, oo = 0;
    for (int d = 0; d < p.rank; ++d) oo += take_dim(dims, d, t) * p.os[d];
    out[oo] = __ldcs(in + i).x;
  }
}

// out (dims with r0 cut to h) <- in (full dims): the first h entries along
// r0; `half` holds (pre, h, post), n the full length along r0
template <typename R>
__global__ void k_extract_half(const cplx<R>* in, cplx<R>* out, Dims half, int64_t n,
                               int64_t count) {
  grid_release();
  grid_wait();
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < count;
       q += (int64_t)gridDim.x * blockDim.x) {
    int64_t t = q;
    const int64_t a = take_dim(half, 0, t), k = take_dim(half, 1, t);
    out[q] = __ldcs(in + (a + half.n[0] * (k + n * t)));
  }
}

// z (full dims) <- Hermitian extension of x (r0 cut to h): entries with index
// k < h along r0 are copied; the others are conj(x at the mirrored index
// (-k mod n) in every transformed dim), the symmetry of a real signal's
// spectrum.
template <typename R>
__global__ void k_herm_extend(const cplx<R>* in, cplx<R>* z, RealGeom g, int64_t total) {
  grid_release();
  grid_wait();
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < total;
       q += (int64_t)gridDim.x * blockDim.x) {
    // offsets of the entry itself and of its mirror image in `in`
    int64_t t = q, src = 0, mir = 0;
    bool mirror = false;
    for (int d = 0; d < g.dims.rank; ++d) {
      const int64_t k = take_dim(g.dims, d, t);
      const int64_t m = ((g.region >> d) & 1) && k ? g.dims.n[d] - k : k;
      if (d == g.r0) mirror = k >= g.h;
      src += k * g.xs[d];
      mir += m * g.xs[d];
    }
    const cplx<R> v = __ldca(in + (mirror ? mir : src));
    z[q] = mirror ? Sc<R>::mk(v.x, -v.y) : v;
  }
}

// The split of the half-length rfft (fast_real_kernel's formulas) as a pass of
// its own, behind a complex plan of length L = n/2 on the real line read as L
// complex values: for halves without a one-kernel real transform.  Thread (k,
// line) handles the outputs k and L-k; a thread keeps w^k for all its lines.
// Bound by memory: one read of the line and one write of the half spectrum.
// The full-length path these lengths took before (real to complex, a transform
// of 2L points, extraction) moved 2.5 times as much.
// Each output is rounded about once, by double arithmetic and double w for
// float data and by sums with their errors (Knuth's two-sum) for double data,
// so that what is left is the error of the transform of length L.
template <typename R> struct Two;  // a sum of two reals, exact
template <> struct Two<float> {
  double v;
};
template <> struct Two<double> {
  double v, e;
};
__device__ __forceinline__ Two<float> exact_sum(float a, float b) {
  return {__dadd_rn((double)a, (double)b)};
}
__device__ __forceinline__ Two<double> exact_sum(double a, double b) {
  const double s = __dadd_rn(a, b), t = __dsub_rn(s, a);
  return {s, __dadd_rn(__dsub_rn(a, __dsub_rn(s, t)), __dsub_rn(b, t))};
}
__device__ __forceinline__ Two<float> half_sum(float a, float b) {
  return {0.5 * exact_sum(a, b).v};
}
__device__ __forceinline__ Two<double> half_sum(double a, double b) {
  const Two<double> s = exact_sum(a, b);
  return {0.5 * s.v, 0.5 * s.e};
}
// x + p a + q b
__device__ __forceinline__ float sum_products(Two<float> x, double p, Two<float> a, double q,
                                              Two<float> b) {
  return __double2float_rn(__fma_rn(p, a.v, __fma_rn(q, b.v, x.v)));
}
__device__ __forceinline__ double sum_products(Two<double> x, double p, Two<double> a, double q,
                                               Two<double> b) {
  const double pa = __dmul_rn(p, a.v), qb = __dmul_rn(q, b.v);
  const Two<double> s = exact_sum(x.v, pa), t = exact_sum(s.v, qb);
  double e = __dadd_rn(__dadd_rn(s.e, t.e), x.e);
  e = __dadd_rn(e, __dadd_rn(__fma_rn(p, a.v, -pa), __fma_rn(q, b.v, -qb)));
  e = __fma_rn(p, a.e, __fma_rn(q, b.e, e));
  return __dsub_rn(e, e) == 0.0 ? __dadd_rn(t.v, e) : t.v;  // infinities: e is not a number
}
template <typename R>
__global__ void __launch_bounds__(256)
    k_real_half(const cplx<R>* in, cplx<R>* out, const double2* __restrict__ wk, int L,
                 int64_t lines, R scale) {
  typedef cplx<R> C;
  typedef Sc<R> S;
  grid_release();
  grid_wait();
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k > L / 2) return;
  const double2 w = __ldg(wk + k);
  for (int64_t l = blockIdx.y * (int64_t)blockDim.y + threadIdx.y; l < lines;
       l += (int64_t)gridDim.y * blockDim.y) {
    const C* z = in + l * L;
    C* o = out + l * (L + 1);
    const C A = __ldcs(z + k);
    if (k == 0) {
      o[0] = S::mk(S::mul(S::add(A.x, A.y), scale), R(0));
      o[L] = S::mk(S::mul(S::sub(A.x, A.y), scale), R(0));
      continue;
    }
    const C B = __ldcs(z + (L - k));
    // XX + w XY and conj(XX - w XY), with XX = (A + conj B)/2 and XY = -i (A -
    // conj B)/2
    const Two<R> xx = half_sum(A.x, B.x), xi = half_sum(A.y, -B.y);
    const Two<R> yx = half_sum(B.y, A.y), yi = half_sum(B.x, -A.x);
    o[k] = cscale<R>(S::mk(sum_products(xx, w.x, yx, -w.y, yi), sum_products(xi, w.x, yi, w.y, yx)),
                     scale);
    if (k != L - k)
      o[L - k] = cscale<R>(S::mk(sum_products(xx, -w.x, yx, w.y, yi),
                                 -sum_products(xi, -w.x, yi, -w.y, yx)), scale);
  }
}

template <typename R>
static cudaError_t real_half_t(const void* in, void* out, const void* wk, int L, int64_t lines,
                               double scale, cudaStream_t s) {
  typedef cplx<R> C;
  int tx = 1;
  while (tx < 256 && tx < L / 2 + 1) tx *= 2;
  const dim3 block(tx, 256 / tx);
  const int64_t gx = (L / 2 + 1 + tx - 1) / tx, want = (lines + block.y - 1) / block.y;
  // about 16 blocks per SM in all: a thread of a long launch reuses its w^k
  const int64_t gy = std::min<int64_t>(std::min<int64_t>(want, 65535),
                                       std::max<int64_t>(1, 16 * kSms / gx));
  return launch_overlapped(true, k_real_half<R>, dim3((unsigned)gx, (unsigned)gy), block, 0, s,
                           (const C*)in, (C*)out, (const double2*)wk, L, lines, (R)scale);
}
cudaError_t real_half(int dtype, const void* in, void* out, const void* wk, int L, int64_t lines,
                      double scale, cudaStream_t s) {
  if (lines <= 0) return cudaSuccess;
  return dtype == 0 ? real_half_t<float>(in, out, wk, L, lines, scale, s)
                    : real_half_t<double>(in, out, wk, L, lines, scale, s);
}

cudaError_t real_to_complex(int dtype, const void* in, void* out, int64_t count, cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  if (dtype == 0)
    return launch_overlapped(true, k_real_to_complex<float>, grid_for(count), 256, 0, s, (const float*)in, (float2*)out, count);
  else
    return launch_overlapped(true, k_real_to_complex<double>, grid_for(count), 256, 0, s, (const double*)in, (double2*)out, count);
}

cudaError_t complex_to_real(int dtype, const void* in, void* out, int64_t count, cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  if (dtype == 0)
    return launch_overlapped(true, k_complex_to_real<float>, grid_for(count), 256, 0, s, (const float2*)in, (float*)out, count);
  else
    return launch_overlapped(true, k_complex_to_real<double>, grid_for(count), 256, 0, s, (const double2*)in, (double*)out, count);
}

cudaError_t real_part(int dtype, const void* in, void* out, const PermCopy& p, cudaStream_t s) {
  if (p.count <= 0) return cudaSuccess;
  const Dims dims = make_dims(p.rank, p.dims);
  if (dtype == 0)
    return launch_overlapped(true, k_real_part<float>, grid_for(p.count), 256, 0, s, (const float2*)in, (float*)out, p, dims);
  else
    return launch_overlapped(true, k_real_part<double>, grid_for(p.count), 256, 0, s, (const double2*)in, (double*)out, p, dims);
}

cudaError_t extract_half(int dtype, const void* in, void* out, int64_t pre, int64_t n, int64_t h,
                         int64_t post, cudaStream_t s) {
  const int64_t count = pre * h * post;
  if (count <= 0) return cudaSuccess;
  const int64_t hd[3] = {pre, h, post};
  const Dims half = make_dims(3, hd);
  if (dtype == 0)
    return launch_overlapped(true, k_extract_half<float>, grid_for(count), 256, 0, s, (const float2*)in, (float2*)out, half, n, count);
  else
    return launch_overlapped(true, k_extract_half<double>, grid_for(count), 256, 0, s, (const double2*)in, (double2*)out, half, n, count);
}

cudaError_t herm_extend(int dtype, const void* x, void* z, int rank, const int64_t* dims,
                        const int64_t* xs, int r0, int64_t h, uint32_t region, cudaStream_t s) {
  RealGeom g;
  memset(&g, 0, sizeof(g));
  g.dims = make_dims(rank, dims);
  for (int d = 0; d < rank; ++d) g.xs[d] = xs[d];
  g.r0 = r0;
  g.h = h;
  g.region = region;
  int64_t total = 1;
  for (int d = 0; d < rank; ++d) total *= dims[d];
  if (total <= 0) return cudaSuccess;
  if (dtype == 0)
    return launch_overlapped(true, k_herm_extend<float>, grid_for(total), 256, 0, s, (const float2*)x, (float2*)z, g, total);
  else
    return launch_overlapped(true, k_herm_extend<double>, grid_for(total), 256, 0, s, (const double2*)x, (double2*)z, g, total);
}

// out[sum_d k_d * os[d]] = in[sum_d k_d * is[d]] for every index (k_d < dims[d]):
// a strided copy that moves an array between two layouts (rank <= 8).
template <typename E>
__global__ void k_permute(const E* in, E* out, PermCopy p, Dims dims) {
  grid_release();
  grid_wait();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < p.count;
       i += (int64_t)gridDim.x * blockDim.x) {
    int64_t t = i, oi = 0, oo = 0;
    for (int d = 0; d < p.rank; ++d) {
      const int64_t k = take_dim(dims, d, t);
      oi += k * p.is[d];
      oo += k * p.os[d];
    }
    out[oo] = __ldca(in + oi);
  }
}

cudaError_t permute_copy(int elem_bytes, const void* in, void* out, const PermCopy& p,
                         cudaStream_t s) {
  if (p.count <= 0) return cudaSuccess;
  const Dims dims = make_dims(p.rank, p.dims);
  switch (elem_bytes) {
    case 4: return launch_overlapped(true, k_permute<float>, grid_for(p.count), 256, 0, s, (const float*)in, (float*)out, p, dims);
    case 8: return launch_overlapped(true, k_permute<float2>, grid_for(p.count), 256, 0, s, (const float2*)in, (float2*)out, p, dims);
    case 16: return launch_overlapped(true, k_permute<double2>, grid_for(p.count), 256, 0, s, (const double2*)in, (double2*)out, p, dims);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t gen_prime_tables(void* f32tab, void* f64tab, cudaStream_t s) {
  const int total = prime_table_total();
  k_prime_tables<<<grid_for(total), 256, 0, s>>>((float*)f32tab, (double*)f64tab, total);
  return cudaGetLastError();
}

}  // namespace fb
