// Batched DST-I and the Dirichlet spectral solvers built on it
// (moljax/core/fft_nonperiodic.py:97-162, 244-330, 360-398).
//
// DST-I of x[0..N-1]:  X[k] = sum_n x[n] sin(pi (k+1)(n+1) / (N+1)).
// As in dst_I_fast, it is read off the DFT of the odd extension of length
// M = 2(N+1):  z = [0, x, 0, -reverse(x)],  X[k] = -Im(DFT(z))[k+1] / 2.
// Two real rows a, b ride one complex sequence z = a_ext + i b_ext:
// DFT(z)[k] = 2 S_b[k] - 2i S_a[k], so S_a = -Im/2 and S_b = Re/2.
//
// When M is a power of two the DFT is the tile Stockham FFT; for any
// other M it is Bluestein's chirp-z form, a circular convolution of length
// L = 2^ceil(log2(2M - 1)) done with two FFTs of length L:
//   DFT_M(z)[k] = c[k] * IFFT_L( FFT_L(z c) * FFT_L(b) )[k],
//   c[n] = exp(-i pi n^2 / M),  b[n] = conj(c[|n|]) for |n| < M (periodic in L).
// The plan holds the length-L twiddles, c, FFT_L(b) / L and sin^2(pi k / (2(N+1))).
//
// One CTA transforms a tile of row pairs (tfft.cuh); the Helmholtz, Poisson and ETD1 solvers multiply the coefficients
// and run the same transform again (DST-I is its own inverse up to 2/(N+1)).
#include <math.h>
#include <string.h>

#include <vector>

#include "tfft.cuh"

namespace mjx {

mjx_status ensure_kernel_attrs();
int elem_size(int dtype);
void set_last_error(cudaError_t e, const char* file, int line);

enum { DST_PLAIN = 0, DST_HELMHOLTZ = 1, DST_POISSON = 2, DST_ETD1 = 3 };
enum { DCT_FWD = 0, DCT_INV = 1, DCT_HELMHOLTZ = 2, DCT_POISSON = 3, DCT_ETD1 = 4 };

static inline size_t a256(size_t b) { return (b + 255) & ~size_t(255); }

struct Dst1Geom {
  int N, M, L, log2L, bluestein;
  size_t tw, chirp, bhat, shift, total;  // plan byte offsets (per element size)
};

// kind 0: DST-I, DFT length M = 2(N+1); kind 1: DCT-II, M = 2N (plus the N phase factors)
static Dst1Geom dst1_geom(int N, int elem, int kind = 0) {
  Dst1Geom g;
  g.N = N;
  g.M = kind == 0 ? 2 * (N + 1) : 2 * N;
  g.bluestein = ilog2_exact(g.M) < 0;
  g.L = g.M;
  if (g.bluestein) {
    g.L = 1;
    while (g.L < 2 * g.M - 1) g.L <<= 1;
  }
  g.log2L = ilog2_exact(g.L);
  const size_t c = 2 * (size_t)elem;
  size_t o = 0;
  g.tw = o; o += a256((g.L + (elem == 4 ? fft_pass_entries(g.L) : 0)) * c);
  g.chirp = o; o += a256(g.M * c);
  g.bhat = o; o += a256(g.L * c);
  g.shift = o; o += kind == 0 ? 0 : a256(N * c);
  g.total = o;
  return g;
}

// ---------------------------------------------------------------- FP32
// One radix-16 butterfly per thread and pass, in place: FP32 is not bound by its arithmetic, and
// half the shared memory and three passes instead of four beat the flat tile (3000 rows of 600,
// L = 4096: 148 us against 213 us; 300 rows of 200: 36 against 39 us).
struct Dst32Args {
  const float* x;       // rows of N values (mode ETD1: rows u, then rows of N(u) at offset nrows*N)
  float* out;
  const float* lam;     // per-mode symbol of length N (Helmholtz/Poisson: laplacian_symbol; ETD1: eigenvalues)
  const float2* tw;  // length-L twiddles
  const float2* chirp;
  const float2* bhat;
  long long nrows;  // rows to transform
  int N, M, L, log2L, bluestein, nseq, mode;
  float scale;          // output scale of a plain transform
  double h, D;      // Helmholtz: dt, D; ETD1: dt
};

// DFT of length M of each sequence in buf (segments of L), in place in [0, M).
__device__ void dft_m(const Dst32Args& a, float2* buf, int s_loc, int lt, int tps, int tid) {
  typedef float2 C;
  const int L = a.L;
  if (!a.bluestein) {
    fft_smem<float, false, false>(buf, L, a.log2L, a.nseq, L, 1, a.tw, tid);
    return;
  }
  const int base = s_loc * L;
  const bool active = s_loc < a.nseq;
  if (active)
    for (int j = lt; j < L; j += tps) {
      const C v = buf[sp(base + j)];
      buf[sp(base + j)] = j < a.M ? cmul(v, __ldg(&a.chirp[j])) : mk<C>(0.f, 0.f);
    }
  __syncthreads();
  fft_smem<float, false, false>(buf, L, a.log2L, a.nseq, L, 1, a.tw, tid);
  if (active)
    for (int j = lt; j < L; j += tps) buf[sp(base + j)] = cmul(buf[sp(base + j)], __ldg(&a.bhat[j]));
  __syncthreads();
  fft_smem<float, true, false>(buf, L, a.log2L, a.nseq, L, 1, a.tw, tid);
  if (active)
    for (int j = lt; j < a.M; j += tps) buf[sp(base + j)] = cmul(buf[sp(base + j)], __ldg(&a.chirp[j]));
  __syncthreads();
}

// odd extension of (va, vb) into the sequence: z[0] = z[N+1] = 0, z[j] = v[j-1], z[M-j] = -v[j-1]
__device__ __forceinline__ void put_odd(float2* buf, int base, int N, int M, int j, float va, float vb) {
  typedef float2 C;
  buf[sp(base + j + 1)] = mk<C>(va, vb);
  buf[sp(base + M - 1 - j)] = mk<C>(-va, -vb);
}

__global__ void __launch_bounds__(256) dst1_kernel32(const __grid_constant__ Dst32Args a) {
  typedef float2 C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);
  const int L = a.L, M = a.M, N = a.N;
  const int tps = L >= 16 ? L / 16 : 1;
  const int tid = threadIdx.x, s_loc = tid / tps, lt = tid % tps;
  const bool active = s_loc < a.nseq;
  const int base = s_loc * L;
  // sequence q holds rows 2q and 2q+1 (ETD1: row q of u and of N(u))
  const long long q = (long long)blockIdx.x * a.nseq + s_loc;
  const bool etd = a.mode == DST_ETD1;
  const long long ra = etd ? q : 2 * q, rb = etd ? a.nrows + q : 2 * q + 1;
  const long long nr_a = a.nrows;  // rows available for a (and for b, except ETD1)
  const bool has_a = active && ra < nr_a;
  const bool has_b = active && (etd ? q < a.nrows : rb < nr_a);

  if (active) {
    if (lt == 0) { buf[sp(base)] = mk<C>(0.f, 0.f); buf[sp(base + N + 1)] = mk<C>(0.f, 0.f); }
    for (int j = lt; j < N; j += tps) {
      const float va = has_a ? a.x[ra * N + j] : (float)0;
      const float vb = has_b ? a.x[rb * N + j] : (float)0;
      put_odd(buf, base, N, M, j, va, vb);
    }
  }
  __syncthreads();
  dft_m(a, buf, s_loc, lt, tps, tid);

  if (a.mode != DST_PLAIN) {
    // coefficients S_a, S_b -> multiplied coefficients, written back as a new odd extension
    float ca[16], cb[16];  // N <= 2047 and tps >= L/16 >= N/8, so each thread owns <= 16 entries
    int cnt = 0;
    if (active)
      for (int j = lt; j < N; j += tps, ++cnt) {
        const C Z = buf[sp(base + j + 1)];
        const float sa = (float)-0.5 * Z.y, sb = (float)0.5 * Z.x;
        const float lam = a.lam[j];
        const float inv = (float)2 / (float)(N + 1);
        if (a.mode == DST_HELMHOLTZ) {
          const float m = (float)1 / ((float)1 - (float)(a.h * a.D) * lam);  // fft_nonperiodic.py:327-330
          ca[cnt] = sa * m * inv; cb[cnt] = sb * m * inv;
        } else if (a.mode == DST_POISSON) {
          ca[cnt] = sa / lam * inv; cb[cnt] = sb / lam * inv;  // 265-271
        } else {  // ETD1 (360-398): exp(z) u^ + dt phi1(z) N^, z = dt * eigenvalue
          const float z = (float)a.h * lam;
          const float ez = exp(z);
          const float phi1 = fabs(z) < (float)1e-4 ? (float)1 + z / (float)2 + z * z / (float)6 : (ez - (float)1) / z;
          ca[cnt] = (ez * sa + (float)a.h * phi1 * sb) * inv; cb[cnt] = (float)0;
        }
      }
    __syncthreads();
    if (active) {
      cnt = 0;
      for (int j = lt; j < N; j += tps, ++cnt) put_odd(buf, base, N, M, j, ca[cnt], cb[cnt]);
      if (lt == 0) {
        buf[sp(base)] = mk<C>(0.f, 0.f);
        buf[sp(base + N + 1)] = mk<C>(0.f, 0.f);
      }
    }
    __syncthreads();
    dft_m(a, buf, s_loc, lt, tps, tid);
  }

  if (active) {
    const float sc = a.mode == DST_PLAIN ? a.scale : (float)1;
    for (int j = lt; j < N; j += tps) {
      const C Z = buf[sp(base + j + 1)];
      if (has_a) a.out[ra * N + j] = (float)-0.5 * Z.y * sc;
      if (has_b && !etd) a.out[rb * N + j] = (float)0.5 * Z.x * sc;
    }
  }
}

__global__ void __launch_bounds__(256) dct2_kernel32(const __grid_constant__ Dst32Args a,
                                                   const float2* __restrict__ shift) {
  typedef float2 C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);
  const int L = a.L, M = a.M, N = a.N;
  const int tps = L >= 16 ? L / 16 : 1;
  const int tid = threadIdx.x, s_loc = tid / tps, lt = tid % tps;
  const bool active = s_loc < a.nseq;
  const int base = s_loc * L;
  const long long q = (long long)blockIdx.x * a.nseq + s_loc;
  const bool etd = a.mode == DCT_ETD1;
  const long long ra = etd ? q : 2 * q, rb = etd ? a.nrows + q : 2 * q + 1;
  const bool has_a = active && ra < a.nrows;
  const bool has_b = active && (etd ? q < a.nrows : rb < a.nrows);
  const float f0 = (float)sqrt(0.25 / N), fk = (float)sqrt(0.5 / N);  // forward ortho factors
  const float w0 = (float)sqrt(1.0 / N), wk = (float)sqrt(2.0 / N);   // inverse ortho factors
  float ca[16], cb[16];  // this thread's coefficients k = lt + m tps (N <= 8 tps)

  if (a.mode != DCT_INV) {
    if (active)
      for (int j = lt; j < N; j += tps) {
        const float va = has_a ? a.x[ra * N + j] : (float)0, vb = has_b ? a.x[rb * N + j] : (float)0;
        buf[sp(base + j)] = mk<C>(va, vb);
        buf[sp(base + M - 1 - j)] = mk<C>(va, vb);
      }
    __syncthreads();
    dft_m(a, buf, s_loc, lt, tps, tid);
    int m = 0;
    if (active)
      for (int k = lt; k < N; k += tps, ++m) {
        const C t = cmul(buf[sp(base + k)], __ldg(&shift[k]));
        const float f = k == 0 ? f0 : fk;
        ca[m] = t.x * f; cb[m] = t.y * f;
      }
  } else {
    int m = 0;
    if (active)
      for (int k = lt; k < N; k += tps, ++m) {
        ca[m] = has_a ? a.x[ra * N + k] : (float)0;
        cb[m] = has_b ? a.x[rb * N + k] : (float)0;
      }
  }
  if (a.mode == DCT_FWD) {
    int m = 0;
    if (active)
      for (int k = lt; k < N; k += tps, ++m) {
        if (has_a) a.out[ra * N + k] = ca[m] * a.scale;
        if (has_b) a.out[rb * N + k] = cb[m] * a.scale;
      }
    return;
  }
  if (a.mode != DCT_INV) {  // spectral multipliers
    int m = 0;
    if (active)
      for (int k = lt; k < N; k += tps, ++m) {
        const float lam = a.lam[k];
        if (a.mode == DCT_HELMHOLTZ) {  // fft_nonperiodic.py:352-355
          const float mu = (float)1 / ((float)1 - (float)(a.h * a.D) * lam);
          ca[m] *= mu; cb[m] *= mu;
        } else if (a.mode == DCT_POISSON) {  // 297-303: the null mode is set to zero
          const bool null = fabs(lam) < (float)1e-14;
          ca[m] = null ? (float)0 : ca[m] / lam; cb[m] = null ? (float)0 : cb[m] / lam;
        } else {  // ETD1 (431-437): exp(z) u^ + dt phi1(z) N^
          const float z = (float)a.h * lam, ez = exp(z);
          const float phi1 = fabs(z) < (float)1e-4 ? (float)1 + z / (float)2 + z * z / (float)6 : (ez - (float)1) / z;
          ca[m] = ez * ca[m] + (float)a.h * phi1 * cb[m];
          cb[m] = (float)0;
        }
      }
  }
  // inverse: conj of the Hermitian spectrum, forward DFT, conj back
  __syncthreads();
  if (active) {
    for (int j = lt; j < L; j += tps) buf[sp(base + j)] = mk<C>(0.f, 0.f);
  }
  __syncthreads();
  if (active) {
    int m = 0;
    for (int k = lt; k < N; k += tps, ++m) {
      const C X = mk<C>(ca[m], cb[m]);
      if (k == 0) {
        buf[sp(base)] = cconj(cscale(X, w0));
      } else {
        const C sh = __ldg(&shift[k]);         // e^{-i pi k / 2N}
        const C zk = cscale(cmulc(X, sh), (float)0.5 * wk);  // (wk/2) e^{+i..} X
        const C zm = cscale(cmul(X, sh), (float)0.5 * wk);   // (wk/2) e^{-i..} X
        buf[sp(base + k)] = cconj(zk);
        buf[sp(base + M - k)] = cconj(zm);
      }
    }
  }
  __syncthreads();
  dft_m(a, buf, s_loc, lt, tps, tid);
  if (active) {
    const float sc = a.mode == DCT_INV ? a.scale : (float)1;
    for (int j = lt; j < N; j += tps) {
      const C z = buf[sp(base + j)];  // conj(DFT(conj Z)) = inverse DFT of Z
      if (has_a) a.out[ra * N + j] = z.x * sc;
      if (has_b && !etd) a.out[rb * N + j] = -z.y * sc;
    }
  }
}

// ---------------------------------------------------------------- FP64
template <typename T>
struct Dst1Args {
  Dft<T> d;         // the DFT of length M
  const T* x;       // rows of N values (mode ETD1: rows u, then rows of N(u) at offset nrows*N)
  T* out;
  const T* lam;     // per-mode symbol of length N (Helmholtz/Poisson: laplacian_symbol; ETD1: eigenvalues)
  long long nrows;  // rows to transform
  int N, M, lS, mode;
  T scale;          // output scale of a plain transform
  double h, D;      // Helmholtz: dt, D; ETD1: dt
};

// Sequence q holds rows 2q and 2q + 1 (ETD1: row q of u and of N(u)).
template <typename T>
__device__ __forceinline__ cx<T> load_pair(const Dst1Args<T>& a, bool etd, long long q, int j) {
  const long long ra = etd ? q : 2 * q, rb = etd ? a.nrows + q : 2 * q + 1;
  const bool has_a = ra < a.nrows, has_b = etd ? q < a.nrows : rb < a.nrows;
  return mk<cx<T>>(has_a ? a.x[ra * a.N + j] : (T)0, has_b ? a.x[rb * a.N + j] : (T)0);
}
template <typename T>
__device__ __forceinline__ void store_pair(const Dst1Args<T>& a, bool etd, long long q, int j, T va, T vb) {
  const long long ra = etd ? q : 2 * q, rb = ra + 1;
  if (ra < a.nrows) a.out[ra * a.N + j] = va;
  if (!etd && rb < a.nrows) a.out[rb * a.N + j] = vb;
}

// The transform of S = 2^lS row pairs per CTA, all butterflies and points of the tile flat over
// the threads.  16 pairs per CTA and radix-16 butterflies kept two SMs and a part of their
// sub-partitions busy on 64 rows of 100 FP64 points: 180 us a solve; one pair per CTA here,
// 39 us.  What bounds it: FP64 issue of the SMs that hold a pair.
template <typename T>
__global__ void __launch_bounds__(512) dst1_kernel(const __grid_constant__ Dst1Args<T> a) {
  typedef cx<T> C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int M = a.M, N = a.N, lS = a.lS, S = 1 << lS, tid = threadIdx.x, nth = blockDim.x;
  const float rN = 1.0f / (float)N;
  const long long q0 = (long long)blockIdx.x << lS;
  const bool etd = a.mode == DST_ETD1;
  Tile<T> t = tile_begin<T>(a.d, smem_raw, lS);
  // odd extension: z[0] = z[N+1] = 0, z[j+1] = v[j], z[M-1-j] = -v[j]
  for (int s = tid; s < S; s += nth) t.cur[sp(s)] = t.cur[sp(((N + 1) << lS) + s)] = mk<C>((T)0, (T)0);
  for (int e = tid; e < S * N; e += nth) {
    const int s = fdiv(e, rN), j = e - s * N;
    const C v = load_pair<T>(a, etd, q0 + s, j);
    t.cur[sp(((j + 1) << lS) + s)] = v;
    t.cur[sp(((M - 1 - j) << lS) + s)] = mk<C>(-v.x, -v.y);
  }
  __syncthreads();
  dft_tile<T>(a.d, t);

  if (a.mode != DST_PLAIN) {
    // coefficients S_a = -Im/2, S_b = Re/2 -> multiplied, written back as a new odd extension
    // (in place: only points 1 .. N are read, each by the thread that replaces it)
    const T inv = (T)2 / (T)(N + 1);
    for (int s = tid; s < S; s += nth) t.cur[sp(s)] = t.cur[sp(((N + 1) << lS) + s)] = mk<C>((T)0, (T)0);
    for (int e = tid; e < (N << lS); e += nth) {
      const int j = e >> lS, s = e & (S - 1);
      const C Z = t.cur[sp(((j + 1) << lS) + s)];
      const T sa = (T)-0.5 * Z.y, sb = (T)0.5 * Z.x;
      const T lam = a.lam[j];
      T ca, cb;
      if (a.mode == DST_HELMHOLTZ) {
        const T m = (T)1 / ((T)1 - (T)(a.h * a.D) * lam);  // fft_nonperiodic.py:327-330
        ca = sa * m * inv; cb = sb * m * inv;
      } else if (a.mode == DST_POISSON) {
        ca = sa / lam * inv; cb = sb / lam * inv;  // 265-271
      } else {  // ETD1 (360-398): exp(z) u^ + dt phi1(z) N^, z = dt * eigenvalue
        const T z = (T)a.h * lam;
        const T ez = exp(z);
        const T phi1 = fabs(z) < (T)1e-4 ? (T)1 + z / (T)2 + z * z / (T)6 : (ez - (T)1) / z;
        ca = (ez * sa + (T)a.h * phi1 * sb) * inv; cb = (T)0;
      }
      t.cur[sp(((j + 1) << lS) + s)] = mk<C>(ca, cb);
      t.cur[sp(((M - 1 - j) << lS) + s)] = mk<C>(-ca, -cb);
    }
    __syncthreads();
    dft_tile<T>(a.d, t);
  }

  const T sc = a.mode == DST_PLAIN ? a.scale : (T)1;
  for (int e = tid; e < S * N; e += nth) {
    const int s = fdiv(e, rN), j = e - s * N;
    const C Z = t.cur[sp(((j + 1) << lS) + s)];
    store_pair<T>(a, etd, q0 + s, j, (T)-0.5 * Z.y * sc, (T)0.5 * Z.x * sc);
  }
}

// ---------------------------------------------------------------- DCT-II (orthonormal)
// jax.scipy.fft.dct(x, type=2, norm='ortho') and its inverse along rows of N values
// (the Neumann solvers, fft_nonperiodic.py:274-305, 333-355, 401-437).  Forward: the
// even extension v = [x, reverse(x)] of length M = 2N gives
//   2 sum_n x[n] cos(pi k (2n+1) / 2N) = Re(e^{-i pi k / 2N} DFT(v)[k]),
// and for a row pair z = a + i b the real and imaginary parts separate.  Inverse: the
// Hermitian spectrum Z[0] = w0 X0, Z[k] = (wk/2) e^{+i pi k/2N} Xk, Z[2N-k] = conj,
// transformed back (inverse DFT = conj(DFT(conj(.)))), returns both rows of a pair.

template <typename T>
__global__ void __launch_bounds__(512) dct2_kernel(const __grid_constant__ Dst1Args<T> a,
                                                   const cx<T>* __restrict__ shift) {
  typedef cx<T> C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int M = a.M, N = a.N, lS = a.lS, S = 1 << lS, tid = threadIdx.x, nth = blockDim.x;
  const float rN = 1.0f / (float)N;
  const long long q0 = (long long)blockIdx.x << lS;
  const bool etd = a.mode == DCT_ETD1;
  const T f0 = (T)sqrt(0.25 / N), fk = (T)sqrt(0.5 / N);  // forward ortho factors
  const T w0 = (T)sqrt(1.0 / N), wk = (T)sqrt(2.0 / N);   // inverse ortho factors
  Tile<T> t = tile_begin<T>(a.d, smem_raw, lS);

  if (a.mode != DCT_INV) {
    for (int e = tid; e < S * N; e += nth) {
      const int s = fdiv(e, rN), j = e - s * N;
      const C v = load_pair<T>(a, etd, q0 + s, j);
      t.cur[sp((j << lS) + s)] = v;
      t.cur[sp(((M - 1 - j) << lS) + s)] = v;
    }
    __syncthreads();
    dft_tile<T>(a.d, t);
    if (a.mode == DCT_FWD) {
      for (int e = tid; e < S * N; e += nth) {
        const int s = fdiv(e, rN), k = e - s * N;
        const C c = cmul(t.cur[sp((k << lS) + s)], __ldg(&shift[k]));
        const T f = k == 0 ? f0 : fk;
        store_pair<T>(a, etd, q0 + s, k, c.x * f * a.scale, c.y * f * a.scale);
      }
      return;
    }
  }
  // coefficients, spectral multipliers and the conjugate of the Hermitian spectrum (in place:
  // only points 0 .. N - 1 are read, each by the thread that replaces it)
  for (int e = tid; e < S * N; e += nth) {
    const int s = fdiv(e, rN), k = e - s * N;
    const C sh = __ldg(&shift[k]);  // e^{-i pi k / 2N}
    C X;
    if (a.mode == DCT_INV) {
      X = load_pair<T>(a, false, q0 + s, k);
    } else {
      const C c = cmul(t.cur[sp((k << lS) + s)], sh);
      const T f = k == 0 ? f0 : fk;
      X = mk<C>(c.x * f, c.y * f);
      const T lam = a.lam[k];
      if (a.mode == DCT_HELMHOLTZ) {  // fft_nonperiodic.py:352-355
        const T mu = (T)1 / ((T)1 - (T)(a.h * a.D) * lam);
        X.x *= mu; X.y *= mu;
      } else if (a.mode == DCT_POISSON) {  // 297-303: the null mode is set to zero
        const bool null = fabs(lam) < (T)1e-14;
        X = null ? mk<C>((T)0, (T)0) : mk<C>(X.x / lam, X.y / lam);
      } else {  // ETD1 (431-437): exp(z) u^ + dt phi1(z) N^
        const T z = (T)a.h * lam, ez = exp(z);
        const T phi1 = fabs(z) < (T)1e-4 ? (T)1 + z / (T)2 + z * z / (T)6 : (ez - (T)1) / z;
        X = mk<C>(ez * X.x + (T)a.h * phi1 * X.y, (T)0);
      }
    }
    if (k == 0) {
      t.cur[sp(s)] = cconj(cscale(X, w0));
      t.cur[sp((N << lS) + s)] = mk<C>((T)0, (T)0);
    } else {
      const C zk = cscale(cmulc(X, sh), (T)0.5 * wk);  // (wk/2) e^{+i..} X
      const C zm = cscale(cmul(X, sh), (T)0.5 * wk);   // (wk/2) e^{-i..} X
      t.cur[sp((k << lS) + s)] = cconj(zk);
      t.cur[sp(((M - k) << lS) + s)] = cconj(zm);
    }
  }
  __syncthreads();
  dft_tile<T>(a.d, t);
  const T sc = a.mode == DCT_INV ? a.scale : (T)1;
  for (int e = tid; e < S * N; e += nth) {
    const int s = fdiv(e, rN), j = e - s * N;
    const C z = t.cur[sp((j << lS) + s)];  // conj(DFT(conj Z)) = inverse DFT of Z
    store_pair<T>(a, etd, q0 + s, j, z.x * sc, -z.y * sc);
  }
}

// FP32 launch: sequences per CTA to 256 threads, fewer until every SM has a CTA
static Dst32Args trig_args32(const Dst1Geom& g, const char* p, long long nrows, long long nseq_total, int mode,
                             const float* x, float* out, const float* lam, double h, double D, float scale) {
  Dst32Args a;
  memset(&a, 0, sizeof(a));
  a.x = x; a.out = out; a.lam = lam;
  a.tw = (const float2*)(p + g.tw); a.chirp = (const float2*)(p + g.chirp); a.bhat = (const float2*)(p + g.bhat);
  a.nrows = nrows; a.N = g.N; a.M = g.M; a.L = g.L; a.log2L = g.log2L; a.bluestein = g.bluestein;
  a.mode = mode; a.scale = scale; a.h = h; a.D = D;
  const int tps = g.L >= 16 ? g.L / 16 : 1;
  a.nseq = 256 / tps;
  if (a.nseq < 1) a.nseq = 1;
  while (a.nseq > 1 && (nseq_total + a.nseq - 1) / a.nseq < 152) a.nseq >>= 1;
  return a;
}

template <typename T>
static Dst1Args<T> trig_args(const Dst1Geom& g, const char* p, long long nrows, int mode, const T* x, T* out,
                             const T* lam, double h, double D, T scale) {
  Dst1Args<T> a;
  memset(&a, 0, sizeof(a));
  a.x = x; a.out = out; a.lam = lam;
  a.d.tw = (const cx<T>*)(p + g.tw); a.d.chirp = (const cx<T>*)(p + g.chirp); a.d.bhat = (const cx<T>*)(p + g.bhat);
  a.d.n = g.M; a.d.L = g.L; a.d.bluestein = g.bluestein;
  a.d.log2L = g.log2L;
  a.d.tps = g.L / 8 < 1 ? 1 : (g.L / 8 > 256 ? 256 : g.L / 8);
  a.nrows = nrows; a.N = g.N; a.M = g.M; a.mode = mode; a.scale = scale; a.h = h; a.D = D;
  return a;
}

template <typename T>
static mjx_status dst1_run(const void* plan, int N, long long nrows, int mode, const T* x, T* out,
                           const T* lam, double h, double D, T scale, cudaStream_t s) {
  const Dst1Geom g = dst1_geom(N, sizeof(T));
  const char* p = (const char*)plan;
  const long long nseq_total = mode == DST_ETD1 ? nrows : (nrows + 1) / 2;
  if (nseq_total == 0) return MJX_OK;
  if constexpr (sizeof(T) == 4) {
    const Dst32Args a = trig_args32(g, p, nrows, nseq_total, mode, x, out, lam, h, D, scale);
    const long long nblk = (nseq_total + a.nseq - 1) / a.nseq;
    if (nblk > 0x7fffffffLL) return MJX_BAD_SHAPE;
    const int tps = g.L >= 16 ? g.L / 16 : 1;
    const size_t smem = (size_t)sp_size(a.nseq * g.L) * sizeof(float2);
    dst1_kernel32<<<(unsigned)nblk, a.nseq * tps, smem, s>>>(a);
  } else {
    Dst1Args<T> a = trig_args<T>(g, p, nrows, mode, x, out, lam, h, D, scale);
    a.lS = tile_log<T>(a.d, nseq_total, 8);
    const long long nblk = (nseq_total + (1 << a.lS) - 1) >> a.lS;
    if (nblk > 0x7fffffffLL) return MJX_BAD_SHAPE;
    dst1_kernel<T><<<(unsigned)nblk, tile_threads<T>(a.d, a.lS), tile_smem<T>(a.d, a.lS), s>>>(a);
  }
  return cuda_status(cudaGetLastError());
}

static mjx_status dst1_attrs() {
  static ContextOnce once;
  return once.run([]() -> mjx_status {
    int dev = 0, optin = 0;
    MJX_CUDA_TRY(cudaGetDevice(&dev));
    MJX_CUDA_TRY(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    MJX_CUDA_TRY(cudaFuncSetAttribute(dst1_kernel32, cudaFuncAttributeMaxDynamicSharedMemorySize, optin));
    MJX_CUDA_TRY(cudaFuncSetAttribute(dst1_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin));
    MJX_CUDA_TRY(cudaFuncSetAttribute(dct2_kernel32, cudaFuncAttributeMaxDynamicSharedMemorySize, optin));
    MJX_CUDA_TRY(cudaFuncSetAttribute(dct2_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin));
    return MJX_OK;
  });
}

template <typename T>
static mjx_status dct2_run(const void* plan, int n, long long nrows, int mode, const T* x, T* out,
                           const T* lam, double h, double D, T scale, cudaStream_t s) {
  const Dst1Geom g = dst1_geom(n, sizeof(T), 1);
  const char* p = (const char*)plan;
  const long long nseq_total = mode == DCT_ETD1 ? nrows : (nrows + 1) / 2;
  if (nseq_total == 0) return MJX_OK;
  if constexpr (sizeof(T) == 4) {
    const Dst32Args a = trig_args32(g, p, nrows, nseq_total, mode, x, out, lam, h, D, scale);
    const long long nblk = (nseq_total + a.nseq - 1) / a.nseq;
    if (nblk > 0x7fffffffLL) return MJX_BAD_SHAPE;
    const int tps = g.L >= 16 ? g.L / 16 : 1;
    const size_t smem = (size_t)sp_size(a.nseq * g.L) * sizeof(float2);
    dct2_kernel32<<<(unsigned)nblk, a.nseq * tps, smem, s>>>(a, (const float2*)(p + g.shift));
  } else {
    Dst1Args<T> a = trig_args<T>(g, p, nrows, mode, x, out, lam, h, D, scale);
    a.lS = tile_log<T>(a.d, nseq_total, 8);
    const long long nblk = (nseq_total + (1 << a.lS) - 1) >> a.lS;
    if (nblk > 0x7fffffffLL) return MJX_BAD_SHAPE;
    dct2_kernel<T><<<(unsigned)nblk, tile_threads<T>(a.d, a.lS), tile_smem<T>(a.d, a.lS), s>>>(
        a, (const cx<T>*)(p + g.shift));
  }
  return cuda_status(cudaGetLastError());
}

// host-side tables of a length-N transform of the given kind (twiddles; Bluestein chirp and
// filter when M is not a power of two; DCT phase factors e^{-i pi k / 2N})
static void trig_tables(std::vector<unsigned char>& host, const Dst1Geom& g, int e, int kind) {
  const double pi = 3.1415926535897932384626433832795;
  auto put = [&](size_t off, int i, double re, double im) {
    if (e == 4) { float* q = (float*)(host.data() + off); q[2 * i] = (float)re; q[2 * i + 1] = (float)im; }
    else { double* q = (double*)(host.data() + off); q[2 * i] = re; q[2 * i + 1] = im; }
  };
  const Roots roots(g.L);
  for (int j = 0; j < g.L; ++j) {
    double re, im;
    tile_twiddle(roots, j, e, &re, &im);
    put(g.tw, j, re, im);
  }
  if (e == 4) fft_pass_table((float*)(host.data() + g.tw), g.L);
  if (g.bluestein) {
    std::vector<double> chirp, bhat;
    bluestein_tables(g.M, roots, e == 8, &chirp, &bhat);
    for (int j = 0; j < g.M; ++j) put(g.chirp, j, chirp[2 * j], chirp[2 * j + 1]);
    for (int j = 0; j < g.L; ++j) put(g.bhat, j, bhat[2 * j], bhat[2 * j + 1]);
  }
  if (kind == 1)
    for (int k = 0; k < g.N; ++k) put(g.shift, k, cos(pi * k / (2.0 * g.N)), -sin(pi * k / (2.0 * g.N)));
}

}  // namespace mjx

using namespace mjx;

extern "C" {

// lengths the one-CTA transform handles: the FFT length L is at most 4096
static bool dst1_size_ok(int n) { return n >= 1 && n <= 2047 && dst1_geom(n, 8).L <= 4096; }

size_t mjx_dst1_plan_bytes(int n, int dtype) {
  const int e = elem_size(dtype);
  if (!e || !dst1_size_ok(n)) return 0;
  return dst1_geom(n, e).total;
}

mjx_status mjx_dst1_plan_init(void* plan, int n, int dtype, void* stream) {
  const int e = elem_size(dtype);
  if (!e) return MJX_BAD_DTYPE;
  if (plan == nullptr) return MJX_BAD_ARG;
  if (!dst1_size_ok(n)) return MJX_BAD_SHAPE;
  const Dst1Geom g = dst1_geom(n, e);
  std::vector<unsigned char> host(g.total, 0);
  trig_tables(host, g, e, 0);
  MJX_CUDA_TRY(cudaMemcpyAsync(plan, host.data(), g.total, cudaMemcpyHostToDevice, (cudaStream_t)stream));
  MJX_CUDA_TRY(cudaStreamSynchronize((cudaStream_t)stream));
  return MJX_OK;
}

mjx_status mjx_dst1(const void* plan, int n, long long nrows, int dtype, int mode, const void* x,
                    void* out, const void* lam, double h, double D, double scale, void* stream) {
  const int e = elem_size(dtype);
  if (!e) return MJX_BAD_DTYPE;
  if (!dst1_size_ok(n) || nrows < 0) return MJX_BAD_SHAPE;
  if (plan == nullptr || x == nullptr || out == nullptr) return MJX_BAD_ARG;
  if (mode < DST_PLAIN || mode > DST_ETD1 || (mode != DST_PLAIN && lam == nullptr)) return MJX_BAD_ARG;
  MJX_TRY(dst1_attrs());
  cudaStream_t s = (cudaStream_t)stream;
  if (e == 4)
    return dst1_run<float>(plan, n, nrows, mode, (const float*)x, (float*)out, (const float*)lam, h, D,
                           (float)scale, s);
  return dst1_run<double>(plan, n, nrows, mode, (const double*)x, (double*)out, (const double*)lam, h, D,
                          scale, s);
}

// DCT-II lengths: 2N a power of two up to 4096 or Bluestein with L <= 4096 (N <= 1024)
static bool dct2_size_ok(int n) { return n >= 1 && n <= 2048 && dst1_geom(n, 8, 1).L <= 4096; }

size_t mjx_dct2_plan_bytes(int n, int dtype) {
  const int e = elem_size(dtype);
  if (!e || !dct2_size_ok(n)) return 0;
  return dst1_geom(n, e, 1).total;
}

mjx_status mjx_dct2_plan_init(void* plan, int n, int dtype, void* stream) {
  const int e = elem_size(dtype);
  if (!e) return MJX_BAD_DTYPE;
  if (plan == nullptr) return MJX_BAD_ARG;
  if (!dct2_size_ok(n)) return MJX_BAD_SHAPE;
  const Dst1Geom g = dst1_geom(n, e, 1);
  std::vector<unsigned char> host(g.total, 0);
  trig_tables(host, g, e, 1);
  MJX_CUDA_TRY(cudaMemcpyAsync(plan, host.data(), g.total, cudaMemcpyHostToDevice, (cudaStream_t)stream));
  MJX_CUDA_TRY(cudaStreamSynchronize((cudaStream_t)stream));
  return MJX_OK;
}

mjx_status mjx_dct2(const void* plan, int n, long long nrows, int dtype, int mode, const void* x,
                    void* out, const void* lam, double h, double D, double scale, void* stream) {
  const int e = elem_size(dtype);
  if (!e) return MJX_BAD_DTYPE;
  if (!dct2_size_ok(n) || nrows < 0) return MJX_BAD_SHAPE;
  if (plan == nullptr || x == nullptr || out == nullptr) return MJX_BAD_ARG;
  if (mode < DCT_FWD || mode > DCT_ETD1 || (mode >= DCT_HELMHOLTZ && lam == nullptr)) return MJX_BAD_ARG;
  MJX_TRY(dst1_attrs());
  cudaStream_t s = (cudaStream_t)stream;
  if (e == 4)
    return dct2_run<float>(plan, n, nrows, mode, (const float*)x, (float*)out, (const float*)lam, h, D,
                           (float)scale, s);
  return dct2_run<double>(plan, n, nrows, mode, (const double*)x, (double*)out, (const double*)lam, h, D,
                          scale, s);
}

}  // extern "C"
