// Periodic 2D spectral passes: fused row r2c/c2r (+ pointwise work) and
// column forward-multiply-inverse kernels, plans, and the C ABI for the
// Helmholtz / CN / exponential multipliers and the FFT-CN stepper.
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <mutex>
#include <vector>

#include "spectral.cuh"
#include "tfft.cuh"
#include "tma.cuh"
#include "wfft.cuh"

namespace mjx {

static inline size_t align256(size_t b) { return (b + 255) & ~size_t(255); }

int spec_ldc(int nx) { return ((nx / 2 + 1) + 3) & ~3; }

// Entries of the x twiddle table: FP32 plans of 1024-point rows append the same 1024 values
// transposed for the one-warp transform (entry kW1024 + 32 k1 + l holds w^(l k1)), so that
// the 32 lanes of a warp read one contiguous 256-byte run per twiddle instead of 32 rows
// of the table.
static int twx_count(int nx, int elem) {
  return elem == 8 ? 2 * nx : nx + fft_pass_entries(nx) + (nx == 1024 ? 1024 : 0);
}
// FP64 tables are followed by their (cos, tan) form (tfft.cuh)
static int twy_count(int ny, int elem) { return elem == 8 ? 2 * ny : ny + fft_pass_entries(ny); }

size_t plan_bytes(int ny, int nx, int elem) {
  const size_t c = 2 * (size_t)elem;
  return align256(twx_count(nx, elem) * c) + align256(twy_count(ny, elem) * c) + align256(spec_ldc(nx) * (size_t)elem) +
         align256(ny * (size_t)elem);
}

PlanView plan_view(const void* plan, int ny, int nx, int elem) {
  const size_t c = 2 * (size_t)elem;
  const char* p = (const char*)plan;
  PlanView v;
  v.twx = p; p += align256(twx_count(nx, elem) * c);
  v.twy = p; p += align256(twy_count(ny, elem) * c);
  v.lamx = p; p += align256(spec_ldc(nx) * (size_t)elem);
  v.lamy = p;
  return v;
}

// Sequences (row pairs) per CTA: ~128 threads per CTA, so that the 1024-row passes
// launch enough CTAs to fill every SM (n = 1024: 2 sequences, n = 4096: one of 256 threads).
int row_nseq(int n, int nrows) {
  const int tps = n >= 16 ? n / 16 : 1;
  int ns = 128 / tps;
  if (ns < 1) ns = 1;
  if (ns > nrows) ns = nrows;
  return ns;
}

int row_ctas(int n, int nrows, int npairs) { return npairs * nrows / row_nseq(n, nrows); }

template <typename T> __device__ __forceinline__ bool finite_(T v) { return isfinite(v); }

// ------------------------------------------------------------------ row pass
template <typename T> struct Occ { static constexpr int row = sizeof(T) == 4 ? 4 : 2, col = sizeof(T) == 4 ? 2 : 1; };

// LOG2N > 0: the row length 2^LOG2N (above 1024 one sequence per CTA) is a compile-time constant,
// so that the transform's index arithmetic and radix schedule fold into the code; LOG2N = 0
// (rows of at most 16 points) reads it from the arguments.  A thread keeps its elements
// lt + m tps in registers from the load to the store (fft_regs); shared memory carries the
// exchanges inside the transforms and the mirrored half of a spectrum, which the two-for-one
// packing pairs with the other half.  FP32, fused (c2r, reaction, r2c), 256, 2048 and 4096 points:
// 6.9, 58 and 100 us; through shared memory 14.7 (length at run time), 63 and 125 us.  1024 points:
// 13.2 us (2048 row pairs), 18.0 with 32 points a lane of one warp a row (row_kernel_w32).  The long
// rows are bound by the SMs' issue and shared-memory bandwidth alike, the short ones by the
// latency of one chain (load, five exchanges, store) on a few warps an SM.
template <typename T, int RX, int LOG2N = 0>
__global__ void __launch_bounds__(256, Occ<T>::row) row_kernel(const __grid_constant__ RowArgs<T> a) {
  typedef cx<T> C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);
  const DevState* st = a.st;
  pdl_wait();
  if (st != nullptr && st->done) return;

  const int n = LOG2N ? (1 << LOG2N) : a.n, half = n >> 1;
  const int log2n = LOG2N ? LOG2N : a.log2n, nseq = LOG2N > 10 ? 1 : a.nseq;
  const int tps = n >= 16 ? n / 16 : 1;
  const int tid = threadIdx.x;
  const int s_loc = tid / tps, lt = tid % tps;
  const int seq0 = blockIdx.x * nseq;
  const int q = seq0 / a.nrows;  // uniform within the CTA (nrows % nseq == 0)
  const RowPair pr = a.pr[q];
  const int flags = pr.flags;
  const long long y = (seq0 % a.nrows) + s_loc;
  const int cur = st != nullptr ? st->cur : 0;
  const T* rin = a.rin_sel < 0 ? a.rin[0] : a.rin[a.rin_sel == 0 ? cur : 1 - cur];
  T* rout = a.rout_sel < 0 ? a.rout[0] : a.rout[a.rout_sel == 0 ? cur : 1 - cur];
  const int zb = s_loc * n;  // this sequence's first logical smem element
  // element lt + m tps of the sequence, m < 16, is in x[m]; a mirrored index needs its own padding
#define Z(x) buf[sp(zb + (x))]
  C x[16];

  // 1. load: spectrum rows (c2r) or real rows
  if (flags & ROW_LOAD_SPEC) {
    const C* A = a.spec + pr.sa + y * a.ldc;
    const C* B = a.spec + pr.sb + y * a.ldc;
    // every thread owns kk = lt + m*tps <= n/2, m < 9: issue all loads first
    C Ak[9], Bk[9];
#pragma unroll
    for (int m = 0; m < 9; ++m) {
      const int kk = lt + m * tps;
      if (kk <= half) { Ak[m] = A[kk]; Bk[m] = B[kk]; }
    }
#pragma unroll
    for (int m = 0; m < 9; ++m) {
      const int kk = lt + m * tps;
      if (kk <= half) {
        x[m] = mk<C>(Ak[m].x - Bk[m].y, Ak[m].y + Bk[m].x);                                  // A_k + i B_k
        if (kk > 0 && kk < half) Z(n - kk) = mk<C>(Ak[m].x + Bk[m].y, Bk[m].x - Ak[m].y);  // conj(A_k) + i conj(B_k)
      }
    }
    __syncthreads();
    const C* zt = buf + sp(zb + lt);
#pragma unroll
    for (int m = 1; m < 16; ++m) {
      const int kk = lt + m * tps;
      if (kk > half && kk < n) x[m] = zt[sp(m * tps)];
    }
    __syncthreads();
    fft_regs<T, true, true>(x, buf, n, log2n, lt, zb, 1, a.tw);
  } else {
    const T* ra = rin + pr.ra + y * a.rstride;
    const T* rb = rin + pr.rb + y * a.rstride;
#pragma unroll
    for (int m = 0; m < 16; ++m) {
      const int i = lt + m * tps;
      if (i < n) x[m] = mk<C>(ra[i], rb[i]);
    }
  }

  // 2. pointwise work on the real rows
  const T sc = (flags & ROW_LOAD_SPEC) ? a.inv_scale : (T)1;
  T h = (T)0;
  if (flags & ROW_REACT) h = (T)((st != nullptr ? st->dtc : a.hfixed) * pr.hfac);
  T esum = (T)0;
  int bad = 0;
  T* oa = rout + pr.ra + y * a.rstride;
  T* ob = rout + pr.rb + y * a.rstride;
  const T* ea = a.eref + pr.ra + y * a.rstride;
  const T* eb = a.eref + pr.rb + y * a.rstride;
  // parameters converted once (the per-element double arithmetic would occupy the FP64 pipe)
  const T pF = (T)a.F, pK = (T)a.k, pR = (T)a.r, pFK = (T)(a.F + a.k);
  const T pAtol = (T)a.atol, pRtol = (T)a.rtol;
#pragma unroll
  for (int m0 = 0; m0 < 16; m0 += 4) {
    T ra_[4], rb_[4];  // four references ahead of the stores, which may alias them for the compiler
    if (flags & ROW_ERRNORM) {
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const int i = lt + (m0 + m) * tps;
        if (i < n) { ra_[m] = ea[i]; rb_[m] = eb[i]; }
      }
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const int i = lt + (m0 + m) * tps;
      if (i >= n) continue;
      const C v = x[m0 + m];
      T va = v.x * sc, vb = v.y * sc;
      if (flags & ROW_NONLIN) {
        // Gray-Scott reaction terms (operators.py:655-667); Fisher-KPP r u (1-u)
        if (RX == RX_GRAY_SCOTT) {
          const T uvv = va * vb * vb;
          const T nu = -uvv + pF * ((T)1 - va), nv = uvv - pFK * vb;
          va = nu; vb = nv;
        } else if (RX == RX_FISHER) {
          va = pR * va * ((T)1 - va); vb = pR * vb * ((T)1 - vb);
        } else {
          va = (T)0; vb = (T)0;
        }
      }
      if (flags & ROW_REACT) {
        if (flags & ROW_DELTA) react_delta<T, RX>(va, vb, h, pF, pK, pR);
        else if (flags & ROW_EULER) {
          react_euler<T, RX>(va, vb, h, pF, pK, pR);
          if (flags & ROW_EULER2) react_euler<T, RX>(va, vb, h, pF, pK, pR);
        }
        else react_heun<T, RX>(va, vb, h, pF, pK, pR);
      }
      if (flags & ROW_STORE_REAL) { oa[i] = va; ob[i] = vb; }
      if (flags & ROW_ERRNORM) {
        // moljax/core/state.py:335-339: (err / (atol + rtol |y_new|))^2
        const T da = (va - ra_[m]) / (pAtol + pRtol * fabs(va));
        const T db = (vb - rb_[m]) / (pAtol + pRtol * fabs(vb));
        esum += da * da + db * db;
        bad |= !(finite_(va) && finite_(vb));
      }
      if (flags & ROW_ERRPAIR) {
        const T da = va / (pAtol + pRtol * fabs(vb));
        esum += da * da;
        bad |= !(finite_(va) && finite_(vb));
      }
      x[m0 + m] = mk<C>(va, vb);
    }
  }

  // 3. r2c and split into the two half spectra
  if (flags & ROW_STORE_SPEC) {
    if (flags & ROW_LOAD_SPEC) __syncthreads();
    fft_regs<T, false, true>(x, buf, n, log2n, lt, zb, 1, a.tw);
    C* A = a.spec + ((flags & ROW_SPEC_ALT) ? pr.oa : pr.sa) + y * a.ldc;
    C* B = a.spec + ((flags & ROW_SPEC_ALT) ? pr.ob : pr.sb) + y * a.ldc;
    __syncthreads();
    C* zt = buf + sp(zb + lt);
#pragma unroll
    for (int m = 1; m < 16; ++m) {
      const int kk = lt + m * tps;
      if (kk > half && kk < n) zt[sp(m * tps)] = x[m];
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < 9; ++m) {
      const int kk = lt + m * tps;
      if (kk > half) continue;
      const C Zk = x[m], Zm = kk > 0 && kk < half ? Z(n - kk) : Zk;
      A[kk] = mk<C>((T)0.5 * (Zk.x + Zm.x), (T)0.5 * (Zk.y - Zm.y));
      B[kk] = mk<C>((T)0.5 * (Zk.y + Zm.y), (T)0.5 * (Zm.x - Zk.x));
    }
  }

  // 4. block reduction of the error partials (FP64 across threads)
  if (flags & (ROW_ERRNORM | ROW_ERRPAIR)) {
    __shared__ double red[32];
    __shared__ int redbad[32];
    double v = (double)esum;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      v += __shfl_xor_sync(0xffffffffu, v, o);
      bad |= __shfl_xor_sync(0xffffffffu, bad, o);
    }
    const int w = tid >> 5, nw = (blockDim.x + 31) >> 5;
    if ((tid & 31) == 0) { red[w] = v; redbad[w] = bad; }
    __syncthreads();
    if (tid == 0) {
      double s = 0.0, c = 0.0;  // Kahan
      int b2 = 0;
      for (int i = 0; i < nw; ++i) {
        const double yv = red[i] - c;
        const double tv = s + yv;
        c = (tv - s) - yv;
        s = tv;
        b2 |= redbad[i];
      }
      a.partial[blockIdx.x] = s;
      a.nonfinite[blockIdx.x] = b2;
    }
  }
#undef Z
}

// ------------------------------------------------------------------ column pass
template <typename T> struct ColThreads { static constexpr int v = sizeof(T) == 4 ? 1024 : 512; };

// C ny/16 threads (C below 16 rows) per output of a tile of C columns; a thread keeps its 16
// elements in registers from the load to the store (fft_regs).  A second output has its own threads
// and its own half of the shared memory, and repeats the forward transform there: the threads would
// be idle meanwhile.  LOG2NY > 0 fixes the length at compile time.  Chained with its rows, FFT-CN
// FP32 takes 29 us a step at 256^2 (48 with the elements in shared memory between the transforms
// and the length at run time), 38 at 1024^2 (61).  512 and 1024 rows get 128 registers a thread
// (their CTAs have at most 512): 12.8 and 18.9 us against 14.8 and 21.6; shorter columns fit in 64,
// and a box's passes want the CTAs (128 rows: 25.7 us against 29.6).  The other lengths, five steps:
// 4 x 256 51 us (157), 16 x 4096 80 (167), 2048 x 256 103 (228), 4096 x 1024 235 (312).
template <typename T, int LOG2NY = 0>
__global__ void __launch_bounds__(LOG2NY == 9 || LOG2NY == 10 ? 512 : ColThreads<T>::v, 1) col_kernel(const __grid_constant__ ColArgs<T> a) {
  typedef cx<T> C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_wait();
  if (a.st != nullptr && a.st->done) return;
  const ColJob jb = a.job[blockIdx.y];
  const int ny = LOG2NY ? (1 << LOG2NY) : a.ny, log2ny = LOG2NY ? LOG2NY : a.log2ny;
  const int Cn = a.C, tps = ny >= 16 ? ny >> 4 : 1, per = Cn * tps;  // C: a power of two
  const int o = threadIdx.x >= per ? 1 : 0, r = threadIdx.x - o * per, c = r & (Cn - 1), lt = r >> (__ffs(Cn) - 1);
  const int kx = blockIdx.x * Cn + c;
  const bool active = o < jb.nout, in = active && kx < a.ncols;
  const long long ldc = a.ldc, po = (long long)blockIdx.z * a.pstride;
  C* buf = reinterpret_cast<C*>(smem_raw) + o * sp_size(ny * Cn);
  C x[16];

  const C* src = a.spec + po + jb.sin + kx;
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    const int ky = lt + q * tps;
    x[q] = mk<C>((T)0, (T)0);
    if (in && ky < ny) x[q] = src[ky * ldc];
  }
  const int dirs = jb.dirs ? jb.dirs : 3;
  if (dirs & 1) fft_regs<T, false, false>(x, buf, ny, log2ny, lt, c, Cn, a.tw, active);

  const T jscale = jb.scale != 0.0 ? (T)jb.scale : a.scale;
  const double h = a.st != nullptr ? a.st->dtc : a.hfixed;
  const T hD = (T)(h * jb.hfac[o] * jb.D);
  T lxy = (T)0;
  if (in) lxy = a.ldc3 ? a.lamx[kx % a.ldc3] + a.lamy2[kx / a.ldc3] : a.lamx[kx];
  if (jb.mul == MUL_ADVDIFF || jb.mul == MUL_ADV_LAP || jb.mul == MUL_ADV_EXP || jb.mul == MUL_ADV_CN) {
    // one copy of the complex multiplier's code: the elements pass through their places in shared memory
    C* own = buf + sp(lt * Cn + c);
    __syncthreads();
    if (in) {
#pragma unroll
      for (int q = 0; q < 16; ++q)
        if (q * tps < ny) own[sp(q * tps * Cn)] = x[q];
#pragma unroll 1
      for (int ky = lt, q = 0; ky < ny && q < 16; ky += tps, ++q) {
        const double2 f = adv_multiplier<T>(a, jb, (double)hD, h * jb.hfac[0], (double)(lxy + a.lamy[ky]), kx, ky);
        const T mr = (T)f.x, mi = (T)f.y;
        C& e = own[sp(q * tps * Cn)];
        e = cscale(mk<C>(e.x * mr - e.y * mi, e.x * mi + e.y * mr), jscale);
      }
#pragma unroll
      for (int q = 0; q < 16; ++q)
        if (q * tps < ny) x[q] = own[sp(q * tps * Cn)];
    }
  } else {
    const int mul = jb.mul, pw = jb.pow[o];
    const T* tab = mul == MUL_TABLED ? a.mtab + jb.sin + kx : a.mtab + kx;
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const int ky = lt + q * tps;
      if (!in || ky >= ny) continue;
      T m;
      if (mul == MUL_TABLED) m = tab[ky * ldc];
      else if (mul == MUL_TABLE) m = jscale * tab[ky * ldc];
      else m = jscale * multiplier<T>(mul, hD, lxy + a.lamy[ky], pw);
      x[q] = cscale(x[q], m);
    }
  }
  if (dirs & 2) {
    if (dirs & 1 || jb.mul >= MUL_ADVDIFF) __syncthreads();
    fft_regs<T, true, false>(x, buf, ny, log2ny, lt, c, Cn, a.tw, active);
  }

  if (!in) return;
  C* dst = a.spec + po + jb.sout[o] + kx;
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    const int ky = lt + q * tps;
    if (ky < ny) dst[ky * ldc] = x[q];
  }
}

// ------------------------------------------------------------------ warp row pass (n = 1024)
// The row pass of row_kernel (same flags, pair table, pointwise work and error partials) for
// FP32 rows of 1024 points, one warp per sequence: the row transform of the FP32 adaptive IMEX
// loop.  Its error estimate is a difference of FP32 solutions, so the step sizes and with them the
// end state follow the transform's rounding (1024^2, t = 6: 2.8e-5 apart between this kernel and
// row_kernel; their errors against FP64 8.8e-5 and 6.7e-5).  That loop keeps the transform that its
// results were made with, although row_kernel is nearer and faster (13.2 against 18.0 us).
template <int RX>
__global__ void __launch_bounds__(128) row_kernel_w32(const __grid_constant__ RowArgs<float> a) {
  typedef float2 C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const DevState* st = a.st;
  pdl_wait();
  if (st != nullptr && st->done) return;
  const int lane = threadIdx.x & 31, s_loc = threadIdx.x >> 5;
  C* tile = reinterpret_cast<C*>(smem_raw) + s_loc * (32 * 33);
  const int seq0 = blockIdx.x * a.nseq;
  const int q = seq0 / a.nrows;  // uniform within the CTA (nrows % nseq == 0)
  const RowPair pr = a.pr[q];
  const int flags = pr.flags;
  const long long y = (seq0 % a.nrows) + s_loc;
  const int cur = st != nullptr ? st->cur : 0;
  const float* rin = a.rin_sel < 0 ? a.rin[0] : a.rin[a.rin_sel == 0 ? cur : 1 - cur];
  float* rout = a.rout_sel < 0 ? a.rout[0] : a.rout[a.rout_sel == 0 ? cur : 1 - cur];
  const int src = (32 - lane) & 31;  // the lane holding index 1024 - k of this lane's k
  C z[32];
  // 1. load: spectrum rows (c2r) or real rows, element lane + 32 j in z[j]
  if (flags & ROW_LOAD_SPEC) {
    const C* A = a.spec + pr.sa + y * a.ldc;
    const C* B = a.spec + pr.sb + y * a.ldc;
    C Ar[17], Br[17];
#pragma unroll
    for (int j = 0; j < 16; ++j) { Ar[j] = A[32 * j + lane]; Br[j] = B[32 * j + lane]; }
    Ar[16] = lane == 0 ? A[512] : mk<C>(0.f, 0.f);
    Br[16] = lane == 0 ? B[512] : mk<C>(0.f, 0.f);
#pragma unroll
    for (int j = 0; j < 16; ++j) z[j] = mk<C>(Ar[j].x - Br[j].y, Ar[j].y + Br[j].x);  // A_k + i B_k
#pragma unroll
    for (int j = 16; j < 32; ++j) {  // k = 32 j + lane > 512 (and k = 512 on lane 0)
      C av = shfl2(Ar[31 - j], src), bv = shfl2(Br[31 - j], src);
      if (lane == 0) { av = Ar[32 - j]; bv = Br[32 - j]; }
      if (lane == 0 && j == 16) z[j] = mk<C>(av.x - bv.y, av.y + bv.x);
      else z[j] = mk<C>(av.x + bv.y, bv.x - av.y);  // conj(A_k') + i conj(B_k'), k' = 1024 - k
    }
    wfft1024<true>(z, tile, a.tw, lane);
  } else {
    const float* ra = rin + pr.ra + y * a.rstride;
    const float* rb = rin + pr.rb + y * a.rstride;
#pragma unroll
    for (int j = 0; j < 32; ++j) z[j] = mk<C>(ra[32 * j + lane], rb[32 * j + lane]);
  }

  // 2. pointwise work on element x = lane + 32 j (as row_kernel)
  const float sc = (flags & ROW_LOAD_SPEC) ? a.inv_scale : 1.0f;
  float h = 0.f;
  if (flags & ROW_REACT) h = (float)((st != nullptr ? st->dtc : a.hfixed) * pr.hfac);
  float esum = 0.f;
  int bad = 0;
  float* oa = rout + pr.ra + y * a.rstride;
  float* ob = rout + pr.rb + y * a.rstride;
  const float* ea = a.eref + pr.ra + y * a.rstride;
  const float* eb = a.eref + pr.rb + y * a.rstride;
  const float pF = (float)a.F, pK = (float)a.k, pR = (float)a.r, pFK = (float)(a.F + a.k);
  const float pAtol = (float)a.atol, pRtol = (float)a.rtol;
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    const int x = lane + 32 * j;
    float va = z[j].x * sc, vb = z[j].y * sc;
    if (flags & ROW_NONLIN) {
      if (RX == RX_GRAY_SCOTT) {
        const float uvv = va * vb * vb;
        const float nu = -uvv + pF * (1.f - va), nv = uvv - pFK * vb;
        va = nu; vb = nv;
      } else if (RX == RX_FISHER) {
        va = pR * va * (1.f - va); vb = pR * vb * (1.f - vb);
      } else {
        va = 0.f; vb = 0.f;
      }
    }
    if (flags & ROW_REACT) {
      if (flags & ROW_DELTA) react_delta<float, RX>(va, vb, h, pF, pK, pR);
      else if (flags & ROW_EULER) {
        react_euler<float, RX>(va, vb, h, pF, pK, pR);
        if (flags & ROW_EULER2) react_euler<float, RX>(va, vb, h, pF, pK, pR);
      }
      else react_heun<float, RX>(va, vb, h, pF, pK, pR);
    }
    if (flags & ROW_STORE_REAL) { oa[x] = va; ob[x] = vb; }
    if (flags & ROW_ERRNORM) {
      const float da = (va - ea[x]) / (pAtol + pRtol * fabsf(va));
      const float db = (vb - eb[x]) / (pAtol + pRtol * fabsf(vb));
      esum += da * da + db * db;
      bad |= !(finite_(va) && finite_(vb));
    }
    if (flags & ROW_ERRPAIR) {
      const float da = va / (pAtol + pRtol * fabsf(vb));
      esum += da * da;
      bad |= !(finite_(va) && finite_(vb));
    }
    z[j] = mk<C>(va, vb);
  }

  // 3. r2c and split into the two half spectra: X_k in z[k2] of lane k1, k = k1 + 32 k2
  if (flags & ROW_STORE_SPEC) {
    wfft1024<false>(z, tile, a.tw, lane);
    C* A = a.spec + ((flags & ROW_SPEC_ALT) ? pr.oa : pr.sa) + y * a.ldc;
    C* B = a.spec + ((flags & ROW_SPEC_ALT) ? pr.ob : pr.sb) + y * a.ldc;
#pragma unroll
    for (int k2 = 0; k2 <= 16; ++k2) {
      C Zm = shfl2(z[k2 <= 15 ? 31 - k2 : 15], src);  // X_{1024-k} (lanes > 0)
      if (lane == 0) Zm = z[(32 - k2) & 31];
      const int k = lane + 32 * k2;
      if (k2 == 16 && lane != 0) continue;
      const C Zk = z[k2];
      A[k] = mk<C>(0.5f * (Zk.x + Zm.x), 0.5f * (Zk.y - Zm.y));
      B[k] = mk<C>(0.5f * (Zk.y + Zm.y), 0.5f * (Zm.x - Zk.x));
    }
  }

  // 4. block reduction of the error partials (FP64 across warps)
  if (flags & (ROW_ERRNORM | ROW_ERRPAIR)) {
    __shared__ double red[4];
    __shared__ int redbad[4];
    double v = (double)esum;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      v += __shfl_xor_sync(0xffffffffu, v, o);
      bad |= __shfl_xor_sync(0xffffffffu, bad, o);
    }
    if (lane == 0) { red[s_loc] = v; redbad[s_loc] = bad; }
    __syncthreads();
    if (threadIdx.x == 0) {
      double sum = 0.0, c = 0.0;  // Kahan
      int b2 = 0;
      for (int i = 0; i < a.nseq; ++i) {
        const double yv = red[i] - c;
        const double tv = sum + yv;
        c = (tv - sum) - yv;
        sum = tv;
        b2 |= redbad[i];
      }
      a.partial[blockIdx.x] = sum;
      a.nonfinite[blockIdx.x] = b2;
    }
  }
}

// ------------------------------------------------------------------ launchers
static size_t row_smem(int n, int nseq, int elem) { return (size_t)sp_size(nseq * n) * 2 * elem; }

template <typename T, int RX>
cudaError_t launch_row(const RowArgs<T>& a0, cudaStream_t s) {
  if constexpr (sizeof(T) == 8)
    if (row64_takes(a0.n)) return launch_row64<RX>(a0, s);
  // Small grids: fewer row pairs per CTA until the pass covers every SM (the partial-sum
  // passes keep their CTA count, which sizes the controller's reduction).  FP64 transforms
  // are bound by the FP64 units, so a pass on a few SMs is a few times slower.
  RowArgs<T> a = a0;
  bool partials = false;
  for (int q = 0; q < a.npairs && q < MJX_MAXPAIR; ++q)
    partials |= (a.pr[q].flags & (ROW_ERRNORM | ROW_ERRPAIR)) != 0;
  if (!partials)
    while (a.nseq > 1 && a.npairs * a.nrows / a.nseq < 152) a.nseq >>= 1;
  const int tps = a.n >= 16 ? a.n / 16 : 1;
  const int grid = a.npairs * a.nrows / a.nseq;
  if constexpr (sizeof(T) == 4) {
    if (a.n == 1024 && a.warp && a.nseq <= 4) {  // one warp per 1024-point row
      return launch_chain(row_kernel_w32<RX>, dim3(grid), 32 * a.nseq, (size_t)a.nseq * 32 * 33 * sizeof(float2), s,
                          a.pdl, a);
    }
  }
  const size_t smem = row_smem(a.n, a.nseq, sizeof(T));
  const int threads = a.nseq * tps;
#define MJX_ROW(L) case L: return launch_chain(row_kernel<T, RX, L>, dim3(grid), threads, smem, s, a.pdl, a);
  if constexpr (sizeof(T) == 4) {
    switch (a.log2n) {
      MJX_ROW(5) MJX_ROW(6) MJX_ROW(7) MJX_ROW(8) MJX_ROW(9) MJX_ROW(10) MJX_ROW(11) MJX_ROW(12)
      default: return launch_chain(row_kernel<T, RX>, dim3(grid), threads, smem, s, a.pdl, a);
    }
  } else {
    return launch_chain(row_kernel<T, RX, 12>, dim3(grid), threads, smem, s, a.pdl, a);  // the others: row64_takes
  }
#undef MJX_ROW
}

template <typename T>
cudaError_t launch_col(const ColArgs<T>& a0, cudaStream_t s) {
  if constexpr (sizeof(T) == 8)
    if (col64_takes(a0.ny)) return launch_col64(a0, s);
  ColArgs<T> a = a0;
  int maxout = 1;
  for (int j = 0; j < a.njobs; ++j) maxout = a.job[j].nout > maxout ? a.job[j].nout : maxout;
  const int tps = a.ny >= 16 ? a.ny / 16 : 1;
  // small grids: narrower tiles until the pass covers every SM (as launch_row)
  const long long planes = a.nplanes > 1 ? a.nplanes : 1;
  while (a.C > 1 && (long long)((a.ncols + a.C - 1) / a.C) * a.njobs * planes < 152) a.C >>= 1;
  dim3 grid((a.ncols + a.C - 1) / a.C, a.njobs, a.nplanes > 1 ? a.nplanes : 1);
  const size_t smem = (size_t)sp_size(a.ny * a.C) * maxout * sizeof(cx<T>);
  const int threads = a.C * maxout * tps;
#define MJX_COL(L) case L: return launch_chain(col_kernel<T, L>, grid, threads, smem, s, a.pdl, a);
  if constexpr (sizeof(T) == 4) {
    switch (a.log2ny) {
      MJX_COL(5) MJX_COL(6) MJX_COL(7) MJX_COL(8) MJX_COL(9) MJX_COL(10) MJX_COL(11) MJX_COL(12)
      default: return launch_chain(col_kernel<T>, grid, threads, smem, s, a.pdl, a);
    }
  } else {
    return launch_chain(col_kernel<T, 12>, grid, threads, smem, s, a.pdl, a);  // the others: col64_takes
  }
#undef MJX_COL
}

#define MJX_INST_ROW(T, RX) template cudaError_t launch_row<T, RX>(const RowArgs<T>&, cudaStream_t);
MJX_INST_ROW(float, RX_NONE)
MJX_INST_ROW(float, RX_GRAY_SCOTT)
MJX_INST_ROW(float, RX_FISHER)
MJX_INST_ROW(double, RX_NONE)
MJX_INST_ROW(double, RX_GRAY_SCOTT)
MJX_INST_ROW(double, RX_FISHER)
template cudaError_t launch_col<float>(const ColArgs<float>&, cudaStream_t);
template cudaError_t launch_col<double>(const ColArgs<double>&, cudaStream_t);

// Column tile width: ~256 threads per output, capped by 512 threads and ~200 KB smem.
int col_tile(int ny, int ncols, int nout, int elem) {
  const int tps = ny >= 16 ? ny / 16 : 1;
  int C = 256 / tps;
  if (C < 1) C = 1;
  // at least one 32-byte sector of every row per CTA (4 FP32 / 2 FP64 complex columns)
  const int cmin = 32 / (2 * elem);
  if (C < cmin) C = cmin;
  if (C > 16) C = 16;
  const int cap = elem == 4 ? 1024 : 512;  // col_kernel thread limit per precision
  while (C > 1 && (C * nout * tps > cap || (size_t)sp_size(ny * C * nout) * 2 * elem > 200 * 1024)) C >>= 1;
  (void)ncols;
  return C;
}

// Raises a kernel's dynamic shared-memory limit to the device's opt-in maximum
// minus the kernel's static shared memory.
template <typename K>
static mjx_status raise_smem(K kernel, int optin) {
  cudaFuncAttributes fa;
  MJX_CUDA_TRY(cudaFuncGetAttributes(&fa, kernel));
  MJX_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    optin - (int)fa.sharedSizeBytes));
  return MJX_OK;
}

template <int RX>
static mjx_status row_attrs(int optin) {
  MJX_TRY(raise_smem(row_kernel<float, RX>, optin));
  MJX_TRY(raise_smem(row_kernel<float, RX, 5>, optin));
  MJX_TRY(raise_smem(row_kernel<float, RX, 6>, optin));
  MJX_TRY(raise_smem(row_kernel<float, RX, 7>, optin));
  MJX_TRY(raise_smem(row_kernel<float, RX, 8>, optin));
  MJX_TRY(raise_smem(row_kernel<float, RX, 9>, optin));
  MJX_TRY(raise_smem(row_kernel<float, RX, 10>, optin));
  MJX_TRY(raise_smem(row_kernel<float, RX, 11>, optin));
  MJX_TRY(raise_smem(row_kernel<float, RX, 12>, optin));
  return raise_smem(row_kernel<double, RX, 12>, optin);
}

// Raise the dynamic shared-memory limit of every kernel once per CUDA context
// (function attributes belong to the context the kernels are loaded in).
mjx_status ensure_kernel_attrs() {
  static ContextOnce once;
  return once.run([]() -> mjx_status {
    int dev = 0, optin = 0;
    MJX_CUDA_TRY(cudaGetDevice(&dev));
    MJX_CUDA_TRY(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    MJX_TRY(row_attrs<RX_NONE>(optin));
    MJX_TRY(row_attrs<RX_GRAY_SCOTT>(optin));
    MJX_TRY(row_attrs<RX_FISHER>(optin));
    MJX_TRY(raise_smem(row_kernel_w32<RX_NONE>, optin));
    MJX_TRY(raise_smem(row_kernel_w32<RX_GRAY_SCOTT>, optin));
    MJX_TRY(raise_smem(row_kernel_w32<RX_FISHER>, optin));
    MJX_TRY(raise_smem(col_kernel<float>, optin));
    MJX_TRY(raise_smem(col_kernel<float, 5>, optin));
    MJX_TRY(raise_smem(col_kernel<float, 6>, optin));
    MJX_TRY(raise_smem(col_kernel<float, 7>, optin));
    MJX_TRY(raise_smem(col_kernel<float, 8>, optin));
    MJX_TRY(raise_smem(col_kernel<float, 9>, optin));
    MJX_TRY(raise_smem(col_kernel<float, 10>, optin));
    MJX_TRY(raise_smem(col_kernel<float, 11>, optin));
    MJX_TRY(raise_smem(col_kernel<float, 12>, optin));
    MJX_TRY(raise_smem(col_kernel<double, 12>, optin));
    MJX_TRY(spectral64_attrs(optin));
    return MJX_OK;
  });
}

typedef CUresult (*PfnTensorMapEncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                            const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                            CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                            CUtensorMapFloatOOBfill);

mjx_status make_tmap_2d_f32(CUtensorMap* map, const void* base, unsigned long long inner, unsigned long long rows,
                            unsigned long long row_bytes, unsigned box_inner, unsigned box_rows) {
  static PfnTensorMapEncodeTiled encode = nullptr;
  static std::once_flag resolved;
  std::call_once(resolved, []() {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) ==
            cudaSuccess && q == cudaDriverEntryPointSuccess)
      encode = (PfnTensorMapEncodeTiled)f;
  });
  if (encode == nullptr) return cuda_status(cudaErrorNotSupported);
  // the copy rules: 16-byte aligned base and row stride, inner box a multiple of 16 bytes
  if (((uintptr_t)base & 15) || (row_bytes & 15) || ((box_inner * 4) & 15) || box_rows < 1 || box_rows > 256 ||
      box_inner < 1 || box_inner > 256)
    return MJX_BAD_ARG;
  const cuuint64_t dims[2] = {inner, rows};
  const cuuint64_t strides[1] = {row_bytes};
  const cuuint32_t box[2] = {box_inner, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box,
                            estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return cuda_status(cudaErrorInvalidValue);
  return MJX_OK;
}

mjx_status make_tmap_3d_f32(CUtensorMap* map, const void* base, unsigned long long nx, unsigned long long ny,
                            unsigned long long nz, unsigned box_x, unsigned box_y) {
  static PfnTensorMapEncodeTiled encode = nullptr;
  static std::once_flag resolved;
  std::call_once(resolved, []() {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) ==
            cudaSuccess && q == cudaDriverEntryPointSuccess)
      encode = (PfnTensorMapEncodeTiled)f;
  });
  if (encode == nullptr) return cuda_status(cudaErrorNotSupported);
  if (((uintptr_t)base & 15) || ((nx * 4) & 15) || ((box_x * 4) & 15) || box_x < 1 || box_x > 256 || box_y < 1 ||
      box_y > 256)
    return MJX_BAD_ARG;
  const cuuint64_t dims[3] = {nx, ny, nz};
  const cuuint64_t strides[2] = {nx * 4, nx * ny * 4};
  const cuuint32_t box[3] = {box_x, box_y, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(base), dims, strides, box,
                            estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return cuda_status(cudaErrorInvalidValue);
  return MJX_OK;
}

typedef CUresult (*PfnCtxGetCurrent)(CUcontext*);
typedef CUresult (*PfnCtxGetId)(CUcontext, unsigned long long*);

mjx_status current_context_id(unsigned long long* id) {
  static PfnCtxGetCurrent get_current = nullptr;
  static PfnCtxGetId get_id = nullptr;
  static std::once_flag resolved;
  std::call_once(resolved, []() {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_current = (PfnCtxGetCurrent)f;
    f = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_id = (PfnCtxGetId)f;
  });
  if (get_current == nullptr || get_id == nullptr) return cuda_status(cudaErrorNotSupported);
  CUcontext ctx = nullptr;
  if (get_current(&ctx) != 0) return cuda_status(cudaErrorDeviceUninitialized);
  if (ctx == nullptr) {  // nothing current yet: the runtime's default is the primary context
    int dev = 0;
    MJX_CUDA_TRY(cudaGetDevice(&dev));
    MJX_CUDA_TRY(cudaSetDevice(dev));
    if (get_current(&ctx) != 0 || ctx == nullptr) return cuda_status(cudaErrorDeviceUninitialized);
  }
  if (get_id(ctx, id) != 0) return cuda_status(cudaErrorDeviceUninitialized);
  return MJX_OK;
}

static thread_local char g_last_error[256] = "";

void set_last_error(cudaError_t e, const char* file, int line) {
  const char* f = strrchr(file, '/');
  snprintf(g_last_error, sizeof(g_last_error), "%s (%s) at %s:%d", cudaGetErrorName(e),
           cudaGetErrorString(e), f ? f + 1 : file, line);
}

mjx_status check_grid(const mjx_grid2d* g) {
  if (g == nullptr) return MJX_BAD_ARG;
  if (ilog2_exact(g->nx) < 1 || ilog2_exact(g->ny) < 1) return MJX_BAD_SHAPE;
  if (g->nx > 4096 || g->ny > 4096) return MJX_BAD_SHAPE;
  if (!(g->dx > 0) || !(g->dy > 0)) return MJX_BAD_ARG;
  return MJX_OK;
}

int elem_size(int dtype) { return dtype == MJX_F32 ? 4 : (dtype == MJX_F64 ? 8 : 0); }

// Row pass over nfields single fields, pairing rows y and y + ny/2 of each field.
template <typename T>
RowArgs<T> field_rows(const mjx_grid2d* g, int nfields, const PlanView& pv, cx<T>* spec) {
  RowArgs<T> r;
  memset(&r, 0, sizeof(r));
  r.n = g->nx; r.log2n = ilog2_exact(g->nx); r.ldc = spec_ldc(g->nx);
  r.nrows = g->ny / 2; r.npairs = nfields; r.nseq = row_nseq(g->nx, r.nrows);
  r.rstride = g->nx; r.rin_sel = -1; r.rout_sel = -1;
  r.spec = spec; r.tw = (const cx<T>*)pv.twx; r.inv_scale = (T)1;
  for (int f = 0; f < nfields; ++f) {
    r.pr[f].ra = (long long)f * g->ny * g->nx;
    r.pr[f].rb = r.pr[f].ra + (long long)(g->ny / 2) * g->nx;
    r.pr[f].sa = (long long)f * g->ny * r.ldc;
    r.pr[f].sb = r.pr[f].sa + (long long)(g->ny / 2) * r.ldc;
    r.pr[f].hfac = 1.0;
  }
  return r;
}

template <typename T>
ColArgs<T> field_cols(const mjx_grid2d* g, const PlanView& pv, cx<T>* spec, int nout) {
  ColArgs<T> c;
  memset(&c, 0, sizeof(c));
  c.ny = g->ny; c.log2ny = ilog2_exact(g->ny); c.ncols = g->nx / 2 + 1; c.ldc = spec_ldc(g->nx);
  c.C = col_tile(g->ny, c.ncols, nout, sizeof(T));
  c.spec = spec; c.lamx = (const T*)pv.lamx; c.lamy = (const T*)pv.lamy;
  c.tw = (const cx<T>*)pv.twy; c.scale = (T)(1.0 / ((double)g->nx * (double)g->ny));
  return c;
}

template <typename T>
mjx_status spectral_apply(const void* plan, const mjx_grid2d* g, int nfields, const double* D,
                          double h, int mult, const T* in, T* out, void* ws, cudaStream_t s,
                          const double* vx = nullptr, const double* vy = nullptr,
                          const T* mtab = nullptr) {
  const PlanView pv = plan_view(plan, g->ny, g->nx, sizeof(T));
  cx<T>* spec = (cx<T>*)ws;
  const size_t fsz = (size_t)g->ny * g->nx;
  // gather the fields that diffuse (or, for MUL_ADVDIFF, move); pass the others through
  auto moves = [&](int f) { return vx && vy && (fabs(vx[f]) > 1e-14 || fabs(vy[f]) > 1e-14); };
  int idx[4], nd = 0;
  for (int f = 0; f < nfields; ++f) {
    if (mult == MUL_TABLE || D[f] > 1e-14 || moves(f)) idx[nd++] = f;
    else if (mult == MUL_LAP || mult == MUL_ADV_LAP)  // L u = 0
      MJX_CUDA_TRY(cudaMemsetAsync(out + f * fsz, 0, fsz * sizeof(T), s));
    else if (in != out)
      MJX_CUDA_TRY(cudaMemcpyAsync(out + f * fsz, in + f * fsz, fsz * sizeof(T), cudaMemcpyDeviceToDevice, s));
  }
  if (nd == 0) return MJX_OK;
  RowArgs<T> r = field_rows<T>(g, nd, pv, spec);
  for (int i = 0; i < nd; ++i) {
    const long long off = (long long)idx[i] * fsz;
    r.pr[i].ra += off - (long long)i * fsz;
    r.pr[i].rb += off - (long long)i * fsz;
  }
  r.rin[0] = in; r.rout[0] = out;
  for (int i = 0; i < nd; ++i) r.pr[i].flags = ROW_STORE_SPEC;
  MJX_CUDA_TRY((launch_row<T, RX_NONE>(r, s)));
  ColArgs<T> c = field_cols<T>(g, pv, spec, 1);
  c.hfixed = h; c.njobs = nd; c.mtab = mtab;
  c.kxs = 6.283185307179586476925286766559 / ((double)g->nx * g->dx);
  c.kys = 6.283185307179586476925286766559 / ((double)g->ny * g->dy);
  for (int i = 0; i < nd; ++i) {
    ColJob& j = c.job[i];
    j.sin = j.sout[0] = j.sout[1] = (long long)i * g->ny * spec_ldc(g->nx);
    j.D = D[idx[i]]; j.hfac[0] = j.hfac[1] = 1.0; j.pow[0] = j.pow[1] = 1; j.nout = 1; j.mul = mult;
    if (vx && vy) { j.vx = vx[idx[i]]; j.vy = vy[idx[i]]; }
  }
  MJX_CUDA_TRY(launch_col<T>(c, s));
  for (int i = 0; i < nd; ++i) r.pr[i].flags = ROW_LOAD_SPEC | ROW_STORE_REAL;
  MJX_CUDA_TRY((launch_row<T, RX_NONE>(r, s)));
  return MJX_OK;
}

// Bytes of nfields half spectra; FP64 workspaces hold their multiplier table after them.
static size_t spec_bytes(int ny, int nx, int nfields, int elem) {
  return (size_t)nfields * ny * spec_ldc(nx) * 2 * elem;
}

// A step is one column pass and one row pass: the rows go from spectrum to spectrum (c2r, then
// r2c of the same registers and shared memory; the real field of a step that is not the last
// is not stored), and FP64 steps read their multipliers from a table formed once.
template <typename T>
mjx_status fft_cn(const void* plan, const mjx_grid2d* g, double D, double dt, int n_steps,
                  const T* u_in, T* u_out, void* ws, size_t ws_bytes, cudaStream_t s) {
  const PlanView pv = plan_view(plan, g->ny, g->nx, sizeof(T));
  cx<T>* spec = (cx<T>*)ws;
  RowArgs<T> fwd = field_rows<T>(g, 1, pv, spec);
  RowArgs<T> inv = fwd, both = fwd;
  fwd.pr[0].flags = ROW_STORE_SPEC;
  fwd.rin[0] = u_in;
  both.pr[0].flags = ROW_LOAD_SPEC | ROW_STORE_SPEC;
  inv.pr[0].flags = ROW_LOAD_SPEC | ROW_STORE_REAL;
  inv.rout[0] = u_out;
  ColArgs<T> c = field_cols<T>(g, pv, spec, 1);
  c.hfixed = dt; c.njobs = 1;
  c.job[0].D = D; c.job[0].hfac[0] = c.job[0].hfac[1] = 1.0; c.job[0].pow[0] = c.job[0].pow[1] = 1;
  c.job[0].nout = 1; c.job[0].mul = MUL_CN;
  if (n_steps <= 0) {
    if (u_in != u_out)
      MJX_CUDA_TRY(cudaMemcpyAsync(u_out, u_in, sizeof(T) * g->ny * g->nx, cudaMemcpyDeviceToDevice, s));
    return MJX_OK;
  }
  if constexpr (sizeof(T) == 8) {
    const size_t sb = spec_bytes(g->ny, g->nx, 1, 8);
    if (n_steps > 1 && ws_bytes >= sb + sb / 2) MJX_CUDA_TRY(tabulate_cols(c, (double*)ws + sb / 8, s));
  }
  MJX_CUDA_TRY((launch_row<T, RX_NONE>(fwd, s)));
  both.pdl = inv.pdl = c.pdl = 1;
  for (int i = 0; i < n_steps; ++i) {
    MJX_CUDA_TRY(launch_col<T>(c, s));
    MJX_CUDA_TRY((launch_row<T, RX_NONE>(i < n_steps - 1 ? both : inv, s)));
  }
  return MJX_OK;
}

// Fixed device scratch for mjx_fft_cn2d_noalloc.  It lives in the library's
// own device memory: every GPU that loads the library holds these bytes until
// the process exits.  Host code must not pass the symbol itself to a kernel
// (in host code it is only a stand-in); the device address comes from
// cudaGetSymbolAddress, once per CUDA context.
static __device__ __align__(256) unsigned char g_noalloc_scratch[MJX_NOALLOC_SCRATCH_BYTES];

// Scratch addresses by CUDA context.  A __device__ array has a separate
// address in every context that loads the library (the primary context, a
// driver-API context of an embedding host, the new primary context after
// cudaDeviceReset), so the lookup is cached per context id, never per device.
static std::mutex g_noalloc_mu;
static unsigned long long g_noalloc_ctx[32];
static void* g_noalloc_ptr[32];
static int g_noalloc_n = 0;

static mjx_status noalloc_scratch(void** out) {
  unsigned long long ctx = 0;
  MJX_TRY(current_context_id(&ctx));
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  const int m = g_noalloc_n < 32 ? g_noalloc_n : 32;
  for (int i = 0; i < m; ++i)
    if (g_noalloc_ctx[i] == ctx) {
      *out = g_noalloc_ptr[i];
      return MJX_OK;
    }
  void* p = nullptr;
  MJX_CUDA_TRY(cudaGetSymbolAddress(&p, g_noalloc_scratch));
  g_noalloc_ctx[g_noalloc_n % 32] = ctx;
  g_noalloc_ptr[g_noalloc_n % 32] = p;
  ++g_noalloc_n;
  *out = p;
  return MJX_OK;
}

}  // namespace mjx

using namespace mjx;

extern "C" {

const char* mjx_version(void) { return "moljax_gb300 0.1.0 (sm_103a)"; }

const char* mjx_last_error(void) { return g_last_error; }

const char* mjx_status_string(int st) {
  switch (st) {
    case MJX_OK: return "ok";
    case MJX_BAD_SHAPE: return "unsupported or inconsistent shape";
    case MJX_BAD_DTYPE: return "unsupported dtype";
    case MJX_NOT_FINITE: return "non-finite values";
    case MJX_MAX_ITERS: return "maximum steps/iterations reached";
    case MJX_DT_TOO_SMALL: return "time step below dt_min";
    case MJX_NK_FAILED: return "Newton-Krylov failed";
    case MJX_OOM: return "out of memory";
    case MJX_CUDA_ERROR: return "CUDA error";
    case MJX_BAD_ARG: return "bad argument";
    case MJX_WORKSPACE: return "workspace too small";
    default: return "unknown status";
  }
}

size_t mjx_spec2d_plan_bytes(int ny, int nx, int dtype) {
  const int e = elem_size(dtype);
  if (!e || ilog2_exact(nx) < 1 || ilog2_exact(ny) < 1) return 0;
  return plan_bytes(ny, nx, e);
}

size_t mjx_spec2d_ws_bytes(int ny, int nx, int nfields, int dtype) {
  const int e = elem_size(dtype);
  if (!e || ilog2_exact(nx) < 1 || ilog2_exact(ny) < 1 || nfields < 1) return 0;
  const size_t sb = spec_bytes(ny, nx, nfields, e);
  return e == 8 ? sb + sb / 2 : sb;
}

mjx_status mjx_spec2d_plan_init(void* plan, const mjx_grid2d* g, int symbol, int dtype,
                                void* stream) {
  MJX_TRY(check_grid(g));
  const int e = elem_size(dtype);
  if (!e) return MJX_BAD_DTYPE;
  if (plan == nullptr) return MJX_BAD_ARG;
  if (symbol != MJX_SYMBOL_FD && symbol != MJX_SYMBOL_SPECTRAL) return MJX_BAD_ARG;
  const int nx = g->nx, ny = g->ny, ldc = spec_ldc(nx);
  const size_t bytes = plan_bytes(ny, nx, e);
  std::vector<unsigned char> host(bytes, 0);
  PlanView pv = plan_view(host.data(), ny, nx, e);
  const double twopi = 6.283185307179586476925286766559;
  auto put_tw = [&](const void* dst, int n) {
    for (int j = 0; j < n; ++j) {
      const double ang = twopi * (double)j / (double)n;
      const double c = cos(ang), s = -sin(ang);
      if (e == 4) { float* p = (float*)dst; p[2 * j] = (float)c; p[2 * j + 1] = (float)s; }
      else { double* p = (double*)dst; p[2 * j] = c; p[2 * j + 1] = s; }
    }
    if (e == 4) {
      fft_pass_table((float*)dst, n);
    } else {
      double* p = (double*)dst + 2 * n;
      const Roots roots(n);
      for (int j = 0; j < n; ++j) tile_twiddle(roots, j, 8, &p[2 * j], &p[2 * j + 1]);
    }
  };
  // eigenvalue of the 1D periodic Laplacian for integer frequency m on n points of spacing d
  auto lam1 = [&](int m, int n, double d) {
    if (symbol == MJX_SYMBOL_FD) return (2.0 * cos(twopi * (double)m / (double)n) - 2.0) / (d * d);
    const double k = twopi * (double)m / ((double)n * d);
    return -k * k;
  };
  put_tw(pv.twx, nx);
  if (e == 4 && nx == 1024) {  // the transposed copy for the one-warp 1024-point transform
    float* p = (float*)pv.twx;
    for (int k1 = 0; k1 < 32; ++k1)
      for (int l = 0; l < 32; ++l) {
        p[2 * (kW1024 + 32 * k1 + l)] = p[2 * (l * k1)];
        p[2 * (kW1024 + 32 * k1 + l) + 1] = p[2 * (l * k1) + 1];
      }
  }
  if (ny == nx && e == 8) memcpy((void*)pv.twy, pv.twx, (size_t)twy_count(ny, e) * 2 * e);
  else put_tw(pv.twy, ny);
  for (int kx = 0; kx < ldc; ++kx) {
    const double v = kx <= nx / 2 ? lam1(kx, nx, g->dx) : 0.0;
    if (e == 4) ((float*)pv.lamx)[kx] = (float)v; else ((double*)pv.lamx)[kx] = v;
  }
  for (int ky = 0; ky < ny; ++ky) {
    const int m = ky < ny / 2 ? ky : ky - ny;  // fftfreq order
    const double v = lam1(m, ny, g->dy);
    if (e == 4) ((float*)pv.lamy)[ky] = (float)v; else ((double*)pv.lamy)[ky] = v;
  }
  MJX_CUDA_TRY(cudaMemcpyAsync(plan, host.data(), bytes, cudaMemcpyHostToDevice, (cudaStream_t)stream));
  MJX_CUDA_TRY(cudaStreamSynchronize((cudaStream_t)stream));
  return MJX_OK;
}

mjx_status mjx_spectral_apply2d(const void* plan, const mjx_grid2d* g, int dtype, int nfields,
                                const double* D, double h, int mult, const void* in, void* out,
                                void* ws, size_t ws_bytes, void* stream) {
  MJX_TRY(check_grid(g));
  if (nfields < 1 || nfields > 4 || D == nullptr || plan == nullptr || in == nullptr || out == nullptr)
    return MJX_BAD_ARG;
  if ((mult < MJX_MULT_SCALE || mult > MJX_MULT_EXP) && mult != MJX_MULT_LAP) return MJX_BAD_ARG;
  const int e = elem_size(dtype);
  if (!e) return MJX_BAD_DTYPE;
  if (ws == nullptr || ws_bytes < spec_bytes(g->ny, g->nx, nfields, e)) return MJX_WORKSPACE;
  MJX_TRY(ensure_kernel_attrs());
  cudaStream_t s = (cudaStream_t)stream;
  if (e == 4) return spectral_apply<float>(plan, g, nfields, D, h, mult, (const float*)in, (float*)out, ws, s);
  return spectral_apply<double>(plan, g, nfields, D, h, mult, (const double*)in, (double*)out, ws, s);
}

mjx_status mjx_advdiff_op2d(const void* plan, const mjx_grid2d* g, int dtype, int nfields,
                            const double* D, const double* vx, const double* vy, double h, int op,
                            const void* in, void* out, void* ws, size_t ws_bytes, void* stream) {
  MJX_TRY(check_grid(g));
  if (nfields < 1 || nfields > 4 || D == nullptr || vx == nullptr || vy == nullptr || plan == nullptr ||
      in == nullptr || out == nullptr || op < 0 || op > 3)
    return MJX_BAD_ARG;
  const int e = elem_size(dtype);
  if (!e) return MJX_BAD_DTYPE;
  if (ws == nullptr || ws_bytes < spec_bytes(g->ny, g->nx, nfields, e)) return MJX_WORKSPACE;
  MJX_TRY(ensure_kernel_attrs());
  cudaStream_t s = (cudaStream_t)stream;
  const int mul = op == 0 ? MUL_ADVDIFF : (op == 1 ? MUL_ADV_LAP : (op == 2 ? MUL_ADV_EXP : MUL_ADV_CN));
  if (e == 4)
    return spectral_apply<float>(plan, g, nfields, D, h, mul, (const float*)in, (float*)out, ws, s, vx, vy);
  return spectral_apply<double>(plan, g, nfields, D, h, mul, (const double*)in, (double*)out, ws, s, vx, vy);
}

mjx_status mjx_spectral_filter2d(const void* plan, const mjx_grid2d* g, int dtype, int nfields,
                                 const void* table, const void* in, void* out, void* ws, size_t ws_bytes,
                                 void* stream) {
  MJX_TRY(check_grid(g));
  if (nfields < 1 || nfields > 4 || plan == nullptr || table == nullptr || in == nullptr || out == nullptr)
    return MJX_BAD_ARG;
  const int e = elem_size(dtype);
  if (!e) return MJX_BAD_DTYPE;
  if (ws == nullptr || ws_bytes < spec_bytes(g->ny, g->nx, nfields, e)) return MJX_WORKSPACE;
  MJX_TRY(ensure_kernel_attrs());
  cudaStream_t s = (cudaStream_t)stream;
  const double D[4] = {1.0, 1.0, 1.0, 1.0};
  if (e == 4)
    return spectral_apply<float>(plan, g, nfields, D, 1.0, MUL_TABLE, (const float*)in, (float*)out, ws, s,
                                 nullptr, nullptr, (const float*)table);
  return spectral_apply<double>(plan, g, nfields, D, 1.0, MUL_TABLE, (const double*)in, (double*)out, ws, s,
                                nullptr, nullptr, (const double*)table);
}

mjx_status mjx_advdiff_apply2d(const void* plan, const mjx_grid2d* g, int dtype, int nfields,
                               const double* D, const double* vx, const double* vy, double h,
                               const void* in, void* out, void* ws, size_t ws_bytes, void* stream) {
  MJX_TRY(check_grid(g));
  if (nfields < 1 || nfields > 4 || D == nullptr || vx == nullptr || vy == nullptr || plan == nullptr ||
      in == nullptr || out == nullptr)
    return MJX_BAD_ARG;
  const int e = elem_size(dtype);
  if (!e) return MJX_BAD_DTYPE;
  if (ws == nullptr || ws_bytes < spec_bytes(g->ny, g->nx, nfields, e)) return MJX_WORKSPACE;
  MJX_TRY(ensure_kernel_attrs());
  cudaStream_t s = (cudaStream_t)stream;
  if (e == 4)
    return spectral_apply<float>(plan, g, nfields, D, h, MUL_ADVDIFF, (const float*)in, (float*)out, ws, s, vx, vy);
  return spectral_apply<double>(plan, g, nfields, D, h, MUL_ADVDIFF, (const double*)in, (double*)out, ws, s, vx, vy);
}

mjx_status mjx_fft_cn2d(const void* plan, const mjx_grid2d* g, int dtype, double D, double dt,
                        int n_steps, const void* u_in, void* u_out, void* ws, size_t ws_bytes,
                        void* stream) {
  MJX_TRY(check_grid(g));
  if (plan == nullptr || u_in == nullptr || u_out == nullptr || n_steps < 0) return MJX_BAD_ARG;
  const int e = elem_size(dtype);
  if (!e) return MJX_BAD_DTYPE;
  if (ws == nullptr || ws_bytes < spec_bytes(g->ny, g->nx, 1, e)) return MJX_WORKSPACE;
  MJX_TRY(ensure_kernel_attrs());
  cudaStream_t s = (cudaStream_t)stream;
  if (e == 4) return fft_cn<float>(plan, g, D, dt, n_steps, (const float*)u_in, (float*)u_out, ws, ws_bytes, s);
  return fft_cn<double>(plan, g, D, dt, n_steps, (const double*)u_in, (double*)u_out, ws, ws_bytes, s);
}

// FFT-CN stepping for callers that cannot allocate device memory: the
// spectrum scratch is the fixed library buffer above instead of a workspace.
mjx_status mjx_fft_cn2d_noalloc(const void* plan, const mjx_grid2d* g, int dtype, double D, double dt,
                                int n_steps, const void* u_in, void* u_out, void* stream) {
  MJX_TRY(check_grid(g));
  if (plan == nullptr || u_in == nullptr || u_out == nullptr || n_steps < 0) return MJX_BAD_ARG;
  const int e = elem_size(dtype);
  if (!e) return MJX_BAD_DTYPE;
  // the spectrum of one field must fit the fixed scratch
  if (spec_bytes(g->ny, g->nx, 1, e) > (size_t)MJX_NOALLOC_SCRATCH_BYTES) return MJX_WORKSPACE;
  void* ws = nullptr;
  MJX_TRY(noalloc_scratch(&ws));  // first call on a device: symbol lookup (no allocation)
  MJX_TRY(ensure_kernel_attrs());
  cudaStream_t s = (cudaStream_t)stream;
  if (e == 4) return fft_cn<float>(plan, g, D, dt, n_steps, (const float*)u_in, (float*)u_out, ws, MJX_NOALLOC_SCRATCH_BYTES, s);
  return fft_cn<double>(plan, g, D, dt, n_steps, (const double*)u_in, (double*)u_out, ws, MJX_NOALLOC_SCRATCH_BYTES, s);
}

}  // extern "C"
