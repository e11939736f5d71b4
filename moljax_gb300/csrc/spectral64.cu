// FP64 row and column spectral passes for lengths up to 2048 (spectral.cuh describes the
// passes; row_kernel and col_kernel of spectral.cu are their FP32 form).
//
// GB300 runs an FP64 instruction of a warp in 64 cycles of its sub-partition, whatever the
// number of active lanes (1.7 lanes a clock and SM), so these passes are bound by FP64 issue
// once the SMs are full and by the longest chain of one warp where they are not.  Hence the
// flat tile transform with (cos, tan) twiddles (tfft.cuh): 18.5 FP64 instructions a point at
// n = 128 against 22 for radix 16 with rebuilt twiddles or radix 4, full warps, and the radix
// chosen so that each sub-partition gets one.  Steps of fixed size read their multipliers from
// a table (a division or an exponential is 12 to 25 FP64 instructions a point).  Measured with
// the table and the fused row pass of fft_cn and apply3d (spectral.cu, spectral3d.cu):
//   FFT-CN 128^2, 100 steps   4713 -> 1790 us
//   FFT-CN 128^3, 10 steps    4754 -> 3060 us
//   Strang 256^2, 100 steps   4665 -> 3015 us
// What bounds them now: in the box's passes FP64 issue (82 to 86 % of the busy SMs' rate); at 256^2
// (128 and 130 CTAs of four warps) it is 55 % of it in the rows and 43 % in the columns, the rest the
// dependent chain of one warp a sub-partition; at 128^2 that chain (seven radix-2 passes, 23 %).
// Columns of 4096 rows in col_kernel<double, 12>: a step at 4096 x 64 and 4096 x 1024 133 and 686 us
// (164 and 820 with every element in shared memory between the transforms).
// Longer transforms stay with spectral.cu: two buffers of 4096 FP64 points leave one CTA an SM
// and no second phase to overlap with.
#include <string.h>

#include "spectral.cuh"
#include "tfft.cuh"

namespace mjx {

struct Geo64 {
  int lS, threads, odd, staged;
  unsigned long long rad;
  size_t smem;
};

// Tile of `total` sequences of length n = 2^log2n (elements of `nout` outputs a sequence at the
// end): about 1024 points a CTA, fewer sequences until there is about one CTA per SM; `fixed`
// >= 0 gives the sequences (log2) instead.  The radix falls from 8 while the warps that an SM
// gets are fewer than its four sub-partitions.
static Geo64 geo64(int n, int log2n, long long total, int nout, int cap, int fixed) {
  Geo64 g;
  int l = 0;
  while (l < cap && (n << (l + 1)) <= 1024) ++l;
  if (l < 1 && cap >= 1) l = 1;  // a 32-byte sector of two columns
  while (l > 0 && (total + (1 << l) - 1) >> l < 128) --l;
  if (fixed >= 0) l = fixed;
  const long long ctas = (total + (1 << l) - 1) >> l;
  const long long per_sm = ctas < 152 ? 1 : ctas / 152;
  int top = 8;
  while (top > 2 && (((n / top) << l) + 31) / 32 * per_sm < 4) top >>= 1;
  int passes = 0;
  g.rad = tile_pow2_radices(log2n, top, &passes);
  g.odd = passes & 1;
  g.lS = l;
  g.threads = (((n / top) << l) + 31) & ~31;
  if (g.threads < 128) g.threads = 128;
  if (g.threads > 256) g.threads = 256;
  const size_t buf = 2 * (size_t)sp_size((n * nout) << l) * sizeof(double2);
  g.staged = buf + n * sizeof(double2) <= 100 * 1024;
  g.smem = buf + (g.staged ? n * sizeof(double2) : 0);
  return g;
}

// the (cos, tan) table that follows the plan's FP64 twiddles, staged in shared memory if it fits
__device__ __forceinline__ const double2* stage_tw(const double2* tw, double2* smem, int n, int staged, int tid, int nth) {
  if (!staged) return tw + n;
  for (int i = tid; i < n; i += nth) smem[i] = __ldg(&tw[n + i]);
  return smem;
}

template <int RX>
__global__ void __launch_bounds__(256) row64_kernel(const __grid_constant__ RowArgs<double> a, const Geo64 g) {
  typedef double2 C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const DevState* st = a.st;
  const int n = a.n, half = n >> 1, lS = g.lS, S = 1 << lS, tid = threadIdx.x, nth = blockDim.x;
  C* cur = reinterpret_cast<C*>(smem_raw);
  C* alt = cur + sp_size(n << lS);
  const C* tw = stage_tw(a.tw, alt + sp_size(n << lS), n, g.staged, tid, nth);
  pdl_wait();
  if (st != nullptr && st->done) return;
  const int seq0 = blockIdx.x << lS;
  const int q = seq0 / a.nrows;  // uniform within the CTA (nrows % S == 0)
  const RowPair pr = a.pr[q];
  const int flags = pr.flags;
  const long long y0 = seq0 - q * a.nrows;
  const int cu = st != nullptr ? st->cur : 0;
  const int ldc = a.ldc, lh = a.log2n - 1;

  // 1. spectrum rows to the conjugate of Z = A + i B, and its forward transform (the inverse by
  // conjugation); points k < n/2 of all rows flat over the threads, then the Nyquist points
  if (flags & ROW_LOAD_SPEC) {
    const C* A = a.spec + pr.sa + y0 * ldc;
    const C* B = a.spec + pr.sb + y0 * ldc;
    for (int e = tid; e < (half << lS); e += nth) {
      const int s = e >> lh, k = e & (half - 1), g0 = s * ldc + k;
      const C u = A[g0], v = B[g0];
      cur[sp((k << lS) + s)] = mk<C>(u.x - v.y, -(u.y + v.x));
      if (k > 0) cur[sp(((n - k) << lS) + s)] = mk<C>(u.x + v.y, u.y - v.x);
    }
    if (tid < S) {
      const C u = A[tid * ldc + half], v = B[tid * ldc + half];
      cur[sp((half << lS) + tid)] = mk<C>(u.x - v.y, -(u.y + v.x));
    }
    __syncthreads();
    tile_dft<double, true>(cur, alt, n, g.rad, lS, tw, tid, nth);
    if (g.odd) { C* t = cur; cur = alt; alt = t; }
  }

  // 2. pointwise work on the real rows
  const double sc = a.inv_scale;
  double h = 0.0;
  if (flags & ROW_REACT) h = (st != nullptr ? st->dtc : a.hfixed) * pr.hfac;
  double esum = 0.0;
  int bad = 0;
  const double pF = a.F, pK = a.k, pR = a.r, pFK = a.F + a.k;
  const long long oa = pr.ra + y0 * a.rstride, ob = pr.rb + y0 * a.rstride;
  const double* rin = a.rin_sel < 0 ? a.rin[0] : a.rin[a.rin_sel == 0 ? cu : 1 - cu];
  double* rout = a.rout_sel < 0 ? a.rout[0] : a.rout[a.rout_sel == 0 ? cu : 1 - cu];
  const int rs = (int)a.rstride;
  for (int e = tid; e < (n << lS); e += nth) {
    const int s = e >> (lh + 1), x = e & (n - 1), at = sp((x << lS) + s), i = s * rs + x;
    double va, vb;
    if (flags & ROW_LOAD_SPEC) {
      const C v = cur[at];
      va = v.x * sc;
      vb = -v.y * sc;
    } else {
      va = rin[oa + i];
      vb = rin[ob + i];
    }
    if (flags & ROW_NONLIN) nonlin_terms<double, RX>(va, vb, pF, pFK, pR);
    if (flags & ROW_REACT) {
      if (flags & ROW_DELTA) {
        react_delta<double, RX>(va, vb, h, pF, pK, pR);
      } else if (flags & ROW_EULER) {
        react_euler<double, RX>(va, vb, h, pF, pK, pR);
        if (flags & ROW_EULER2) react_euler<double, RX>(va, vb, h, pF, pK, pR);
      } else {
        react_heun<double, RX>(va, vb, h, pF, pK, pR);
      }
    }
    if (flags & ROW_STORE_REAL) { rout[oa + i] = va; rout[ob + i] = vb; }
    if (flags & ROW_ERRNORM) {
      // moljax/core/state.py:335-339: (err / (atol + rtol |y_new|))^2
      const double da = (va - a.eref[oa + i]) / (a.atol + a.rtol * fabs(va));
      const double db = (vb - a.eref[ob + i]) / (a.atol + a.rtol * fabs(vb));
      esum += da * da + db * db;
      bad |= !(isfinite(va) && isfinite(vb));
    }
    if (flags & ROW_ERRPAIR) {
      const double da = va / (a.atol + a.rtol * fabs(vb));
      esum += da * da;
      bad |= !(isfinite(va) && isfinite(vb));
    }
    if (flags & ROW_STORE_SPEC) cur[at] = mk<C>(va, vb);
  }

  // 3. r2c and split into the two half spectra
  if (flags & ROW_STORE_SPEC) {
    __syncthreads();
    tile_dft<double, true>(cur, alt, n, g.rad, lS, tw, tid, nth);
    if (g.odd) { C* t = cur; cur = alt; alt = t; }
    C* A = a.spec + ((flags & ROW_SPEC_ALT) ? pr.oa : pr.sa) + y0 * ldc;
    C* B = a.spec + ((flags & ROW_SPEC_ALT) ? pr.ob : pr.sb) + y0 * ldc;
    auto split = [&](int s, int k) {
      const C Zk = cur[sp((k << lS) + s)], Zm = cur[sp((((n - k) & (n - 1)) << lS) + s)];
      A[s * ldc + k] = mk<C>(0.5 * (Zk.x + Zm.x), 0.5 * (Zk.y - Zm.y));
      B[s * ldc + k] = mk<C>(0.5 * (Zk.y + Zm.y), 0.5 * (Zm.x - Zk.x));
    };
    for (int e = tid; e < (half << lS); e += nth) split(e >> lh, e & (half - 1));
    if (tid < S) split(tid, half);
  }

  // 4. block reduction of the error partials
  if (flags & (ROW_ERRNORM | ROW_ERRPAIR)) {
    __shared__ double red[8];
    __shared__ int redbad[8];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      esum += __shfl_xor_sync(0xffffffffu, esum, o);
      bad |= __shfl_xor_sync(0xffffffffu, bad, o);
    }
    if ((tid & 31) == 0) { red[tid >> 5] = esum; redbad[tid >> 5] = bad; }
    __syncthreads();
    if (tid == 0) {
      double s = 0.0, c = 0.0;  // Kahan
      int b2 = 0;
      for (int i = 0; i < (nth >> 5); ++i) {
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
}

// C = 2^lS columns of one job (blockIdx.y), one or two outputs side by side.
__global__ void __launch_bounds__(256) col64_kernel(const __grid_constant__ ColArgs<double> a, const Geo64 g, int lout) {
  typedef double2 C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const ColJob jb = a.job[blockIdx.y];
  const int ny = a.ny, lC = g.lS, Cn = 1 << lC, tid = threadIdx.x, nth = blockDim.x;
  const int nout = jb.nout, lW = lC + (nout > 1 ? 1 : 0);
  C* cur = reinterpret_cast<C*>(smem_raw);
  const int bufn = sp_size(ny << (lC + lout));
  C* alt = cur + bufn;
  const C* tw = stage_tw(a.tw, alt + bufn, ny, g.staged, tid, nth);
  pdl_wait();
  if (a.st != nullptr && a.st->done) return;
  const int kx0 = blockIdx.x << lC;
  const long long ldc = a.ldc;
  C* spec = a.spec + (long long)blockIdx.z * a.pstride;
  const int dirs = jb.dirs ? jb.dirs : 3;

  const C* in = spec + jb.sin + kx0;
  for (int e = tid; e < (ny << lC); e += nth) {
    const int ky = e >> lC, c = e & (Cn - 1);
    C v = kx0 + c < a.ncols ? in[ky * ldc + c] : mk<C>(0.0, 0.0);
    if (!(dirs & 1)) v.y = -v.y;
    cur[sp(e)] = v;
  }
  __syncthreads();
  if (dirs & 1) {
    tile_dft<double, true>(cur, alt, ny, g.rad, lC, tw, tid, nth);
    if (g.odd) { C* t = cur; cur = alt; alt = t; }
  }
  if (dirs == 3 || jb.mul != MUL_SCALE || jb.scale != 1.0) {
    const double jscale = jb.scale != 0.0 ? jb.scale : a.scale;
    const double h = a.st != nullptr ? a.st->dtc : a.hfixed;
    const double hD0 = h * jb.hfac[0] * jb.D, hD1 = h * jb.hfac[1] * jb.D;
    const bool two = nout > 1, conj = (dirs & 2) != 0;
    C* dst = two ? alt : cur;
    for (int e = tid; e < (ny << lC); e += nth) {
      const int ky = e >> lC, c = e & (Cn - 1), kx = kx0 + c;
      C v = cur[sp(e)];
      if (!(dirs & 1)) v.y = -v.y;
      double mr = jscale, mi = 0.0, m1 = 0.0;
      if (jb.mul == MUL_TABLED) {
        mr = kx < a.ncols ? a.mtab[jb.sin + ky * ldc + kx] : 0.0;
      } else if (jb.mul == MUL_TABLE) {
        mr = kx < a.ncols ? jscale * a.mtab[ky * ldc + kx] : 0.0;
      } else if (jb.mul != MUL_SCALE) {
        double lam = a.lamy[ky];
        if (kx < a.ncols) lam += a.ldc3 ? a.lamx[kx % a.ldc3] + a.lamy2[kx / a.ldc3] : a.lamx[kx];
        if (jb.mul == MUL_ADVDIFF || jb.mul == MUL_ADV_LAP || jb.mul == MUL_ADV_EXP || jb.mul == MUL_ADV_CN) {
          const double2 f = adv_multiplier<double>(a, jb, hD0, h * jb.hfac[0], lam, kx, ky);
          mr = f.x * jscale; mi = f.y * jscale;
        } else {
          mr = jscale * multiplier<double>(jb.mul, hD0, lam, jb.pow[0]);
          if (two) m1 = jscale * multiplier<double>(jb.mul, hD1, lam, jb.pow[1]);
        }
      }
      C w = mk<C>(v.x * mr, v.y * mr);
      if (mi != 0.0) w = mk<C>(v.x * mr - v.y * mi, v.x * mi + v.y * mr);
      if (conj) w.y = -w.y;
      dst[sp((ky << lW) + c)] = w;
      if (two) dst[sp((ky << lW) + Cn + c)] = mk<C>(v.x * m1, conj ? -v.y * m1 : v.y * m1);
    }
    if (two) { C* t = cur; cur = alt; alt = t; }
    __syncthreads();
  }
  if (dirs & 2) {
    tile_dft<double, true>(cur, alt, ny, g.rad, lW, tw, tid, nth);
    if (g.odd) { C* t = cur; cur = alt; alt = t; }
  }
  for (int e = tid; e < (ny << lW); e += nth) {
    const int ky = e >> lW, col = e & ((1 << lW) - 1), c = col & (Cn - 1);
    C v = cur[sp(e)];
    if (dirs & 2) v.y = -v.y;
    if (kx0 + c < a.ncols) (spec + jb.sout[col >> lC] + kx0)[ky * ldc + c] = v;
  }
}

// Multipliers of fixed-size steps, with the normalisation, for MUL_TABLED: entry sin + ky ldc + kx
__global__ void col_table_kernel(const __grid_constant__ ColArgs<double> a, double* tab) {
  const ColJob jb = a.job[blockIdx.y];
  const double jscale = jb.scale != 0.0 ? jb.scale : a.scale, hD = a.hfixed * jb.hfac[0] * jb.D;
  const long long total = (long long)a.ny * a.ncols;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int ky = (int)(i / a.ncols), kx = (int)(i - (long long)ky * a.ncols);
    const double lxy = a.ldc3 ? a.lamx[kx % a.ldc3] + a.lamy2[kx / a.ldc3] : a.lamx[kx];
    tab[jb.sin + (long long)ky * a.ldc + kx] = jscale * multiplier<double>(jb.mul, hD, lxy + a.lamy[ky], jb.pow[0]);
  }
}

cudaError_t tabulate_cols(ColArgs<double>& a, double* tab, cudaStream_t s) {
  dim3 grid(152 * 2, a.njobs);
  col_table_kernel<<<grid, 256, 0, s>>>(a, tab);
  a.mtab = tab;
  for (int j = 0; j < a.njobs; ++j) a.job[j].mul = MUL_TABLED;
  return cudaGetLastError();
}

bool row64_takes(int n) { return n >= 2 && n <= 2048; }
bool col64_takes(int ny) { return ny >= 2 && ny <= 2048; }

template <int RX>
cudaError_t launch_row64(const RowArgs<double>& a, cudaStream_t s) {
  bool partials = false;
  for (int q = 0; q < a.npairs && q < MJX_MAXPAIR; ++q)
    partials |= (a.pr[q].flags & (ROW_ERRNORM | ROW_ERRPAIR)) != 0;
  int cap = 0;  // sequences of a CTA lie in one pair: S divides nrows
  while (cap < 5 && a.nrows % (2 << cap) == 0) ++cap;
  int fixed = -1;
  if (partials)  // their CTA count sizes the controller's reduction
    for (fixed = 0; (1 << fixed) < a.nseq; ++fixed) {}
  const Geo64 g = geo64(a.n, a.log2n, (long long)a.npairs * a.nrows, 1, cap, fixed);
  return launch_chain(row64_kernel<RX>, dim3((unsigned)((long long)a.npairs * a.nrows >> g.lS)), g.threads, g.smem, s,
                      a.pdl, a, g);
}
template cudaError_t launch_row64<RX_NONE>(const RowArgs<double>&, cudaStream_t);
template cudaError_t launch_row64<RX_GRAY_SCOTT>(const RowArgs<double>&, cudaStream_t);
template cudaError_t launch_row64<RX_FISHER>(const RowArgs<double>&, cudaStream_t);

cudaError_t launch_col64(const ColArgs<double>& a, cudaStream_t s) {
  int lout = 0;
  for (int j = 0; j < a.njobs; ++j) lout |= a.job[j].nout > 1;
  const int planes = a.nplanes > 1 ? a.nplanes : 1;
  Geo64 g = geo64(a.ny, a.log2ny, (long long)a.ncols * a.njobs * planes, 1 << lout, 4, -1);
  while (g.lS > 0 && g.smem > 200 * 1024)
    g = geo64(a.ny, a.log2ny, (long long)a.ncols * a.njobs * planes, 1 << lout, 4, g.lS - 1);
  dim3 grid((a.ncols + (1 << g.lS) - 1) >> g.lS, a.njobs, planes);
  return launch_chain(col64_kernel, grid, g.threads, g.smem, s, a.pdl, a, g, lout);
}

mjx_status spectral64_attrs(int optin) {
  const void* k[4] = {(const void*)row64_kernel<RX_NONE>, (const void*)row64_kernel<RX_GRAY_SCOTT>,
                      (const void*)row64_kernel<RX_FISHER>, (const void*)col64_kernel};
  for (int i = 0; i < 4; ++i) {
    cudaFuncAttributes fa;
    MJX_CUDA_TRY(cudaFuncGetAttributes(&fa, k[i]));
    MJX_CUDA_TRY(cudaFuncSetAttribute(k[i], cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes));
  }
  return MJX_OK;
}

}  // namespace mjx
