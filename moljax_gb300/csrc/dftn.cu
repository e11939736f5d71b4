// Spectral multipliers on periodic 2D grids and 3D boxes of any size (numpy/jnp.fft accept any
// n; the fused row/column passes of spectral.cu take powers of two).
//
// out_f = real(IFFT2( m(kx, ky) FFT2(in_f) )) on the half spectrum kx = 0..nx/2:
//   R   r2c of row pairs (two real rows ride one complex DFT)   spec[f][y][ld]
//   C   forward DFT along y, multiplier, inverse DFT, in place
//   R'  c2r of row pairs
// and on a box R, C along y per plane, C along z with the multiplier, C along y back, R'.
// Several applications in a row fuse R' with the next R (rows go from spectrum to spectrum)
// and read the multiplier from a table formed once.  A DFT of length n is the shared-memory
// Stockham FFT when n is a power of two, a mixed-radix (2, 3, 4, 5) Stockham FFT when n has no
// other prime factor, and Bluestein's chirp-z form otherwise: with c[j] = exp(-i pi j^2 / n),
//   DFT_n(z)[k] = c[k] * IFFT_L( FFT_L(z c) * FFT_L(b) )[k],  b[j] = conj(c[|j|]),
// a circular convolution of length L = 2^ceil(log2(2n - 1)) <= 4096 (n <= 2048).
// Inverse DFTs use IDFT(z) = conj(DFT(conj(z))) / n.  The reference keeps real(ifft2(.)); on
// the half spectrum that is the multiplier (m(k) + conj(m(-k))) / 2, which equals m(k) but on
// the Nyquist lines of the advection forms and for tables without that symmetry.
//
// The full-spectrum form that this replaces (real to complex, row DFTs, transpose, column
// DFTs, a multiplier pass with FP64 cosines per point, and back: nine launches in 2D, fourteen
// in 3D) took 127 us a step at 450 x 600 FP32 and 626 us at 100^3 FP64; this one 17.4 us and
// 198 us.  What bounds it: launch and barrier latency on L2-resident grids, FP64 issue.
// Its rounding: a full spectrum holds every mode twice and its real part averages their errors,
// so a single application here has up to 1.3 times that form's error in FP32 (600 x 450: 2.2e-7
// against 1.7e-7 for a transform pair); over the steps of FFT-CN, whose scaling it does in one
// product, 0.81 (2D) and 0.86 (3D) of it on average, in FP64 0.77 and 0.58 (tfft.cuh, roots.cuh).
#include <math.h>
#include <string.h>

#include <vector>

#include "autotune.cuh"
#include "tfft.cuh"

namespace mjx {

mjx_status ensure_kernel_attrs();
int elem_size(int dtype);
void set_last_error(cudaError_t e, const char* file, int line);

static inline size_t g256(size_t b) { return (b + 255) & ~size_t(255); }

struct DftGeom {
  int n, L, log2L, bluestein, mixed, nrad;
  int rad[16];
  size_t tw, chirp, bhat, sym, total;
};

// radices 4, 2, 3, 5 covering n, or 0 if n has another prime factor
static int radix_plan(int n, int* rad) {
  int m = n, k = 0;
  const int rs[4] = {4, 2, 3, 5};
  for (int i = 0; i < 4; ++i)
    while (m % rs[i] == 0 && k < 16) { rad[k++] = rs[i]; m /= rs[i]; }
  return m == 1 ? k : 0;
}

static DftGeom dft_geom(int n, int elem) {
  DftGeom g;
  memset(&g, 0, sizeof(g));
  g.n = n;
  const bool pow2 = ilog2_exact(n) >= 0;
  g.nrad = pow2 ? 0 : radix_plan(n, g.rad);
  g.mixed = !pow2 && g.nrad > 0;
  DftTune t;
  if (g.mixed && tune_dft_get(n, elem, &t) && t.nrad > 0) {  // an autotuned schedule
    g.nrad = t.nrad;
    for (int i = 0; i < 16; ++i) g.rad[i] = t.rad[i];
  }
  g.bluestein = !pow2 && !g.mixed;
  g.L = n;
  if (g.bluestein) {
    g.L = 1;
    while (g.L < 2 * n - 1) g.L <<= 1;
  }
  g.log2L = g.mixed ? 0 : ilog2_exact(g.L);
  const size_t c = 2 * (size_t)elem;
  size_t o = 0;
  g.tw = o; o += g256(g.L * c);
  g.chirp = o; o += g256(n * c);
  g.bhat = o; o += g256(g.L * c);
  g.sym = o; o += g256((size_t)2 * n * sizeof(double));  // d^2 lambda: FD, then spectral
  g.total = o;
  return g;
}

static bool dft_len_ok(int n) {
  if (n < 1) return false;
  if (ilog2_exact(n) >= 0) return n <= 4096;
  return n <= 2048;
}

// ------------------------------------------------------------------ row pass
enum { GROW_LOAD_SPEC = 1, GROW_STORE_REAL = 2, GROW_STORE_SPEC = 4 };

template <typename T>
struct GRowArgs {
  Dft<T> d;
  const T* in;        // real rows of n values
  T* out;
  cx<T>* spec;        // half-spectrum rows, stride ld
  long long nrows;    // real rows of a field; pair q holds rows 2q and 2q + 1
  int ld, lS, flags;
};

// S = 2^lS row pairs per CTA; blockIdx.y is the field.
template <typename T>
__global__ void __launch_bounds__(512) grow_kernel(const __grid_constant__ GRowArgs<T> a) {
  typedef cx<T> C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n = a.d.n, hx = n / 2 + 1, lS = a.lS, S = 1 << lS, tid = threadIdx.x, nth = blockDim.x;
  Tile<T> t = tile_begin<T>(a.d, smem_raw, lS);
  pdl_wait();
  const long long r0 = ((long long)blockIdx.x << lS) * 2;  // first row of this CTA
  const T* in = a.in + blockIdx.y * a.nrows * n;
  T* out = a.out + blockIdx.y * a.nrows * n;
  C* spec = a.spec + blockIdx.y * a.nrows * a.ld;
  const float rn = 1.0f / (float)n, rh = 1.0f / (float)hx;
  if (a.flags & GROW_LOAD_SPEC) {
    // conj of Z_k = A_k + i B_k and Z_{n-k} = conj(A_k) + i conj(B_k)
    for (int e = tid; e < S * hx; e += nth) {
      const int s = fdiv(e, rh), k = e - s * hx;
      const long long ra = r0 + 2 * s, rb = ra + 1;
      C A = mk<C>((T)0, (T)0), B = A;
      if (ra < a.nrows) A = spec[ra * a.ld + k];
      if (rb < a.nrows) B = spec[rb * a.ld + k];
      t.cur[sp((k << lS) + s)] = mk<C>(A.x - B.y, -(A.y + B.x));
      if (k > 0 && 2 * k < n) t.cur[sp(((n - k) << lS) + s)] = mk<C>(A.x + B.y, A.y - B.x);
    }
    __syncthreads();
    dft_tile<T>(a.d, t);
    if (a.flags & GROW_STORE_REAL) {
      for (int e = tid; e < S * n; e += nth) {
        const int s = fdiv(e, rn), x = e - s * n;
        const long long ra = r0 + 2 * s, rb = ra + 1;
        const C v = t.cur[sp((x << lS) + s)];
        if (ra < a.nrows) out[ra * n + x] = v.x;
        if (rb < a.nrows) out[rb * n + x] = -v.y;
      }
      return;
    }
    for (int e = tid; e < S * n; e += nth) {  // the real rows a + i b, never stored
      const C v = t.cur[sp(e)];
      t.cur[sp(e)] = mk<C>(v.x, -v.y);
    }
  } else {
    for (int e = tid; e < S * n; e += nth) {
      const int s = fdiv(e, rn), x = e - s * n;
      const long long ra = r0 + 2 * s, rb = ra + 1;
      const T va = ra < a.nrows ? in[ra * n + x] : (T)0, vb = rb < a.nrows ? in[rb * n + x] : (T)0;
      t.cur[sp((x << lS) + s)] = mk<C>(va, vb);
    }
  }
  __syncthreads();
  dft_tile<T>(a.d, t);
  for (int e = tid; e < S * hx; e += nth) {
    const int s = fdiv(e, rh), k = e - s * hx;
    const long long ra = r0 + 2 * s, rb = ra + 1;
    const C Zk = t.cur[sp((k << lS) + s)], Zm = t.cur[sp(((k == 0 ? 0 : n - k) << lS) + s)];
    if (ra < a.nrows) spec[ra * a.ld + k] = mk<C>((T)0.5 * (Zk.x + Zm.x), (T)0.5 * (Zk.y - Zm.y));
    if (rb < a.nrows) spec[rb * a.ld + k] = mk<C>((T)0.5 * (Zk.y + Zm.y), (T)0.5 * (Zm.x - Zk.x));
  }
}

// ------------------------------------------------------------------ multipliers
struct GMul {
  int mult, nx, nb, ny;     // sizes along x, the batch axis of a box (0 in 2D), the column
  const double* sx;         // d^2 lambda along x, the batch axis and the column
  const double* sb;
  const double* sy;
  double ix, ib, iy;        // 1 / d^2 of each
  double kxs, kys;          // 2 pi / (n d) along x and the column (advection forms)
  double h, scale;
  double D[4], vx[4], vy[4];
};

// The multiplier of half-spectrum point (ky, kx) of field f (box: ky along z, kb along y),
// times the normalisation, as a complex number; FP64 throughout.
__device__ __forceinline__ double2 gmul_value(const GMul& m, int f, int ky, int kb, int kx) {
  double lam = m.sx[kx] * m.ix + m.sy[ky] * m.iy;
  if (m.nb) lam += m.sb[kb] * m.ib;
  const double zr = m.h * m.D[f] * lam;
  double fr, fi = 0.0;
  if (m.mult < MJX_MULT_ADV_SOLVE) {
    if (m.mult == MJX_MULT_HELMHOLTZ) {
      double den = 1.0 - zr;
      if (fabs(den) < 1e-14) den = 1e-14;
      fr = 1.0 / den;
    } else if (m.mult == MJX_MULT_CN) {
      fr = (1.0 + 0.5 * zr) / (1.0 - 0.5 * zr);
    } else if (m.mult == MJX_MULT_LAP) {
      fr = zr;
    } else if (m.mult == MJX_MULT_EXP) {
      fr = exp(zr);
    } else {
      fr = 1.0;
    }
    return make_double2(fr * m.scale, 0.0);
  }
  // z = h (D lam - i (vx kx + vy ky)) with fftfreq indices (the Nyquist index of an even
  // length negative), averaged with the conjugate at -k
  const int mx = kx < (m.nx + 1) / 2 ? kx : kx - m.nx, my = ky < (m.ny + 1) / 2 ? ky : ky - m.ny;
  double mre = 0.0, mim = 0.0;
#pragma unroll 1
  for (int side = 0; side < 2; ++side) {
    const int qx = side ? (2 * mx == -m.nx ? mx : -mx) : mx, qy = side ? (2 * my == -m.ny ? my : -my) : my;
    const double zi = -m.h * (m.vx[f] * m.kxs * qx + m.vy[f] * m.kys * qy);
    if (m.mult == MJX_MULT_ADV_SOLVE) {
      double dr = 1.0 - zr, di = -zi;
      if (sqrt(dr * dr + di * di) < 1e-14) { dr = 1e-14; di = 0.0; }
      const double den = dr * dr + di * di;
      fr = dr / den; fi = -di / den;
    } else if (m.mult == MJX_MULT_ADV_LAP) {
      fr = zr; fi = zi;
    } else if (m.mult == MJX_MULT_ADV_CN) {
      const double nr = 1.0 + 0.5 * zr, ni = 0.5 * zi, dr = 1.0 - 0.5 * zr, di = -0.5 * zi;
      const double den = dr * dr + di * di;
      fr = (nr * dr + ni * di) / den; fi = (ni * dr - nr * di) / den;
    } else {
      double sn, cs;
      sincos(zi, &sn, &cs);
      const double ez = exp(zr);
      fr = ez * cs; fi = ez * sn;
    }
    mre += 0.5 * fr;
    mim += side ? -0.5 * fi : 0.5 * fi;
  }
  return make_double2(mre * m.scale, mim * m.scale);
}

// ------------------------------------------------------------------ column pass
enum { GCOL_NONE = 0, GCOL_VALUE = 1, GCOL_TABLE = 2, GCOL_USER = 3 };

template <typename T>
struct GColArgs {
  Dft<T> d;
  cx<T>* spec;
  const T* tab;        // GCOL_TABLE: formed multipliers [batch][n][ld]; GCOL_USER: the caller's [ny][nx]
  long long bstride;   // complex elements between batch entries (fields or planes)
  int ld, ncols, hx;   // row stride, columns; columns with (col mod ldx) >= hx are padding
  int ldx;             // row length of a z-pass column index (ld in 2D)
  int lC, dirs, mode;
  GMul m;
};

// C = 2^lC columns per CTA; blockIdx.y is the batch entry.
template <typename T>
__global__ void __launch_bounds__(512) gcol_kernel(const __grid_constant__ GColArgs<T> a) {
  typedef cx<T> C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n = a.d.n, lC = a.lC, Cn = 1 << lC, tid = threadIdx.x, nth = blockDim.x;
  Tile<T> t = tile_begin<T>(a.d, smem_raw, lC);
  pdl_wait();
  const int c0 = blockIdx.x << lC, b = blockIdx.y;
  C* g = a.spec + (long long)b * a.bstride + c0;
  const bool inv_first = (a.dirs & 1) == 0;
  for (int e = tid; e < (n << lC); e += nth) {
    const int j = e >> lC, c = e & (Cn - 1);
    C v = c0 + c < a.ncols ? g[(long long)j * a.ld + c] : mk<C>((T)0, (T)0);
    if (inv_first) v.y = -v.y;
    t.cur[sp(e)] = v;
  }
  __syncthreads();
  dft_tile<T>(a.d, t);
  if (a.dirs == 3) {
    for (int e = tid; e < (n << lC); e += nth) {
      const int j = e >> lC, c = e & (Cn - 1), col = c0 + c;
      const C v = t.cur[sp(e)];
      T mr = (T)0, mi = (T)0;
      if (col < a.ncols) {
        if (a.mode == GCOL_TABLE) {
          mr = a.tab[((long long)b * n + j) * a.ld + col];
        } else {
          const int kb = a.m.nb ? col / a.ldx : 0, kx = col - kb * a.ldx;
          if (kx < a.hx) {
            if (a.mode == GCOL_USER) {  // the real kernel's Hermitian part
              const int jm = j == 0 ? 0 : n - j, xm = kx == 0 ? 0 : a.m.nx - kx;
              mr = (T)(0.5 * a.m.scale * ((double)a.tab[(long long)j * a.m.nx + kx] + (double)a.tab[(long long)jm * a.m.nx + xm]));
            } else {
              const double2 f = gmul_value(a.m, b, j, kb, kx);
              mr = (T)f.x; mi = (T)f.y;
            }
          }
        }
      }
      // conj(m v), for the inverse by conjugation
      t.cur[sp(e)] = mk<C>(v.x * mr - v.y * mi, -(v.x * mi + v.y * mr));
    }
    __syncthreads();
    dft_tile<T>(a.d, t);
  }
  const bool neg = (a.dirs & 2) != 0;
  for (int e = tid; e < (n << lC); e += nth) {
    const int j = e >> lC, c = e & (Cn - 1);
    C v = t.cur[sp(e)];
    if (neg) v.y = -v.y;
    if (c0 + c < a.ncols) g[(long long)j * a.ld + c] = v;
  }
}

// the formed multipliers of a real symbol, [batch][n][ld]
template <typename T>
__global__ void gtab_kernel(T* tab, const __grid_constant__ GMul m, int nf, int n, int ld, int ldx, int hx) {
  const long long per = (long long)n * ld, total = per * nf;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int f = (int)(i / per);
    const long long r = i - f * per;
    const int j = (int)(r / ld), col = (int)(r - (long long)j * ld);
    const int kb = m.nb ? col / ldx : 0, kx = col - kb * ldx;
    tab[i] = kx < hx ? (T)gmul_value(m, f, j, kb, kx).x : (T)0;
  }
}

// ------------------------------------------------------------------ launch geometry
// half-spectrum row length: whole 32-byte sectors, but unpadded below four points, where a pad
// would take the spectra beyond the workspace (general_ws) and a row beyond the tuner's scratch
static int gen_ld(int nx, int elem) {
  const int hx = nx / 2 + 1, q = 32 / (2 * elem);
  return nx < 4 ? hx : (hx + q - 1) / q * q;
}

// radices (at most 16 of them, each below 16) as tile_dft takes them
static unsigned long long pack_radices(int k, const int* rad) {
  unsigned long long r = 0;
  for (int i = 0; i < k; ++i) r |= (unsigned long long)rad[i] << (4 * i);
  return r;
}

template <typename T>
static Dft<T> dft_desc(const void* plan, int n) {
  const DftGeom g = dft_geom(n, sizeof(T));
  const char* p = (const char*)plan;
  Dft<T> d;
  memset(&d, 0, sizeof(d));
  d.tw = (const cx<T>*)(p + g.tw); d.chirp = (const cx<T>*)(p + g.chirp); d.bhat = (const cx<T>*)(p + g.bhat);
  d.n = n; d.L = g.L; d.bluestein = g.bluestein;
  if (g.mixed) {
    d.rad = pack_radices(g.nrad, g.rad);
    d.odd = g.nrad & 1;
    DftTune t;
    d.tps = (tune_dft_get(n, (int)sizeof(T), &t) && t.tpsm > 0) ? t.tpsm : n / 8;
  } else {
    d.log2L = g.log2L;
    d.tps = g.L / 8;
  }
  if (d.tps < 1) d.tps = 1;
  if (d.tps > 256) d.tps = 256;
  return d;
}

// nf fields of nrows rows.  The two rows of a pair are of one field: a pair of different fields
// would give each the rounding errors, infinities and NaN of the other (a field of order 1 in FP32
// behind one of order 1e6 was wrong in its second digit).  With an even number of rows the stack
// is one run of pairs; with an odd one each field's last row is alone in its pair.
template <typename T>
static cudaError_t grow(const Dft<T>& d0, const T* in, T* out, cx<T>* spec, long long nrows, int nf, int ld, int flags,
                        int pdl, cudaStream_t s) {
  if (nrows % 2 == 0) { nrows *= nf; nf = 1; }
  GRowArgs<T> a;
  memset(&a, 0, sizeof(a));
  a.d = d0; a.in = in; a.out = out; a.spec = spec; a.nrows = nrows; a.ld = ld; a.flags = flags;
  const long long pairs = (nrows + 1) / 2;
  a.lS = tile_log<T>(a.d, pairs * nf, 8);
  const long long grid = (pairs + (1 << a.lS) - 1) >> a.lS;
  return launch_chain(grow_kernel<T>, dim3((unsigned)grid, nf), tile_threads<T>(a.d, a.lS), tile_smem<T>(a.d, a.lS), s,
                      pdl, a);
}

template <typename T>
static cudaError_t gcol(GColArgs<T> a, int batch, cudaStream_t s) {
  // 4 FP32 or 2 FP64 columns fill a 32-byte sector of each row; twice that where the grid is large
  a.lC = tile_log<T>(a.d, (long long)a.ncols * batch, sizeof(T) == 4 ? 8 : 4);
  dim3 grid((a.ncols + (1 << a.lC) - 1) >> a.lC, batch);
  return launch_chain(gcol_kernel<T>, grid, tile_threads<T>(a.d, a.lC), tile_smem<T>(a.d, a.lC), s, 1, a);
}

static const double* plan_symbol(const void* plan, int n, int elem, int symbol) {
  const DftGeom g = dft_geom(n, elem);
  return (const double*)((const char*)plan + g.sym) + (symbol == MJX_SYMBOL_FD ? 0 : n);
}

static void symbol_axis(const void* plan, int n, int elem, int symbol, double d, const double** s, double* inv) {
  *s = plan_symbol(plan, n, elem, symbol);
  *inv = 1.0 / (d * d);
}

template <typename T>
static mjx_status general_apply(const void* plan_y, const void* plan_x, const mjx_grid2d* g, int symbol, int nf,
                                const double* D, const double* vx, const double* vy, double h, int mult,
                                const T* table, int n_steps, const T* in, T* out, void* ws, cudaStream_t s) {
  const int ny = g->ny, nx = g->nx, ld = gen_ld(nx, sizeof(T)), hx = nx / 2 + 1;
  const double twopi = 6.283185307179586476925286766559;
  cx<T>* spec = (cx<T>*)ws;
  T* tab = (T*)(spec + (size_t)nf * ny * ld);
  const Dft<T> dx = dft_desc<T>(plan_x, nx);
  GColArgs<T> c;
  memset(&c, 0, sizeof(c));
  c.d = dft_desc<T>(plan_y, ny);
  c.spec = spec; c.bstride = (long long)ny * ld; c.ld = c.ldx = ld; c.ncols = c.hx = hx; c.dirs = 3;
  GMul& m = c.m;
  m.mult = mult; m.nx = nx; m.nb = 0; m.ny = ny; m.h = h;
  symbol_axis(plan_x, nx, sizeof(T), symbol, g->dx, &m.sx, &m.ix);
  symbol_axis(plan_y, ny, sizeof(T), symbol, g->dy, &m.sy, &m.iy);
  m.kxs = twopi / (nx * g->dx);
  m.kys = twopi / (ny * g->dy);
  m.scale = 1.0 / ((double)nx * (double)ny);
  for (int f = 0; f < nf; ++f) {
    m.D[f] = D ? D[f] : 0.0;
    m.vx[f] = vx ? vx[f] : 0.0;
    m.vy[f] = vy ? vy[f] : 0.0;
  }
  c.mode = mult == MJX_MULT_TABLE ? GCOL_USER : GCOL_VALUE;
  c.tab = table;
  MJX_CUDA_TRY(grow<T>(dx, in, nullptr, spec, ny, nf, ld, GROW_STORE_SPEC, 0, s));
  if (n_steps > 1 && mult < MJX_MULT_ADV_SOLVE) {
    gtab_kernel<T><<<152 * 4, 256, 0, s>>>(tab, m, nf, ny, ld, ld, hx);
    MJX_CUDA_TRY(cudaGetLastError());
    c.mode = GCOL_TABLE;
    c.tab = tab;
  }
  for (int i = 0; i < n_steps; ++i) {
    MJX_CUDA_TRY(gcol<T>(c, nf, s));
    const bool last = i == n_steps - 1;
    MJX_CUDA_TRY(grow<T>(dx, nullptr, out, spec, ny, nf, ld,
                         GROW_LOAD_SPEC | (last ? GROW_STORE_REAL : GROW_STORE_SPEC), 1, s));
  }
  return MJX_OK;
}

// n_steps applications on [nz][ny][nx]
template <typename T>
static mjx_status general_apply3(const void* pz, const void* py, const void* px, const mjx_grid3d* g, int symbol,
                                 double D, double h, int mult, int n_steps, const T* in, T* out, void* ws,
                                 cudaStream_t s) {
  const int nz = g->nz, ny = g->ny, nx = g->nx, ld = gen_ld(nx, sizeof(T)), hx = nx / 2 + 1;
  cx<T>* spec = (cx<T>*)ws;
  T* tab = (T*)(spec + (size_t)nz * ny * ld);
  const Dft<T> dx = dft_desc<T>(px, nx);
  GColArgs<T> y;
  memset(&y, 0, sizeof(y));
  y.d = dft_desc<T>(py, ny);
  y.spec = spec; y.bstride = (long long)ny * ld; y.ld = y.ldx = ld; y.ncols = y.hx = hx;
  GColArgs<T> z = y, yb = y;
  y.dirs = 1;
  yb.dirs = 2;
  z.d = dft_desc<T>(pz, nz);
  z.bstride = 0; z.ld = z.ncols = ny * ld; z.dirs = 3; z.mode = GCOL_VALUE;
  GMul& m = z.m;
  m.mult = mult; m.nx = nx; m.nb = ny; m.ny = nz; m.h = h; m.D[0] = D;
  symbol_axis(px, nx, sizeof(T), symbol, g->dx, &m.sx, &m.ix);
  symbol_axis(py, ny, sizeof(T), symbol, g->dy, &m.sb, &m.ib);
  symbol_axis(pz, nz, sizeof(T), symbol, g->dz, &m.sy, &m.iy);
  m.scale = 1.0 / ((double)nx * (double)ny * (double)nz);
  if (n_steps > 1) {
    gtab_kernel<T><<<152 * 4, 256, 0, s>>>(tab, m, 1, nz, ny * ld, ld, hx);
    MJX_CUDA_TRY(cudaGetLastError());
    z.mode = GCOL_TABLE;
    z.tab = tab;
  }
  const long long rows = (long long)nz * ny;
  MJX_CUDA_TRY(grow<T>(dx, in, nullptr, spec, rows, 1, ld, GROW_STORE_SPEC, 0, s));
  for (int i = 0; i < n_steps; ++i) {
    MJX_CUDA_TRY(gcol<T>(y, nz, s));
    MJX_CUDA_TRY(gcol<T>(z, 1, s));
    MJX_CUDA_TRY(gcol<T>(yb, nz, s));
    const bool last = i == n_steps - 1;
    MJX_CUDA_TRY(grow<T>(dx, nullptr, out, spec, rows, 1, ld,
                         GROW_LOAD_SPEC | (last ? GROW_STORE_REAL : GROW_STORE_SPEC), 1, s));
  }
  return MJX_OK;
}

// workspace: the half spectra (2 gen_ld reals a row) and the formed multipliers (gen_ld), within the
// four reals a point that the query asks for: 3 gen_ld <= 4 nx for every nx
static size_t general_ws(size_t rows, int nx, int elem) { return rows * nx * 4 * elem; }

static mjx_status set_dft_attrs() {
  static ContextOnce once;
  return once.run([]() -> mjx_status {
    int dev = 0, optin = 0;
    MJX_CUDA_TRY(cudaGetDevice(&dev));
    MJX_CUDA_TRY(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    MJX_CUDA_TRY(cudaFuncSetAttribute(grow_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin));
    MJX_CUDA_TRY(cudaFuncSetAttribute(grow_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin));
    MJX_CUDA_TRY(cudaFuncSetAttribute(gcol_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin));
    MJX_CUDA_TRY(cudaFuncSetAttribute(gcol_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin));
    return MJX_OK;
  });
}

}  // namespace mjx

using namespace mjx;

extern "C" {

size_t mjx_dftn_plan_bytes(int n, int dtype) {
  const int e = elem_size(dtype);
  if (!e || !dft_len_ok(n)) return 0;
  return dft_geom(n, e).total;
}

mjx_status mjx_dftn_plan_init(void* plan, int n, int dtype, void* stream) {
  const int e = elem_size(dtype);
  if (!e) return MJX_BAD_DTYPE;
  if (!plan || !dft_len_ok(n)) return MJX_BAD_ARG;
  const DftGeom g = dft_geom(n, e);
  std::vector<unsigned char> host(g.total, 0);
  auto put = [&](size_t off, int i, double re, double im) {
    if (e == 4) { float* q = (float*)(host.data() + off); q[2 * i] = (float)re; q[2 * i + 1] = (float)im; }
    else { double* q = (double*)(host.data() + off); q[2 * i] = re; q[2 * i + 1] = im; }
  };
  const double twopi = 6.283185307179586476925286766559;
  const Roots roots(g.L);  // L = n unless Bluestein
  for (int j = 0; j < g.L; ++j) {
    double re, im;
    tile_twiddle(roots, j, e, &re, &im);
    put(g.tw, j, re, im);
  }
  if (g.bluestein) {
    std::vector<double> chirp, bhat;
    bluestein_tables(n, roots, e == 8, &chirp, &bhat);
    for (int j = 0; j < n; ++j) put(g.chirp, j, chirp[2 * j], chirp[2 * j + 1]);
    for (int j = 0; j < g.L; ++j) put(g.bhat, j, bhat[2 * j], bhat[2 * j + 1]);
  }
  double* sym = (double*)(host.data() + g.sym);
  for (int j = 0; j < n; ++j) {
    const int m = j < (n + 1) / 2 ? j : j - n;  // fftfreq index
    sym[j] = 2.0 * cos(twopi * j / n) - 2.0;
    sym[n + j] = -(twopi * m / n) * (twopi * m / n);
  }
  cudaStream_t s = (cudaStream_t)stream;
  MJX_CUDA_TRY(cudaMemcpyAsync(plan, host.data(), g.total, cudaMemcpyHostToDevice, s));
  MJX_CUDA_TRY(cudaStreamSynchronize(s));
  return MJX_OK;
}

size_t mjx_spectral_general2d_ws_bytes(int ny, int nx, int nfields, int dtype) {
  const int e = elem_size(dtype);
  if (!e || !dft_len_ok(ny) || !dft_len_ok(nx) || nfields < 1 || nfields > 4) return 0;
  return general_ws((size_t)nfields * ny, nx, e);
}

static mjx_status general2d(const void* plan_y, const void* plan_x, const mjx_grid2d* g, int symbol, int dtype,
                            int nfields, const double* D, const double* vx, const double* vy, double h, int mult,
                            const void* table, int n_steps, const void* in, void* out, void* ws, size_t ws_bytes,
                            void* stream) {
  const int e = elem_size(dtype);
  if (!e) return MJX_BAD_DTYPE;
  if (!g || !plan_y || !plan_x || !in || !out || nfields < 1 || nfields > 4) return MJX_BAD_ARG;
  if (!dft_len_ok(g->ny) || !dft_len_ok(g->nx)) return MJX_BAD_SHAPE;
  if (!(g->dx > 0) || !(g->dy > 0)) return MJX_BAD_ARG;
  if (symbol != MJX_SYMBOL_FD && symbol != MJX_SYMBOL_SPECTRAL) return MJX_BAD_ARG;
  const bool ok_mult = mult == MJX_MULT_SCALE || mult == MJX_MULT_HELMHOLTZ || mult == MJX_MULT_CN ||
                       mult == MJX_MULT_EXP || mult == MJX_MULT_LAP || mult == MJX_MULT_TABLE ||
                       mult == MJX_MULT_ADV_SOLVE || mult == MJX_MULT_ADV_LAP || mult == MJX_MULT_ADV_EXP ||
                       mult == MJX_MULT_ADV_CN;
  if (!ok_mult || (mult == MJX_MULT_TABLE && !table)) return MJX_BAD_ARG;
  if (!ws || ws_bytes < mjx_spectral_general2d_ws_bytes(g->ny, g->nx, nfields, dtype)) return MJX_WORKSPACE;
  MJX_TRY(set_dft_attrs());
  cudaStream_t s = (cudaStream_t)stream;
  if (e == 4)
    return general_apply<float>(plan_y, plan_x, g, symbol, nfields, D, vx, vy, h, mult, (const float*)table,
                                n_steps, (const float*)in, (float*)out, ws, s);
  return general_apply<double>(plan_y, plan_x, g, symbol, nfields, D, vx, vy, h, mult, (const double*)table,
                               n_steps, (const double*)in, (double*)out, ws, s);
}

mjx_status mjx_spectral_apply_general2d(const void* plan_y, const void* plan_x, const mjx_grid2d* g, int symbol,
                                        int dtype, int nfields, const double* D, const double* vx,
                                        const double* vy, double h, int mult, const void* table,
                                        const void* in, void* out, void* ws, size_t ws_bytes, void* stream) {
  return general2d(plan_y, plan_x, g, symbol, dtype, nfields, D, vx, vy, h, mult, table, 1, in, out, ws, ws_bytes,
                   stream);
}

mjx_status mjx_spectral_steps_general2d(const void* plan_y, const void* plan_x, const mjx_grid2d* g, int symbol,
                                        int dtype, int nfields, const double* D, double h, int mult, int n_steps,
                                        const void* in, void* out, void* ws, size_t ws_bytes, void* stream) {
  if (!D || n_steps < 1) return MJX_BAD_ARG;
  if (mult != MJX_MULT_SCALE && mult != MJX_MULT_HELMHOLTZ && mult != MJX_MULT_CN && mult != MJX_MULT_EXP &&
      mult != MJX_MULT_LAP)
    return MJX_BAD_ARG;
  return general2d(plan_y, plan_x, g, symbol, dtype, nfields, D, nullptr, nullptr, h, mult, nullptr, n_steps, in, out,
                   ws, ws_bytes, stream);
}

size_t mjx_spectral_general3d_ws_bytes(int nz, int ny, int nx, int dtype) {
  const int e = elem_size(dtype);
  if (!e || !dft_len_ok(nz) || !dft_len_ok(ny) || !dft_len_ok(nx)) return 0;
  return general_ws((size_t)nz * ny, nx, e);
}

mjx_status mjx_spectral_apply_general3d(const void* plan_z, const void* plan_y, const void* plan_x,
                                        const mjx_grid3d* g, int symbol, int dtype, double D, double h, int mult,
                                        int n_steps, const void* in, void* out, void* ws, size_t ws_bytes,
                                        void* stream) {
  const int e = elem_size(dtype);
  if (!e) return MJX_BAD_DTYPE;
  if (!g || !plan_z || !plan_y || !plan_x || !in || !out || n_steps < 1) return MJX_BAD_ARG;
  if (!dft_len_ok(g->nz) || !dft_len_ok(g->ny) || !dft_len_ok(g->nx)) return MJX_BAD_SHAPE;
  if (!(g->dx > 0) || !(g->dy > 0) || !(g->dz > 0)) return MJX_BAD_ARG;
  if (symbol != MJX_SYMBOL_FD && symbol != MJX_SYMBOL_SPECTRAL) return MJX_BAD_ARG;
  if (mult != MJX_MULT_SCALE && mult != MJX_MULT_HELMHOLTZ && mult != MJX_MULT_CN && mult != MJX_MULT_EXP &&
      mult != MJX_MULT_LAP)
    return MJX_BAD_ARG;
  if (!ws || ws_bytes < mjx_spectral_general3d_ws_bytes(g->nz, g->ny, g->nx, dtype)) return MJX_WORKSPACE;
  MJX_TRY(set_dft_attrs());
  cudaStream_t s = (cudaStream_t)stream;
  if (e == 4)
    return general_apply3<float>(plan_z, plan_y, plan_x, g, symbol, D, h, mult, n_steps, (const float*)in,
                                 (float*)out, ws, s);
  return general_apply3<double>(plan_z, plan_y, plan_x, g, symbol, D, h, mult, n_steps, (const double*)in,
                                (double*)out, ws, s);
}

}  // extern "C"

// Autotuner of the mixed-radix DFT of length n: every candidate schedule (dft_schedules) with
// threads per sequence n/4, n/8 and n/16 is timed in the spectrum-to-spectrum row pass (an
// inverse and a forward DFT of every row pair) on nrows rows of scratch (one warm-up launch,
// then reps launches between CUDA events); the fastest is installed in the registry for n and
// this element size.
template <typename T>
static mjx_status tune_dft(const void* plan, int n, long long nrows, cx<T>* data, int reps, double* times,
                           int max_times, int* n_cand, int* best, cudaStream_t s) {
  int sched[64 * 17];
  const int ns = dft_schedules(n, sched, 64);
  if (ns == 0) return MJX_BAD_ARG;
  int tps[3] = {n / 4, n / 8, n / 16}, ntp = 0;
  int uniq[3];
  for (int i = 0; i < 3; ++i) {
    int v = tps[i] < 1 ? 1 : (tps[i] > 256 ? 256 : tps[i]);
    bool dup = false;
    for (int j = 0; j < ntp; ++j) dup |= uniq[j] == v;
    if (!dup) uniq[ntp++] = v;
  }
  tune_dft_clear(n, (int)sizeof(T));
  Dft<T> d = dft_desc<T>(plan, n);
  const int ld = gen_ld(n, sizeof(T));
  cudaEvent_t e0, e1;
  MJX_CUDA_TRY(cudaEventCreate(&e0));
  MJX_CUDA_TRY(cudaEventCreate(&e1));
  double best_t = 1e300;
  int best_i = -1, k = 0;
  mjx_status st = MJX_OK;
  for (int i = 0; i < ns && st == MJX_OK; ++i) {
    for (int j = 0; j < ntp && st == MJX_OK; ++j, ++k) {
      d.rad = pack_radices(sched[17 * i], sched + 17 * i + 1);
      d.odd = sched[17 * i] & 1;
      d.tps = uniq[j];
      auto pass = [&]() {
        return grow<T>(d, nullptr, nullptr, data, nrows, 1, ld, GROW_LOAD_SPEC | GROW_STORE_SPEC, 0, s);
      };
      cudaError_t ce = pass();
      if (ce == cudaSuccess) ce = cudaEventRecord(e0, s);
      for (int r = 0; r < reps && ce == cudaSuccess; ++r) ce = pass();
      if (ce == cudaSuccess) ce = cudaEventRecord(e1, s);
      if (ce == cudaSuccess) ce = cudaEventSynchronize(e1);
      float ms = 0.f;
      if (ce == cudaSuccess) ce = cudaEventElapsedTime(&ms, e0, e1);
      if (ce != cudaSuccess) { set_last_error(ce, __FILE__, __LINE__); st = MJX_CUDA_ERROR; break; }
      const double tpl = (double)ms / reps;
      if (times && k < max_times) times[k] = tpl;
      if (tpl < best_t) { best_t = tpl; best_i = k; }
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (st != MJX_OK) return st;
  const int bi = best_i / ntp, bj = best_i - bi * ntp;
  DftTune t;
  memset(&t, 0, sizeof(t));
  t.nrad = sched[17 * bi];
  for (int q = 0; q < 16; ++q) t.rad[q] = sched[17 * bi + 1 + q];
  t.tpsm = uniq[bj];
  tune_dft_put(n, (int)sizeof(T), t);
  if (n_cand) *n_cand = ns * ntp;
  if (best) *best = best_i;
  return MJX_OK;
}

mjx_status mjx_autotune_dft(const void* plan, int n, int dtype, long long nrows, void* scratch,
                            size_t scratch_bytes, int reps, double* times, int max_times, int* n_cand,
                            int* best, void* stream) {
  const int e = elem_size(dtype);
  if (!e) return MJX_BAD_DTYPE;
  if (!plan || !scratch || !dft_len_ok(n) || nrows < 1 || reps < 1) return MJX_BAD_ARG;
  if (scratch_bytes < (size_t)nrows * n * 2 * e) return MJX_WORKSPACE;
  const DftGeom g = dft_geom(n, e);
  if (!g.mixed) {
    if (n_cand) *n_cand = 0;  // powers of two and Bluestein lengths have no schedule to tune
    if (best) *best = -1;
    return MJX_OK;
  }
  MJX_TRY(set_dft_attrs());
  cudaStream_t s = (cudaStream_t)stream;
  MJX_CUDA_TRY(cudaMemsetAsync(scratch, 0, (size_t)nrows * n * 2 * e, s));
  if (e == 4)
    return tune_dft<float>(plan, n, nrows, (cx<float>*)scratch, reps, times, max_times, n_cand, best, s);
  return tune_dft<double>(plan, n, nrows, (cx<double>*)scratch, reps, times, max_times, n_cand, best, s);
}

mjx_status mjx_dft_schedule_get(int n, int dtype, int* nrad, int* rad, int* tpsm) {
  const int e = elem_size(dtype);
  if (!e) return MJX_BAD_DTYPE;
  if (!nrad || !rad || !tpsm || !dft_len_ok(n)) return MJX_BAD_ARG;
  const DftGeom g = dft_geom(n, e);
  *nrad = g.mixed ? g.nrad : 0;
  for (int i = 0; i < 16; ++i) rad[i] = g.mixed ? g.rad[i] : 0;
  DftTune t;
  *tpsm = g.mixed ? ((tune_dft_get(n, e, &t) && t.tpsm > 0) ? t.tpsm : (n / 8 < 1 ? 1 : (n / 8 > 256 ? 256 : n / 8))) : 0;
  return MJX_OK;
}
