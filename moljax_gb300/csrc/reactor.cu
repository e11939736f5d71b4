// Batched 1D tubular-reactor Crank-Nicolson: one CTA per instance, the whole
// time loop of an instance in shared memory.
//
// Model c_t = (1/Pe) c_zz - c_z - Da c in two reference discretisations:
//  MJX_REACTOR_DANCKWERTS  benchmarks/benchmark_reactor_vs_diffrax.py:40-138:
//    N cells, dz = 1/N, diffusion implicit (CN), upwind advection and
//    reaction explicit, Danckwerts inlet flux -(c0 - 1)/dz, outlet Neumann row.
//  MJX_REACTOR_DIRICHLET   benchmarks/benchmark_method_comparison.py:56-160:
//    N nodes, dz = 1/(N-1), fully implicit CN of L = D2/Pe - D1 - Da with a
//    Dirichlet inlet row and the one-sided outlet row.
//  MJX_REACTOR_DANCKWERTS_CN  the Danckwerts discretisation above, advanced by
//    the fully implicit CN of benchmark_method_comparison.py:134-160: the whole
//    operator M c + s (dispersion, upwind advection with the inlet flux, and
//    reaction; s = e_0/dz) is implicit, so the step is stable at the CN step
//    size of that benchmark, dt = min(10 dz, 0.05, t_final/100) (line 216),
//    which the semi-implicit form above is not (its explicit upwind advection
//    needs dt <= dz).
//  MJX_REACTOR_RK4_DANCKWERTS / _ROBIN / _NEUMANN  benchmarks/benchmark_tubular_reactor.py:
//    N nodes, dz = 1/(N-1), explicit RK4 with penalty end rows (reactor_rk4_kernel).
// The reference solves with a dense inverse / LU (O(N^2) per step); the system
// matrix is tridiagonal and constant in time, so each CTA factorises it once
// (Thomas) and runs every step's two substitution sweeps as parallel affine
// scans over the CTA (x_i = alpha_i x_{i-1} + beta_i composes associatively).
#include <math.h>
#include <string.h>

#include "common.cuh"

namespace mjx {

int elem_size(int dtype);
void set_last_error(cudaError_t e, const char* file, int line);

struct ReactorArgs {
  const mjx_reactor_instance* inst;
  void* out;          // concatenated states, instance i at inst[i].offset
  int n_inst;
};

// shared-memory index with one pad word per 16: the scans give each thread a
// contiguous chunk (stride = chunk length), which would otherwise hit one bank
__device__ __forceinline__ int pz(int i) { return i + (i >> 4); }
__host__ __device__ __forceinline__ int pz_size(int n) { return n + (n >> 4) + 1; }

// affine map y -> a y + b, composition "first p then q"
template <typename T> struct Aff { T a, b; };
template <typename T> __device__ __forceinline__ Aff<T> comp(Aff<T> p, Aff<T> q) {
  Aff<T> r; r.a = q.a * p.a; r.b = q.a * p.b + q.b; return r;
}

// Inclusive scan of x_i = al[i] x_{i-1} + be[i] (x_{-1} = 0) over n elements in
// smem, processed in order ord(i) (forward, or reverse when REV).  Result in be[].
template <typename T, bool REV>
__device__ void affine_scan(T* al, T* be, int n, Aff<T>* wsum) {
  const int tid = threadIdx.x, nt = blockDim.x;
  const int per = (n + nt - 1) / nt;
  const int lo = tid * per, hi = min(n, lo + per);
  auto idx = [&](int i) { return pz(REV ? n - 1 - i : i); };
  Aff<T> acc; acc.a = (T)1; acc.b = (T)0;
  for (int i = lo; i < hi; ++i) {
    Aff<T> e; e.a = al[idx(i)]; e.b = be[idx(i)];
    acc = comp(acc, e);
  }
  // warp inclusive scan of the thread aggregates
  const int lane = tid & 31, w = tid >> 5;
  Aff<T> inc = acc;
  for (int o = 1; o < 32; o <<= 1) {
    Aff<T> up;
    up.a = __shfl_up_sync(0xffffffffu, inc.a, o);
    up.b = __shfl_up_sync(0xffffffffu, inc.b, o);
    if (lane >= o) inc = comp(up, inc);
  }
  if (lane == 31) wsum[w] = inc;
  __syncthreads();
  if (tid == 0) {  // scan of the warp totals (<= 32 warps)
    Aff<T> run; run.a = (T)1; run.b = (T)0;
    for (int q = 0; q < (nt >> 5); ++q) { run = comp(run, wsum[q]); wsum[q] = run; }
  }
  __syncthreads();
  // exclusive prefix for this thread
  Aff<T> ex;
  Aff<T> up;
  up.a = __shfl_up_sync(0xffffffffu, inc.a, 1);
  up.b = __shfl_up_sync(0xffffffffu, inc.b, 1);
  if (lane == 0) { ex.a = (T)1; ex.b = (T)0; } else { ex = up; }
  if (w > 0) ex = comp(wsum[w - 1], ex);
  T y = ex.b;  // value x_{lo-1} (the composite applied to x_{-1} = 0)
  __syncthreads();
  for (int i = lo; i < hi; ++i) {
    y = al[idx(i)] * y + be[idx(i)];
    be[idx(i)] = y;
  }
  __syncthreads();
}

// ------------------------------------------------------------------ n <= 4096: state in registers
// One instance per CTA of 256 threads, P = ceil(n / 256) <= 16 contiguous nodes per thread.
// The time loop is serial, so a step's latency is the run time.  The recurrence coefficients do
// not change with time, so every product of them that the affine scan needs (per thread, per
// shuffle level, per warp) is formed once before the loop and a step scans only the additive
// parts: P dependent FMAs, five shuffles, the totals of the preceding warps, P FMAs.  The
// composition order is that of affine_scan, so the values are the same.  The two sweeps cut the
// nodes into chunks from opposite ends, so the intermediate values and the new state cross
// through one padded shared-memory row (one pad word per chunk of even length: neighbouring
// threads then start on different banks).  P is a template argument: the chunk loops have no
// branches and constant offsets, without which a step takes twice as long.
// Measured at n = 4096: FP32 4.5 us -> 0.9-1.2 us a step, factorisation 2.1 ms -> 0.1-0.27 ms;
// 48 instances of 64..4096 nodes 16.0 -> 2.15 ms; FP64, 16 instances, 36.6 -> 19.5 ms.
// What bounds it: the dependent chains of one CTA (FP32), FP64 issue of one SM (FP64, nine
// operations a node and step at 1.7 lanes a clock).
enum { RMAXP = 16 };

// a product that no neighbouring addition is contracted with (the shared-memory form rounds it)
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }

// b of x_k = a_k x_{k-1} + b_k composed over the preceding threads (affine_scan's order)
template <typename T>
__device__ __forceinline__ T scan_carry(T acc, const T (&la)[5], T ea, const Aff<T>* wt, int lane, int w) {
#pragma unroll
  for (int l = 0; l < 5; ++l) {
    const T up = __shfl_up_sync(0xffffffffu, acc, 1 << l);
    if (lane >= (1 << l)) acc = fma(la[l], up, acc);
  }
  T ex = __shfl_up_sync(0xffffffffu, acc, 1);
  if (lane == 0) ex = (T)0;
  if (lane == 31) const_cast<Aff<T>*>(wt)[w].b = acc;
  __syncthreads();
  T run = (T)0;
#pragma unroll
  for (int q = 0; q < 7; ++q) {
    const Aff<T> t = wt[q];
    if (q < w) run = fma(t.a, run, t.b);
  }
  return w > 0 ? fma(ea, run, ex) : ex;
}

// the time-invariant factors of scan_carry for one sweep: per shuffle level, the exclusive
// product of the warp's preceding threads, and the warp totals' factors in wt
template <typename T>
__device__ __forceinline__ void scan_factors(T prod, T (&la)[5], T& ea, Aff<T>* wt, int lane, int w) {
  T a = prod;
#pragma unroll
  for (int l = 0; l < 5; ++l) {
    la[l] = a;
    const T up = __shfl_up_sync(0xffffffffu, a, 1 << l);
    if (lane >= (1 << l)) a = a * up;
  }
  ea = __shfl_up_sync(0xffffffffu, a, 1);
  if (lane == 0) ea = (T)1;
  if (lane == 31) wt[w].a = a;
}

// The roundings are those of reactor_kernel: its contraction of Ls c_{i-1} + Ld c_i + Lp c_{i+1}
// is written out, since the last digits of a long FP32 run follow it.
template <typename T, int P>
__device__ void reactor_steps(const mjx_reactor_instance& I, T* row, const double* piv, Aff<T>* wt,
                              const double* tri, T* out) {
  const int n = I.n, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const bool dk = I.variant == MJX_REACTOR_DANCKWERTS, dkcn = I.variant == MJX_REACTOR_DANCKWERTS_CN;
  constexpr int pad = (P & 1) ? 0 : 1;
  const int lo = tid * P;                         // forward chunk: nodes lo .. lo + nf - 1
  const int hi = n - 1 - lo;                      // backward chunk: nodes hi .. hi - nb + 1
  const int nf = max(0, min(P, n - lo)), nb = max(0, min(P, hi + 1));
  const int fph = lo + pad * tid;                 // row index of node lo
  const int bq = hi >= 0 ? hi / P : 1, bph = hi >= 0 ? hi + pad * bq : P, brem = (n - 1) % P;
  // tri: sub, dia, sup of the interior rows, sub and dia of the last, sup of row 0.  Places
  // beyond a chunk's nodes get the identity (factor 1, value 0), so that the loops below run
  // without branches; their row reads stay inside the row's slack and are not used.
  T al[P], mi[P], ng[P];
  T pf = (T)1, pb = (T)1;
#pragma unroll
  for (int k = 0; k < P; ++k) {
    const int i = lo + k;
    al[k] = (T)1; mi[k] = (T)0;
    if (k < nf) {
      const double m = piv[i];
      const double sub = i == 0 ? (dk ? tri[0] : 0.0) : (i == n - 1 ? tri[3] : tri[0]);
      mi[k] = (T)m;
      al[k] = (T)(-sub * m);
    }
    pf = al[k] * pf;
    const int j = hi - k;
    ng[k] = (T)1;
    if (k < nb) {
      const double sup = j == n - 1 ? 0.0 : (j == 0 ? tri[5] : tri[2]);
      ng[k] = -(T)(sup * piv[j]);
    }
    pb = ng[k] * pb;
  }
  Aff<T>* wf = wt;
  Aff<T>* wb = wt + 8;
  T laf[5], lab[5], eaf, eab;
  scan_factors<T>(pf, laf, eaf, wf, lane, w);
  scan_factors<T>(pb, lab, eab, wb, lane, w);
  // rhs coefficients: r = c + dt/2 (Ls c_{i-1} + Ld c_i + Lp c_{i+1}) and the source of row 0
  const double* L = tri + 6;
  const T Ls = (T)L[0], Ld = (T)L[1], Lp = (T)L[2], Lsl = (T)L[3], Ldl = (T)L[4];
  const T idz = (T)L[5], kp = (T)L[6], Dat = (T)I.Da, dtt = (T)I.dt, half_dt = (T)(0.5 * I.dt);
  const T cin = (T)I.c_inlet;
#pragma unroll
  for (int k = 0; k < P; ++k)
    if (k < nf) row[fph + k] = (!dk && !dkcn && lo + k == 0) ? cin : (T)I.c_init;
  __syncthreads();
  // Warps whose chunks are whole and hold no end row take loops without masks; the other one or
  // two compute the same loops and then put in the end rows' values and the zeros beyond.
  const bool full = __all_sync(0xffffffffu, lo + P <= n);
  const bool inner = full && __all_sync(0xffffffffu, lo > 0 && lo + P < n);
  const int kl = n - 1 - lo;  // the chunk place of the last node, if it is here
  T d[P];
  for (int step = 0; step < I.n_steps; ++step) {
    T cv[P + 2];  // c at nodes lo - 1 .. lo + P
    cv[0] = row[max(fph - 1 - pad, 0)];
#pragma unroll
    for (int k = 0; k <= P; ++k) cv[k + 1] = row[fph + k + (k >= P ? pad : 0)];
    if (dk) {
      if (lo == 0) cv[0] = (T)0;
#pragma unroll
      for (int k = 0; k < P; ++k) {
        const T cl = cv[k], ci = cv[k + 1], cr = cv[k + 2];
        const T lap = k == kl ? (T)2 * cl - (T)2 * ci : cl - (T)2 * ci + cr;
        const T adv = k == 0 && lo == 0 ? -(ci - (T)1) * idz : -(ci - cl) * idz;
        const T r = ci + kp * lap + dtt * (adv - Dat * ci);
        d[k] = k < nf ? mul_rn(r, mi[k]) : (T)0;
      }
    } else {
      T d0 = (T)0, dl = (T)0;
      if (!inner) {  // rows 0 and n - 1
        const T c1 = n > 1 ? cv[2] : (T)0;  // one node has no right-hand neighbour
        const T r0 = fma(half_dt, fma(Ld, cv[1], mul_rn(Lp, c1)), cv[1]);
        d0 = mul_rn(dkcn ? r0 + mul_rn(dtt, idz) : cin, mi[0]);
        const int last = n - 1 + pad * ((n - 1) / P), prev = n - 2 + pad * ((n - 2) / P);
        const T cn = row[last], cm = row[max(prev, 0)];
        dl = fma(half_dt, fma(Ldl, cn, mul_rn(Lsl, cm)), cn);
      }
#pragma unroll
      for (int k = 0; k < P; ++k) {
        const T Mc = fma(Lp, cv[k + 2], fma(Ld, cv[k + 1], mul_rn(Ls, cv[k])));
        d[k] = mul_rn(fma(half_dt, Mc, cv[k + 1]), mi[k]);
      }
      if (!inner) {
#pragma unroll
        for (int k = 0; k < P; ++k) {
          if (k >= kl) d[k] = k == kl ? mul_rn(dl, mi[k]) : (T)0;
        }
        if (lo == 0) d[0] = d0;
      }
    }
    T acc = (T)0;
#pragma unroll
    for (int k = 0; k < P; ++k) acc = fma(al[k], acc, d[k]);
    T y = scan_carry<T>(acc, laf, eaf, wf, lane, w);  // its barrier also ends the reads of the row
    if (full) {
#pragma unroll
      for (int k = 0; k < P; ++k) {
        y = fma(al[k], y, d[k]);
        row[fph + k] = y;
      }
    } else {
#pragma unroll
      for (int k = 0; k < P; ++k) {
        y = fma(al[k], y, d[k]);
        row[k < nf ? fph + k : -RMAXP - 2] = y;  // the slack's first word takes what is beyond
      }
    }
    __syncthreads();
    acc = (T)0;
#pragma unroll
    for (int k = 0; k < P; ++k) d[k] = row[bph - k - (k > brem ? pad : 0)];
    if (!full) {
#pragma unroll
      for (int k = 0; k < P; ++k)
        if (k >= nb) d[k] = (T)0;
    }
#pragma unroll
    for (int k = 0; k < P; ++k) acc = fma(ng[k], acc, d[k]);
    y = scan_carry<T>(acc, lab, eab, wb, lane, w);
    if (full) {
#pragma unroll
      for (int k = 0; k < P; ++k) {
        y = fma(ng[k], y, d[k]);
        row[bph - k - (k > brem ? pad : 0)] = y;
      }
    } else {
#pragma unroll
      for (int k = 0; k < P; ++k) {
        y = fma(ng[k], y, d[k]);
        row[k < nb ? bph - k - (k > brem ? pad : 0) : -RMAXP - 2] = y;
      }
    }
    __syncthreads();
  }
  for (int i = tid; i < n; i += blockDim.x) out[i] = row[i + pad * (i / P)];
}

// Tridiagonal entries of the implicit matrix (tri[0..5]: sub, dia, sup of the interior rows,
// sub and dia of the last row, sup of row 0; the returned dia0) and of the explicit operator
// (tri[6..]: Ls, Ld, Lp, Lsl, Ldl, 1/dz, kappa), as reactor_kernel builds them.
__device__ __forceinline__ double reactor_entries(const mjx_reactor_instance& I, double* tri) {
  const int n = I.n;
  const double Pe = I.Pe, Da = I.Da, dt = I.dt;
  const bool dk = I.variant == MJX_REACTOR_DANCKWERTS, dkcn = I.variant == MJX_REACTOR_DANCKWERTS_CN;
  const double dz = (dk || dkcn) ? 1.0 / n : 1.0 / (n - 1);
  const double q = (1.0 / Pe) / (dz * dz);
  const double kap = 0.5 * dt / (Pe * dz * dz);
  const double Ls = q + 1.0 / dz, Ld = -2.0 * q - 1.0 / dz - Da, Lp = q;
  const double Lsl = dkcn ? 2.0 * q + 1.0 / dz : q, Ldl = dkcn ? Ld : -q - 1.0 / dz - Da;
  tri[0] = dk ? -kap : -0.5 * dt * Ls;
  tri[1] = dk ? 1.0 + 2.0 * kap : 1.0 - 0.5 * dt * Ld;
  tri[2] = dk ? -kap : -0.5 * dt * Lp;
  tri[3] = dk ? -2.0 * kap : -0.5 * dt * Lsl;
  tri[4] = dk ? 1.0 + 2.0 * kap : 1.0 - 0.5 * dt * Ldl;
  tri[5] = (dk || dkcn) ? tri[2] : 0.0;
  tri[6] = Ls; tri[7] = Ld; tri[8] = Lp; tri[9] = Lsl; tri[10] = Ldl; tri[11] = 1.0 / dz; tri[12] = kap;
  return (dk || dkcn) ? tri[1] : 1.0;
}

template <typename T>
__global__ void __launch_bounds__(256) reactor_reg_kernel(ReactorArgs A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double tri[13];
  __shared__ Aff<T> wt[16];
  __shared__ int filled;
  const mjx_reactor_instance I = A.inst[blockIdx.x];
  const int n = I.n, tid = threadIdx.x;
  T* out = reinterpret_cast<T*>(A.out) + I.offset;
  if (n > 256 * RMAXP) return;  // reactor_kernel's
  if (I.variant < MJX_REACTOR_DANCKWERTS || I.variant > MJX_REACTOR_DANCKWERTS_CN) {  // an RK4 instance
    for (int i = tid; i < n; i += blockDim.x) out[i] = (T)NAN;
    return;
  }
  const int per = (n + 255) / 256;
  double* piv = reinterpret_cast<double*>(smem_raw);  // pivots 1/(b_i - a_i c'_{i-1})
  T* row = reinterpret_cast<T*>(piv + n) + RMAXP + 2;  // slack on both sides
  // Thomas factorisation, sequential in FP64 (each dependent FP64 instruction takes ~64
  // cycles): the interior rows are equal, so once a pivot repeats exactly all later ones do;
  // near that point the reciprocal is two Newton steps from the last pivot.
  if (tid == 0) {
    const double dia0 = reactor_entries(I, tri);
    const double sub = tri[0], dia = tri[1], sup = tri[2];
    double m = 1.0 / dia0;
    double c = (n > 1 ? tri[5] : 0.0) * m;
    piv[0] = m;
    int i = 1;
    for (; i < n - 1; ++i) {
      const double x = dia - sub * c;
      const double last = m;
      const double e = 1.0 - x * m;
      if (fabs(e) < 1e-4) {
        m = m + m * e;
        m = m + m * (1.0 - x * m);
      } else {
        m = 1.0 / x;
      }
      c = sup * m;
      piv[i] = m;
      if (m == last && i > 1) { ++i; break; }
    }
    filled = i;
    if (n > 1) piv[n - 1] = 1.0 / (tri[4] - tri[3] * c);
  }
  __syncthreads();
  const double mlast = piv[filled - 1];
  for (int i = filled + tid; i < n - 1; i += blockDim.x) piv[i] = mlast;
  __syncthreads();
#define MJX_RSTEPS(PP) \
  case PP: reactor_steps<T, PP>(I, row, piv, wt, tri, out); break;
  switch (per) {
    MJX_RSTEPS(1) MJX_RSTEPS(2) MJX_RSTEPS(3) MJX_RSTEPS(4) MJX_RSTEPS(5) MJX_RSTEPS(6) MJX_RSTEPS(7) MJX_RSTEPS(8)
    MJX_RSTEPS(9) MJX_RSTEPS(10) MJX_RSTEPS(11) MJX_RSTEPS(12) MJX_RSTEPS(13) MJX_RSTEPS(14) MJX_RSTEPS(15)
    MJX_RSTEPS(16)
  }
#undef MJX_RSTEPS
}

template <typename T>
__global__ void __launch_bounds__(256) reactor_kernel(ReactorArgs A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const mjx_reactor_instance I = A.inst[blockIdx.x];
  const int n = I.n;
  if (n <= 256 * RMAXP) return;  // reactor_reg_kernel's
  if (I.variant < MJX_REACTOR_DANCKWERTS || I.variant > MJX_REACTOR_DANCKWERTS_CN) {  // an RK4 instance
    T* o = reinterpret_cast<T*>(A.out) + I.offset;
    for (int i = threadIdx.x; i < n; i += blockDim.x) o[i] = (T)NAN;
    return;
  }
  const int np = pz_size(n);               // padded length (index through pz)
  T* c = reinterpret_cast<T*>(smem_raw);   // state
  T* d = c + np;                           // rhs / scan values
  T* al = d + np;                          // forward scan coefficients -a_i m_i
  T* m = al + np;                          // pivots 1/(b_i - a_i c'_{i-1})
  T* cp = m + np;                          // c'_i  (backward coefficients are -c'_i)
  Aff<T>* wsum = reinterpret_cast<Aff<T>*>(cp + np);
  const int tid = threadIdx.x, nt = blockDim.x;
  const double Pe = I.Pe, Da = I.Da, dt = I.dt;
  const bool dk = I.variant == MJX_REACTOR_DANCKWERTS;
  const bool dkcn = I.variant == MJX_REACTOR_DANCKWERTS_CN;
  const double dz = (dk || dkcn) ? 1.0 / n : 1.0 / (n - 1);
  // tridiagonal entries of the implicit matrix and of the explicit operator
  double kap = 0, Ls = 0, Ld = 0, Lp = 0, Lsl = 0, Ldl = 0;
  if (dk) {
    kap = 0.5 * dt / (Pe * dz * dz);
  } else if (dkcn) {
    // M: row 0 (-2q - 1/dz - Da, q), rows 1..N-2 (q + 1/dz, -2q - 1/dz - Da, q),
    // row N-1 (2q + 1/dz, -2q - 1/dz - Da)
    const double q = (1.0 / Pe) / (dz * dz);
    Ls = q + 1.0 / dz; Ld = -2.0 * q - 1.0 / dz - Da; Lp = q;
    Lsl = 2.0 * q + 1.0 / dz; Ldl = Ld;
  } else {
    const double q = (1.0 / Pe) / (dz * dz);
    Ls = q + 1.0 / dz; Ld = -2.0 * q - 1.0 / dz - Da; Lp = q;   // rows 1..N-2
    Lsl = q; Ldl = -q - 1.0 / dz - Da;                           // row N-1
  }
  auto sub = [&](int i) -> double {  // A[i][i-1]
    if (dk) return i == n - 1 ? -2.0 * kap : -kap;
    if (i == 0) return 0.0;
    return i == n - 1 ? -0.5 * dt * Lsl : -0.5 * dt * Ls;
  };
  auto dia = [&](int i) -> double {
    if (dk) return 1.0 + 2.0 * kap;
    if (i == 0) return dkcn ? 1.0 - 0.5 * dt * Ld : 1.0;
    return i == n - 1 ? 1.0 - 0.5 * dt * Ldl : 1.0 - 0.5 * dt * Ld;
  };
  auto sup = [&](int i) -> double {  // A[i][i+1]
    if (dk) return i == n - 1 ? 0.0 : -kap;
    if (i == n - 1 || (i == 0 && !dkcn)) return 0.0;
    return -0.5 * dt * Lp;
  };
  // Thomas factorisation once (sequential, FP64)
  if (tid == 0) {
    double cprev = 0.0;
    for (int i = 0; i < n; ++i) {
      const double mi = 1.0 / (dia(i) - sub(i) * cprev);
      m[pz(i)] = (T)mi;
      al[pz(i)] = (T)(-sub(i) * mi);
      cprev = sup(i) * mi;
      cp[pz(i)] = (T)cprev;
    }
  }
  for (int i = tid; i < n; i += nt) c[pz(i)] = (T)I.c_init;
  if (!dk && !dkcn && tid == 0) c[pz(0)] = (T)I.c_inlet;
  __syncthreads();
  const T idz = (T)(1.0 / dz), Dat = (T)Da, dtt = (T)dt, kp = (T)kap;
  const T half_dt = (T)(0.5 * dt);
  for (int step = 0; step < I.n_steps; ++step) {
    // right-hand side
    for (int i = tid; i < n; i += nt) {
      const T ci = c[pz(i)];
      T r;
      if (dk) {
        const T cl = i > 0 ? c[pz(i - 1)] : (T)0, cr = i < n - 1 ? c[pz(i + 1)] : (T)0;
        T lap;  // (L c)_i dz^2
        if (i == n - 1) lap = (T)2 * cl - (T)2 * ci;
        else lap = cl - (T)2 * ci + cr;
        const T adv = i == 0 ? -(ci - (T)1) * idz : -(ci - cl) * idz;
        r = ci + kp * lap + dtt * (adv - Dat * ci);
      } else if (dkcn) {  // c + dt/2 M c + dt s
        const T cl = i > 0 ? c[pz(i - 1)] : (T)0, cr = i < n - 1 ? c[pz(i + 1)] : (T)0;
        T Mc;
        if (i == 0) Mc = (T)Ld * ci + (T)Lp * cr;
        else if (i == n - 1) Mc = (T)Lsl * cl + (T)Ldl * ci;
        else Mc = (T)Ls * cl + (T)Ld * ci + (T)Lp * cr;
        r = ci + half_dt * Mc + (i == 0 ? dtt * idz : (T)0);
      } else {
        if (i == 0) {
          r = (T)I.c_inlet;
        } else {
          const T cl = c[pz(i - 1)];
          T Lc;
          if (i == n - 1) Lc = (T)Lsl * cl + (T)Ldl * ci;
          else Lc = (T)Ls * cl + (T)Ld * ci + (T)Lp * c[pz(i + 1)];
          r = ci + half_dt * Lc;
        }
      }
      d[pz(i)] = r * m[pz(i)];  // beta_i of the forward sweep
    }
    __syncthreads();
    affine_scan<T, false>(al, d, n, wsum);      // d'_i
    // backward: x_i = d'_i - c'_i x_{i+1}; reuse c[] for the -c' coefficients
    for (int i = tid; i < n; i += nt) c[pz(i)] = -cp[pz(i)];
    __syncthreads();
    affine_scan<T, true>(c, d, n, wsum);         // x in d[]
    for (int i = tid; i < n; i += nt) c[pz(i)] = d[pz(i)];
    __syncthreads();
  }
  T* out = reinterpret_cast<T*>(A.out) + I.offset;
  for (int i = tid; i < n; i += nt) out[i] = c[pz(i)];
}

// Penalty-BC RK4 of benchmarks/benchmark_tubular_reactor.py (57-200, 254-301): n nodes,
// dz = 1/(n-1), interior rows (1/Pe) D2 c - D1 c - Da c with central D1, and the end rows
// replaced by relaxations 100 (target - c) toward the BC value (Danckwerts / Robin inlet
// (c_in + k c_1)/(1 + k), k = (1/Pe)/dz; Neumann c_1; outlet c_{n-2}, Robin written as
// (c_{n-2}/dz)/(1/dz) like the reference).  The RHS is a 3-point stencil and the state fits
// in registers: one CTA of RW warps per instance, P contiguous nodes per lane
// (n <= 32 RW P).  The stages exchange only boundary nodes: by shuffle inside a warp and
// through two shared-memory slots (alternating by stage, one barrier per stage) between
// warps.  FP64 runs at a low rate on this part and each warp issues to one SM sub-
// partition, so spreading an instance over four warps uses all four FP64 units of the SM.
enum { RW = 4 };

template <typename T, int P>
__device__ __forceinline__ void rk4_rhs(T (&s)[P], int i0, int n, int bc, T iPe, T idz2, T hidz, T Da, T kin,
                                        T cin, T idz, T* xch, int stage) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T sl = __shfl_up_sync(0xffffffffu, s[P - 1], 1);
  T sr = __shfl_down_sync(0xffffffffu, s[0], 1);
  T* slot = xch + (stage & 1) * 2 * RW;
  if (lane == 0) slot[2 * warp] = s[0];
  if (lane == 31) slot[2 * warp + 1] = s[P - 1];
  __syncthreads();
  if (lane == 0 && warp > 0) sl = slot[2 * (warp - 1) + 1];
  if (lane == 31 && warp < RW - 1) sr = slot[2 * (warp + 1)];
  // f(s) in place: each node's left neighbour is carried from the previous iteration
  // (the value before it was overwritten), so one array holds both the stage input and k
  T cm = sl;
#pragma unroll
  for (int q = 0; q < P; ++q) {
    const int i = i0 + q;
    const T cc = s[q];
    const T cp = q < P - 1 ? s[q < P - 1 ? q + 1 : 0] : sr;
    T v = iPe * ((cm - (T)2 * cc + cp) * idz2) - (cp - cm) * hidz - Da * cc;
    if (i == 0) {
      const T tgt = bc == MJX_REACTOR_RK4_NEUMANN ? cp : (cin + kin * cp) / ((T)1 + kin);
      v = (T)100 * (tgt - cc);
    } else if (i == n - 1) {
      const T tgt = bc == MJX_REACTOR_RK4_ROBIN ? (idz * cm) / idz : cm;
      v = (T)100 * (tgt - cc);
    } else if (i >= n) {
      v = (T)0;
    }
    s[q] = v;
    cm = cc;
  }
}

template <typename T, int P>
__global__ void __launch_bounds__(32 * RW) reactor_rk4_kernel(ReactorArgs A) {
  __shared__ T xch[2 * 2 * RW];
  const mjx_reactor_instance I = A.inst[blockIdx.x];
  const int n = I.n, bc = I.variant;
  T* out = reinterpret_cast<T*>(A.out) + I.offset;
  const bool ok = n >= 3 && n <= 32 * RW * P && bc >= MJX_REACTOR_RK4_DANCKWERTS && bc <= MJX_REACTOR_RK4_NEUMANN;
  if (!ok) {  // not this kernel's instance: NaN, never an out-of-range write
    for (int i = threadIdx.x; i < n && i < 32 * RW * P; i += blockDim.x) out[i] = (T)NAN;
    return;
  }
  const double dz = 1.0 / (n - 1);
  const T iPe = (T)(1.0 / I.Pe), idz2 = (T)(1.0 / (dz * dz)), hidz = (T)(0.5 / dz), Da = (T)I.Da;
  const T idz = (T)(1.0 / dz), kin = (T)((1.0 / I.Pe) / dz), cin = (T)I.c_inlet;
  const T dt = (T)I.dt, hdt = (T)(0.5 * I.dt), dt6 = (T)(I.dt / 6.0);
  const int i0 = threadIdx.x * P;
  T c[P], acc[P], y[P];
#pragma unroll
  for (int q = 0; q < P; ++q) c[q] = i0 + q < n ? (T)I.c_init : (T)0;
  for (int step = 0; step < I.n_steps; ++step) {
#pragma unroll
    for (int q = 0; q < P; ++q) y[q] = c[q];
    rk4_rhs<T, P>(y, i0, n, bc, iPe, idz2, hidz, Da, kin, cin, idz, xch, 0);  // k1
#pragma unroll
    for (int q = 0; q < P; ++q) { acc[q] = y[q]; y[q] = c[q] + hdt * y[q]; }
    rk4_rhs<T, P>(y, i0, n, bc, iPe, idz2, hidz, Da, kin, cin, idz, xch, 1);  // k2
#pragma unroll
    for (int q = 0; q < P; ++q) { acc[q] += (T)2 * y[q]; y[q] = c[q] + hdt * y[q]; }
    rk4_rhs<T, P>(y, i0, n, bc, iPe, idz2, hidz, Da, kin, cin, idz, xch, 0);  // k3
#pragma unroll
    for (int q = 0; q < P; ++q) { acc[q] += (T)2 * y[q]; y[q] = c[q] + dt * y[q]; }
    rk4_rhs<T, P>(y, i0, n, bc, iPe, idz2, hidz, Da, kin, cin, idz, xch, 1);  // k4
#pragma unroll
    for (int q = 0; q < P; ++q) c[q] = c[q] + dt6 * (acc[q] + y[q]);
  }
#pragma unroll
  for (int q = 0; q < P; ++q)
    if (i0 + q < n) out[i0 + q] = c[q];
}

// dynamic shared memory of reactor_reg_kernel: pivots and one padded row of 256 chunks with
// slack on both sides (per grows with n, so the longest instance needs the most)
static size_t reactor_reg_smem(int max_n, int elem) {
  const int n = max_n < 256 * RMAXP ? max_n : 256 * RMAXP, per = (n + 255) / 256;
  return (size_t)n * 8 + (size_t)(256 * (per + 1) + 2 * RMAXP + 6) * elem;
}

}  // namespace mjx

using namespace mjx;

extern "C" {

size_t mjx_reactor_smem_bytes(int n, int dtype) {
  const int e = elem_size(dtype);
  if (!e || n < 2) return 0;
  return (size_t)5 * pz_size(n) * e + 32 * 2 * e;
}

mjx_status mjx_reactor_cn_batch(const mjx_reactor_instance* inst_dev, int n_inst, int max_n,
                                int dtype, void* out, void* stream) {
  const int e = elem_size(dtype);
  if (!e) return MJX_BAD_DTYPE;
  if (!inst_dev || !out || n_inst < 0 || max_n < 2) return MJX_BAD_ARG;
  if (n_inst == 0) return MJX_OK;
  const size_t smem = mjx_reactor_smem_bytes(max_n, dtype);
  static ContextOnce attr;
  MJX_TRY(attr.run([]() -> mjx_status {
    int dev = 0, optin = 0;
    MJX_CUDA_TRY(cudaGetDevice(&dev));
    MJX_CUDA_TRY(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    MJX_CUDA_TRY(cudaFuncSetAttribute(reactor_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin));
    MJX_CUDA_TRY(cudaFuncSetAttribute(reactor_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin));
    const int reg = (int)reactor_reg_smem(256 * RMAXP, 8);
    MJX_CUDA_TRY(cudaFuncSetAttribute(reactor_reg_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, reg));
    MJX_CUDA_TRY(cudaFuncSetAttribute(reactor_reg_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, reg));
    return MJX_OK;
  }));
  if (smem > 227 * 1024) return MJX_BAD_SHAPE;
  ReactorArgs A;
  A.inst = inst_dev; A.out = out; A.n_inst = n_inst;
  cudaStream_t s = (cudaStream_t)stream;
  // instances of up to 4096 nodes run in registers, longer ones (FP32 up to 10 900, FP64 up to
  // 5 400, whose state does not fit 256 threads) in shared memory; each kernel leaves the
  // other's instances alone, so an instance's result does not depend on the batch
  const size_t rsm = reactor_reg_smem(max_n, e);
  if (e == 4) reactor_reg_kernel<float><<<n_inst, 256, rsm, s>>>(A);
  else reactor_reg_kernel<double><<<n_inst, 256, rsm, s>>>(A);
  MJX_CUDA_TRY(cudaGetLastError());
  if (max_n > 256 * RMAXP) {
    if (e == 4) reactor_kernel<float><<<n_inst, 256, smem, s>>>(A);
    else reactor_kernel<double><<<n_inst, 256, smem, s>>>(A);
  }
  return cuda_status(cudaGetLastError());
}

mjx_status mjx_reactor_rk4_batch(const mjx_reactor_instance* inst_dev, int n_inst, int max_n, int dtype,
                                 void* out, void* stream) {
  const int e = elem_size(dtype);
  if (!e) return MJX_BAD_DTYPE;
  if (!inst_dev || !out || n_inst < 0 || max_n < 3) return MJX_BAD_ARG;
  if (max_n > 32 * RW * 8) return MJX_BAD_SHAPE;  // at most 8 nodes per lane
  if (n_inst == 0) return MJX_OK;
  ReactorArgs A;
  A.inst = inst_dev; A.out = out; A.n_inst = n_inst;
  cudaStream_t s = (cudaStream_t)stream;
  const int per = (max_n + 32 * RW - 1) / (32 * RW);  // nodes per lane
#define MJX_RK4_LAUNCH(PP)                                                         \
  do {                                                                             \
    if (e == 4) reactor_rk4_kernel<float, PP><<<n_inst, 32 * RW, 0, s>>>(A);       \
    else reactor_rk4_kernel<double, PP><<<n_inst, 32 * RW, 0, s>>>(A);             \
  } while (0)
  if (per <= 1) MJX_RK4_LAUNCH(1);
  else if (per <= 2) MJX_RK4_LAUNCH(2);
  else if (per <= 4) MJX_RK4_LAUNCH(4);
  else MJX_RK4_LAUNCH(8);
#undef MJX_RK4_LAUNCH
  return cuda_status(cudaGetLastError());
}

}  // extern "C"
