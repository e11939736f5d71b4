// Mixed-precision (float-float spectral state) building blocks of the adaptive
// IMEX-Strang attempt, shared by the single-solve driver (csrc/imex_mixed.cu)
// and the batched engine (csrc/imex_batch.cu).  See csrc/imex_mixed.cu for the
// attempt's six passes.
#pragma once

#include "spectral.cuh"

namespace mjx {

// The three column passes of an attempt.  The two halves of a CTA's threads take the full step
// (A) and the half steps (B) of the same columns.
enum { MC_SPLIT = 0, MC_MID = 1, MC_HALF_END = 2 };

__device__ __forceinline__ float2 fmk(float x, float y) { float2 r; r.x = x; r.y = y; return r; }

// ---- float-float arithmetic (error-free transformations: Knuth's two-sum,
// Dekker's fast two-sum, the FMA two-product).  The _rn intrinsics are never
// contracted into FMAs or reassociated, which the transformations rely on.
struct FF { float h, l; };

__device__ __forceinline__ FF ff_fast2sum(float a, float b) {  // |a| >= |b| or a == 0
  const float s = __fadd_rn(a, b);
  FF r; r.h = s; r.l = __fsub_rn(b, __fsub_rn(s, a));
  return r;
}
__device__ __forceinline__ float ff_2sum_err(float a, float b, float s) {  // s = fl(a + b)
  const float bb = __fsub_rn(s, a);
  return __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}
// x + d, d an FP32 number
__device__ __forceinline__ FF ff_add_f(FF x, float d) {
  const float s = __fadd_rn(x.h, d);
  return ff_fast2sum(s, __fadd_rn(ff_2sum_err(x.h, d, s), x.l));
}
// x + x * mu
__device__ __forceinline__ FF ff_mstep(FF x, float mu) {
  const float p = __fmul_rn(x.h, mu);
  const float pe = __fmaf_rn(x.l, mu, __fmaf_rn(x.h, mu, -p));  // x*mu - p
  const float s = __fadd_rn(x.h, p);
  return ff_fast2sum(s, __fadd_rn(ff_2sum_err(x.h, p, s), __fadd_rn(x.l, pe)));
}
// s * (x - y) rounded to FP32 (the hi difference is exact when x, y are close)
__device__ __forceinline__ float ff_diff_scaled(FF x, FF y, float s) {
  return __fmul_rn(__fadd_rn(__fsub_rn(x.h, y.h), __fsub_rn(x.l, y.l)), s);
}
// s * x rounded to FP32
__device__ __forceinline__ float ff_scaled(FF x, float s) { return __fmaf_rn(x.l, s, __fmul_rn(x.h, s)); }

__device__ __forceinline__ FF ff_re(float4 v) { FF r; r.h = v.x; r.l = v.z; return r; }
__device__ __forceinline__ FF ff_im(float4 v) { FF r; r.h = v.y; r.l = v.w; return r; }
__device__ __forceinline__ float4 ff_pack(FF re, FF im) { return make_float4(re.h, im.h, re.l, im.l); }

// mu = x/(1-x), x = hD * lam (FP32, |1-x| clamped at 1e-14 like the reference)
__device__ __forceinline__ float mu_of(float hD, float lam) {
  const float x = hD * lam;
  float den = 1.0f - x;
  if (fabsf(den) < 1e-14f) den = 1e-14f;
  return x / den;
}
__device__ __forceinline__ float4 ff_mstep_c(float4 X, float mu) {
  return ff_pack(ff_mstep(ff_re(X), mu), ff_mstep(ff_im(X), mu));
}
__device__ __forceinline__ float4 ff_add_c(float4 X, float2 d) {
  return ff_pack(ff_add_f(ff_re(X), d.x), ff_add_f(ff_im(X), d.y));
}

// Everything one column tile of a mixed attempt needs: the single-solve kernel
// fills it from MColArgs, the batched kernel (csrc/imex_batch.cu) from its
// instance table.
struct MColTile {
  int ny, log2ny, ncols, C, kx0;
  long long ldc, off;       // row stride; field offset shared by every buffer
  const float4* ys_cur;     // state Y^[cur]
  float4* ys_next;          // state Y^[1-cur]
  float4* pa;
  float4* pb;
  float2* za;
  float2* zb;
  const float* lamx;
  const float* lamy;
  const float2* tw;
  float hA, hB, nrm;        // dt/2 D, dt/4 D, 1/(nx ny)
};

// shared memory of a tile: the two halves side by side
inline size_t mcol_smem(int ny, int C) { return 2 * (size_t)sp_size(ny * C) * sizeof(float2); }

// One tile: C adjacent kx columns of one field over all ny rows, C ny/16 threads (C below 16
// rows) for each half.  A thread holds its 16 elements in registers from the load to the store
// (fft_regs; 64 registers, so that four 256-thread or two 512-thread CTAs share an SM and hide
// each other's L2 latency, which bounds these passes at 1024^2), the operands of NB elements at a
// time.  C3 runs its forward transform and its update in both halves: the idle half would save
// nothing and the exchange costs two barriers.
//   C1 MC_SPLIT     PA = M_A Y, PB = M_B Y; ZA, ZB <- inverse of both
//   C2 MC_MID       PA <- M_A (PA + F ZA);  PB <- M_B^2 (PB + F ZB), ZB <- its inverse
//   C3 MC_HALF_END  Y' = M_B (PB + F ZB); ZA <- inverse of Y' - PA, ZB <- inverse of Y'
// LOG2NY, CN > 0 fix the column length and the tile width at compile time (the lengths 64 to
// 4096, in the batch every length), so that the index arithmetic and the radix schedule fold into
// the code; shorter columns of a single solve read both (8 x 64 to 32 x 4096 a solve 1.4 to 1.6 times
// as fast as with every element in shared memory).  C1 / C2 / C3 at 1024^2: 14 / 20 / 21 us, against 24 us each with every element in
// shared memory between the transforms; 256^2 1.8x a solve.  Four operands in flight beat two in
// C1 (13.6 against 14.6 us) and lose in C2 and C3 (24 us), whose registers they overflow; with two
// C2 spills 116 bytes a thread and C3 16 at 1024 rows.
template <int TYPE, int LOG2NY = 0, int CN = 0>
__device__ __forceinline__ void mcol_tile(float2* buf, const MColTile& t, int tid) {
  const int ny = LOG2NY ? (1 << LOG2NY) : t.ny, log2ny = LOG2NY ? LOG2NY : t.log2ny;
  const int Cn = CN ? CN : t.C;  // a power of two
  const int tps = ny >= 16 ? ny >> 4 : 1, per = Cn * tps;
  const bool right = tid >= per, active = tid < 2 * per;
  const int r = right ? tid - per : tid, c = r & (Cn - 1), lt = r >> (__ffs(Cn) - 1);
  const int kx = t.kx0 + c, ldc = (int)t.ldc;
  const bool in = active && kx < t.ncols;
  const long long g0 = t.off + (long long)lt * ldc + kx;
  const int gs = tps * ldc;
  float2* half = buf + (right ? sp_size(ny * Cn) : 0);
  const float nrm = t.nrm, lx = in ? t.lamx[kx] : 0.f;
  const float* lamy = t.lamy + lt;
  float2 x[16];
#pragma unroll
  for (int q = 0; q < 16; ++q) x[q] = fmk(0.f, 0.f);

  if (TYPE != MC_SPLIT) {
    const float2* z = ((TYPE == MC_MID && !right) ? t.za : t.zb) + g0;
    if (in) {
#pragma unroll
      for (int q = 0; q < 16; ++q)
        if (q * tps < ny) x[q] = z[q * gs];
    }
    fft_regs<float, false, false>(x, half, ny, log2ny, lt, c, Cn, t.tw, active);
  }

  // float-float combine
  const bool two = TYPE == MC_HALF_END && !right;  // two operands
  const float4* op = (TYPE == MC_SPLIT ? t.ys_cur : ((TYPE == MC_MID && !right) ? t.pa : t.pb)) + g0;
  const float4* oq = t.pa + g0;
  float4* res = (TYPE == MC_HALF_END ? t.ys_next : (right ? t.pb : t.pa)) + g0;
  const float hD = (TYPE == MC_HALF_END || right) ? t.hB : t.hA;
  constexpr int NB = TYPE == MC_SPLIT ? 4 : 2;  // elements whose operands are in flight together
  if (in) {
#pragma unroll
    for (int q0 = 0; q0 < 16; q0 += NB) {
      float4 P[NB], Q[NB];
      float lam[NB];
#pragma unroll
      for (int h = 0; h < NB; ++h) {
        const int q = q0 + h;
        if (q * tps >= ny) continue;
        P[h] = op[q * gs];
        if (two) Q[h] = oq[q * gs];
        lam[h] = lx + lamy[q * tps];
      }
#pragma unroll
      for (int h = 0; h < NB; ++h) {
        const int q = q0 + h;
        if (q * tps >= ny) continue;
        const float mu = mu_of(hD, lam[h]);
        float4 X = TYPE == MC_SPLIT ? P[h] : ff_add_c(P[h], x[q]);
        X = ff_mstep_c(X, mu);
        if (TYPE == MC_MID && right) X = ff_mstep_c(X, mu);
        if (TYPE != MC_HALF_END || right) res[q * gs] = X;
        x[q] = two ? fmk(ff_diff_scaled(ff_re(X), ff_re(Q[h]), nrm), ff_diff_scaled(ff_im(X), ff_im(Q[h]), nrm))
                   : fmk(ff_scaled(ff_re(X), nrm), ff_scaled(ff_im(X), nrm));
      }
    }
  }
  if (TYPE != MC_SPLIT) __syncthreads();
  const bool back = active && (TYPE != MC_MID || right);  // C2 keeps PA in spectral space
  fft_regs<float, true, false>(x, half, ny, log2ny, lt, c, Cn, t.tw, back);
  float2* z = (right ? t.zb : t.za) + g0;
  if (in && back) {
#pragma unroll
    for (int q = 0; q < 16; ++q)
      if (q * tps < ny) z[q * gs] = x[q];
  }
}

// Initial state: y ([nf][ny][nx], io_dtype) -> FP64 transform (plan64) -> the
// float-float half spectrum ys ([nf][ny][ldc] float4).  real64 is scratch of
// nf*ny*nx doubles (it may alias the PA buffer of a mixed workspace, not ys).
mjx_status mix_state_from_real(const void* plan64, const mjx_grid2d* g, int nf, int io_dtype, const void* y,
                               double* real64, float4* ys, cudaStream_t s);
// Final state: the float-float spectrum Y^[cur] (cur read on the device from st, or 0
// when st is null) -> FP64 inverse transform -> y_out (io_dtype).  spec64 holds
// nf*ny*ldc double2 and real64 nf*ny*nx doubles of scratch; neither may alias ys0/ys1.
mjx_status mix_real_from_state(const void* plan64, const mjx_grid2d* g, int nf, const DevState* st,
                               const float4* ys0, const float4* ys1, double2* spec64, double* real64,
                               int io_dtype, void* y_out, cudaStream_t s);

}  // namespace mjx
