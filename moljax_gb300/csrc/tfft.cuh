// Tile DFT in shared memory: S = 2^lS interleaved sequences (element j of sequence s at
// sp(j S + s)), mixed radices 2, 3, 4, 5, 8, Stockham autosort between two buffers.
//
// All butterflies of a pass (n / R of them for each sequence) are one flat list over which any
// number of threads strides, neighbouring threads on neighbouring words: every warp but the
// last of a pass is full, whatever n and R are.  That matters most in FP64, where a warp's
// instruction takes 64 cycles of its sub-partition with any number of active lanes.  Two
// buffers cost shared memory and save a barrier a pass.
//
// FP64 twiddles are stored as (cos, tan) of their angle: with w = e^{-i theta} = c (1 - i t),
//   a +- w b = (a.x +- c u, a.y +- c v),  u = b.x + t b.y,  v = b.y - t b.x,
// six fused multiply-adds instead of the ten operations of a complex product and two sums, and
// two roundings a component instead of three (the scheme of Linzer and Feig, 1993).  Radix 4
// takes 24 FP64 instructions instead of 34, radix 8 72 instead of 84.  A transform in radix 2 to 8
// has up to twice the passes of one in radix 16, which takes the gain in rounding back in part
// (128^2 FFT-CN 2.5e-14 -> 2.4e-14 after 100 steps, 128^3 3.1e-15 -> 3.2e-15 after 10).  At
// theta = pi/2 and 3 pi/2 the pair is (2^-60, +-2^60), so FP64 points stay below 2^963 (8e289).
// FP32 keeps (cos, -sin): it is not bound by its arithmetic, and the large tangents would shorten
// its range.
#pragma once

#include <math.h>

#include "fft.cuh"
#include "roots.cuh"

namespace mjx {

// host: entry j of a twiddle table in the form that tile_dft reads, from the roots of its length
inline void tile_twiddle(const Roots& r, int j, int elem, double* re, double* im) {
  const DD c = r.c[j], s = r.s[j];
  if (elem == 4) {
    *re = c.h;
    *im = -s.h;
  } else if (c.h == 0.0) {  // pi / 2, 3 pi / 2
    *re = 0x1p-60;
    *im = s.h > 0.0 ? 0x1p60 : -0x1p60;
  } else {  // the tangent belongs to the rounded cosine, so that their product is the sine
    *re = c.h;
    *im = dd_div(s, c.h).h;
  }
}

// w b
__device__ __forceinline__ float2 tw_mul(float2 b, float2 w) { return cmul(b, w); }
__device__ __forceinline__ double2 tw_mul(double2 b, double2 w) {
  return mk<double2>(w.x * fma(w.y, b.y, b.x), w.x * fma(-w.y, b.x, b.y));
}
// (a, b) <- (a + w b, a - w b)
__device__ __forceinline__ void tw_bf(float2& a, float2& b, float2 w) {
  const float2 t = cmul(b, w);
  b = csub(a, t);
  a = cadd(a, t);
}
__device__ __forceinline__ void tw_bf(double2& a, double2& b, double2 w) {
  const double u = fma(w.y, b.y, b.x), v = fma(-w.y, b.x, b.y);
  b = mk<double2>(fma(-w.x, u, a.x), fma(-w.x, v, a.y));
  a = mk<double2>(fma(w.x, u, a.x), fma(w.x, v, a.y));
}
// (a, b) <- (a - i w b, a + i w b)
__device__ __forceinline__ void tw_bfr(float2& a, float2& b, float2 w) {
  const float2 t = rot<false>(cmul(b, w));
  b = csub(a, t);
  a = cadd(a, t);
}
__device__ __forceinline__ void tw_bfr(double2& a, double2& b, double2 w) {
  const double u = fma(w.y, b.y, b.x), v = fma(-w.y, b.x, b.y);
  b = mk<double2>(fma(-w.x, v, a.x), fma(w.x, u, a.y));
  a = mk<double2>(fma(w.x, v, a.x), fma(-w.x, u, a.y));
}

// v <- DFT_R(v_t w^t) in natural order, w^t the table entry at t * i; ne = n / 8 (radix 8).
// FP64 folds the twiddles into the butterfly's sums.  FP32, which gains no operation by that,
// multiplies each point by its own table entry: folded, a point of radix 4 and 8 goes through two or
// three rounded twiddles.  Error of 50 steps against that of the separate full-spectrum passes, mean
// over 40 grids of 5 to 400 points a side: 0.84, folded 1.10.  The longest Bluestein lengths, whose
// tables stay in global memory, take 7 to 10 % longer for it (1600 x 1001: 254 -> 272 us, 3 steps).
template <typename T, int R, bool FIRST>
__device__ __forceinline__ void tile_bf(cx<T>* v, const cx<T>* tw, int i, int ne) {
  if constexpr (sizeof(T) == 4 && R > 2 && !FIRST) {
#pragma unroll
    for (int t = 1; t < R; ++t) v[t] = cmul(v[t], tw[t * i]);
    return tile_bf<T, R, true>(v, tw, 0, 0);
  }
  typedef cx<T> C;
  if constexpr (R == 2) {
    if (FIRST) dft2<false>(v[0], v[1]);
    else tw_bf(v[0], v[1], tw[i]);
  } else if constexpr (R == 3) {
    const T h = (T)0.86602540378443864676;  // sin(2 pi / 3)
    C t, d = v[2];
    if (FIRST) {
      t = cadd(v[1], v[2]); d = csub(v[1], v[2]);
    } else {
      t = tw_mul(v[1], tw[i]);
      tw_bf(t, d, tw[2 * i]);
    }
    const C a = v[0], m = mk<C>(a.x - (T)0.5 * t.x, a.y - (T)0.5 * t.y);
    v[0] = cadd(a, t);
    v[1] = mk<C>(m.x + h * d.y, m.y - h * d.x);
    v[2] = mk<C>(m.x - h * d.y, m.y + h * d.x);
  } else if constexpr (R == 4) {
    if (FIRST) {
      dft4<false>(v[0], v[1], v[2], v[3]);
    } else {
      const C w1 = tw[i], w2 = tw[2 * i];
      tw_bf(v[0], v[2], w2);
      tw_bf(v[1], v[3], w2);
      tw_bf(v[0], v[1], w1);
      tw_bfr(v[2], v[3], w1);
      const C t = v[1];  // X0, X2, X1, X3 -> natural order
      v[1] = v[2]; v[2] = t;
    }
  } else if constexpr (R == 5) {
    // cos / sin of 2 pi/5 and 4 pi/5
    const T c1 = (T)0.30901699437494742410, c2 = (T)-0.80901699437494742410;
    const T s1 = (T)0.95105651629515357212, s2 = (T)0.58778525229247312917;
    C t1, t2, t3 = v[4], t4 = v[3];
    if (FIRST) {
      t1 = cadd(v[1], v[4]); t3 = csub(v[1], v[4]);
      t2 = cadd(v[2], v[3]); t4 = csub(v[2], v[3]);
    } else {
      t1 = tw_mul(v[1], tw[i]);
      tw_bf(t1, t3, tw[4 * i]);
      t2 = tw_mul(v[2], tw[2 * i]);
      tw_bf(t2, t4, tw[3 * i]);
    }
    const C a = v[0];
    const C m1 = mk<C>(a.x + c1 * t1.x + c2 * t2.x, a.y + c1 * t1.y + c2 * t2.y);
    const C m2 = mk<C>(a.x + c2 * t1.x + c1 * t2.x, a.y + c2 * t1.y + c1 * t2.y);
    const C n1 = mk<C>(s1 * t3.x + s2 * t4.x, s1 * t3.y + s2 * t4.y);
    const C n2 = mk<C>(s2 * t3.x - s1 * t4.x, s2 * t3.y - s1 * t4.y);
    v[0] = mk<C>(a.x + t1.x + t2.x, a.y + t1.y + t2.y);
    v[1] = mk<C>(m1.x + n1.y, m1.y - n1.x);  // m1 - i n1
    v[4] = mk<C>(m1.x - n1.y, m1.y + n1.x);  // m1 + i n1
    v[2] = mk<C>(m2.x + n2.y, m2.y - n2.x);
    v[3] = mk<C>(m2.x - n2.y, m2.y + n2.x);
  } else {
    if (FIRST) {
      dft8<false>(v);
    } else {
      // even and odd samples as radix 4 with w^2, then the odd half with w and w e^{-i pi/4}
      const C w1 = tw[i], w2 = tw[2 * i], w4 = tw[4 * i], we = tw[i + ne];
      tw_bf(v[0], v[4], w4);
      tw_bf(v[2], v[6], w4);
      tw_bf(v[1], v[5], w4);
      tw_bf(v[3], v[7], w4);
      tw_bf(v[0], v[2], w2);   // E0, E2
      tw_bfr(v[4], v[6], w2);  // E1, E3
      tw_bf(v[1], v[3], w2);   // O0, O2
      tw_bfr(v[5], v[7], w2);  // O1, O3
      tw_bf(v[0], v[1], w1);   // X0, X4
      tw_bf(v[4], v[5], we);   // X1, X5
      tw_bfr(v[2], v[3], w1);  // X2, X6
      tw_bfr(v[6], v[7], we);  // X3, X7
      const C x1 = v[4], x2 = v[2], x3 = v[6], x4 = v[1], x6 = v[3];
      v[1] = x1; v[2] = x2; v[3] = x3; v[4] = x4; v[6] = x6;
    }
  }
}

// a / b for 0 <= a < 2^20, b >= 1, given 1.0f / b: exact, since the half keeps the quotient
// away from integers by 1/(2b), more than the roundings can move it
__device__ __forceinline__ int fdiv(int a, float rb) { return (int)(((float)a + 0.5f) * rb); }

// One pass: butterfly j (k = j mod p) of each sequence from src[j + t n/R] to
// dst[(j - k) R + k + t p], after the twiddles w^(k t), w = exp(-2 pi i / (p R)).  A stride that
// is a multiple of 16 points keeps the padding's phase, so the R addresses are one base and
// multiples of a constant; on small tiles, with a warp or two on each sub-partition, the index
// arithmetic is as long as the FP64 arithmetic.
template <typename T, int R>
__device__ __forceinline__ void tile_load(cx<T>* v, const cx<T>* src, int i, int stride) {
  if ((stride & 15) == 0) {
    const cx<T>* q = src + sp(i);
    const int d = sp(stride);
#pragma unroll
    for (int t = 0; t < R; ++t) v[t] = q[t * d];
  } else {
#pragma unroll
    for (int t = 0; t < R; ++t) v[t] = src[sp(i + t * stride)];
  }
}
template <typename T, int R>
__device__ __forceinline__ void tile_store(const cx<T>* v, cx<T>* dst, int i, int stride) {
  if ((stride & 15) == 0) {
    cx<T>* q = dst + sp(i);
    const int d = sp(stride);
#pragma unroll
    for (int t = 0; t < R; ++t) q[t * d] = v[t];
  } else {
#pragma unroll
    for (int t = 0; t < R; ++t) dst[sp(i + t * stride)] = v[t];
  }
}

template <typename T, int R>
__device__ __forceinline__ void tile_pass(const cx<T>* src, cx<T>* dst, int n, int p, int lS, const cx<T>* tw,
                                          int tid, int nth) {
  typedef cx<T> C;
  const int nb = n / R, items = nb << lS, S1 = (1 << lS) - 1;
  if (p == 1) {
#pragma unroll 1
    for (int i = tid; i < items; i += nth) {
      const int s = i & S1;
      C v[R];
      tile_load<T, R>(v, src, i, items);
      tile_bf<T, R, true>(v, tw, 0, 0);
      tile_store<T, R>(v, dst, (i - s) * R + s, 1 << lS);
    }
  } else {
    const int step = nb / p, pS = p << lS;
    const bool p2 = (p & (p - 1)) == 0;
    const float rp = 1.0f / (float)p;
#pragma unroll 1
    for (int i = tid; i < items; i += nth) {
      // ks = k 2^lS + s: the place within the block of p butterflies of every sequence
      const int ks = p2 ? i & (pS - 1) : i - fdiv(i >> lS, rp) * pS, k = ks >> lS;
      C v[R];
      tile_load<T, R>(v, src, i, items);
      tile_bf<T, R, false>(v, tw, k * step, n >> 3);
      tile_store<T, R>(v, dst, (i - ks) * R + ks, pS);
    }
  }
  __syncthreads();
}

// A radix-2 FP64 pass with the two components of each butterfly on neighbouring lanes: each needs
// one of the products u, v and two sums, so a tile of fewer than 128 butterflies fills twice the
// warps with half the FP64 instructions each (a 128-point row: 128 lanes, three instructions).
static __device__ __forceinline__ void tile_pass2_split(const double2* src, double2* dst, int n, int p, int lS,
                                                 const double2* tw, int tid, int nth) {
  const int items = (n >> 1) << lS, pS = p << lS, step = (n >> 1) / p;
  const double* sr = reinterpret_cast<const double*>(src);
  double* ds = reinterpret_cast<double*>(dst);
#pragma unroll 1
  for (int e = tid; e < 2 * items; e += nth) {
    const int i = e >> 1, y = e & 1;
    const int ks = (p & (p - 1)) == 0 ? i & (pS - 1) : i % pS;
    const double2 w = tw[(ks >> lS) * step];
    const double2 b = src[sp(i + items)];
    const double a = sr[2 * sp(i) + y];
    const double u = fma(w.y, y ? -b.x : b.y, y ? b.y : b.x);
    const int o = (i - ks) * 2 + ks;
    ds[2 * sp(o) + y] = fma(w.x, u, a);
    ds[2 * sp(o + pS) + y] = fma(-w.x, u, a);
  }
  __syncthreads();
}

// Forward DFT of length n of every sequence in cur; the result is in cur after an even number
// of passes, in alt after an odd one.  The caller has synchronised; on return the tile is
// complete.  Radices are packed four bits each, the first pass lowest.  One copy of the code
// per kernel: a kernel runs two to six transforms, and inlined copies cost more in instruction
// fetches than the passes themselves on small tiles.
// POW2: only the passes of powers of two (the less code, the fewer fetches).
template <typename T, bool POW2>
__device__ __noinline__ void tile_dft(cx<T>* cur, cx<T>* alt, int n, unsigned long long rad, int lS, const cx<T>* tw,
                                      int tid, int nth) {
  for (int p = 1; rad != 0; rad >>= 4) {
    const int r = (int)(rad & 15);
    if (r == 8) tile_pass<T, 8>(cur, alt, n, p, lS, tw, tid, nth);
    else if (r == 4) tile_pass<T, 4>(cur, alt, n, p, lS, tw, tid, nth);
    else if (!POW2 && r == 5) tile_pass<T, 5>(cur, alt, n, p, lS, tw, tid, nth);
    else if (!POW2 && r == 3) tile_pass<T, 3>(cur, alt, n, p, lS, tw, tid, nth);
    else {
      bool split = false;
      if constexpr (sizeof(T) == 8) {
        split = (n >> 1) << lS < 128;
        if (split) tile_pass2_split(cur, alt, n, p, lS, tw, tid, nth);
      }
      if (!split) tile_pass<T, 2>(cur, alt, n, p, lS, tw, tid, nth);
    }
    cx<T>* t = cur;
    cur = alt;
    alt = t;
    p *= r;
  }
}

// packed radices of a power of two 2^l, at most `top` (8, 4 or 2): eights, the rest as fours (or
// one two); *passes their count
inline unsigned long long tile_pow2_radices(int l, int top, int* passes) {
  unsigned long long rad = 0;
  int k = 0, eights = top >= 8 ? l / 3 : 0, rest = l - 3 * eights;
  auto put = [&](int r) { rad |= (unsigned long long)r << (4 * k++); };
  if (rest == 1 && eights > 0) { --eights; rest = 4; }  // 2^(3a+1) = 8^(a-1) 4 4
  for (int i = 0; i < eights; ++i) put(8);
  for (; top >= 4 && rest >= 2; rest -= 2) put(4);
  for (; rest >= 1; --rest) put(2);
  *passes = k;
  return rad;
}

// ------------------------------------------------------------------ lengths of every kind
// A DFT of length n over a tile: powers of two and mixed radices directly (L = n), other
// lengths by Bluestein's chirp-z form with FFTs of length L.
template <typename T>
struct Dft {
  const cx<T>* tw;    // length-L twiddles in the form of tile_dft
  const cx<T>* chirp; // length n
  const cx<T>* bhat;  // length L, FFT_L(b) / L
  int n, L, bluestein;
  int odd;            // an odd number of passes: the buffers swap
  int log2L;          // powers of two and Bluestein; 0 for mixed radices
  int tps;            // threads per sequence
  int staged;         // the tables are copied to shared memory first
  unsigned long long rad;
};

// A tile's two buffers and its tables.  Small tiles copy the tables to shared memory while
// their data loads are in flight: a pass whose twiddles come from a cold L1 waits ~700 cycles
// for L2, several times the pass itself.
template <typename T>
struct Tile {
  cx<T>* cur;
  cx<T>* alt;
  const cx<T>* tw;
  const cx<T>* chirp;
  const cx<T>* bhat;
  int lS, tid, nth;
};

template <typename T>
__device__ __forceinline__ Tile<T> tile_begin(const Dft<T>& d, unsigned char* smem, int lS) {
  typedef cx<T> C;
  Tile<T> t;
  const int m = sp_size(d.L << lS);
  t.cur = reinterpret_cast<C*>(smem);
  t.alt = t.cur + m;
  t.lS = lS; t.tid = threadIdx.x; t.nth = blockDim.x;
  t.tw = d.tw; t.chirp = d.chirp; t.bhat = d.bhat;
  if (d.staged) {
    C* w = t.alt + m;
    for (int i = t.tid; i < d.L; i += t.nth) w[i] = __ldg(&d.tw[i]);
    t.tw = w;
    if (d.bluestein) {
      C* b = w + d.L;
      C* c = b + d.L;
      for (int i = t.tid; i < d.L; i += t.nth) b[i] = __ldg(&d.bhat[i]);
      for (int i = t.tid; i < d.n; i += t.nth) c[i] = __ldg(&d.chirp[i]);
      t.bhat = b; t.chirp = c;
    }
  }
  return t;
}

// Forward DFT of the tile's sequences (elements 0 .. n - 1 of each), left in t.cur.  The caller
// has synchronised.
template <typename T>
__device__ __forceinline__ void dft_tile(const Dft<T>& d, Tile<T>& t) {
  typedef cx<T> C;
  const int lS = t.lS, L = d.L, n = d.n;
  if (d.bluestein) {
    for (int e = t.tid; e < (L << lS); e += t.nth) {
      const int j = e >> lS;
      t.cur[sp(e)] = j < n ? cmul(t.cur[sp(e)], t.chirp[j]) : mk<C>((T)0, (T)0);
    }
    __syncthreads();
  }
  tile_dft<T, false>(t.cur, t.alt, L, d.rad, lS, t.tw, t.tid, t.nth);
  if (d.odd) { C* x = t.cur; t.cur = t.alt; t.alt = x; }
  if (!d.bluestein) return;
  // the inverse transform of the product by conjugation
  for (int e = t.tid; e < (L << lS); e += t.nth) t.cur[sp(e)] = cconj(cmul(t.cur[sp(e)], t.bhat[e >> lS]));
  __syncthreads();
  tile_dft<T, false>(t.cur, t.alt, L, d.rad, lS, t.tw, t.tid, t.nth);
  if (d.odd) { C* x = t.cur; t.cur = t.alt; t.alt = x; }
  for (int e = t.tid; e < (n << lS); e += t.nth) t.cur[sp(e)] = cmul(cconj(t.cur[sp(e)]), t.chirp[e >> lS]);
  __syncthreads();
}

template <typename T>
inline size_t tile_smem(const Dft<T>& d, int l) {
  size_t e = 2 * (size_t)sp_size(d.L << l);
  if (d.staged) e += (size_t)d.L + (d.bluestein ? (size_t)d.L + d.n : 0);
  return e * sizeof(cx<T>);
}

// Sequences per CTA (log2) for `total` sequences: up to `want`, or more where they are short (up
// to 256 threads: fuller warps, 100^3 FP64 2.70 -> 1.99 ms for 10 steps with the schedule that
// the tuner then picks), within 512 threads and 96 KB of shared memory (one sequence may take
// more), halved until the pass has about one CTA per SM;
// tables in shared memory where the whole stays under 96 KB.  A pass with few sequences doubles
// the threads of each (n/4 instead of n/8): its time is a chain of passes, not throughput.
template <typename T>
inline int tile_log(Dft<T>& d, long long total, int want) {
  const size_t cap = 96 * 1024;
  int l = 0;
  while ((2 << l) <= 32 && ((2 << l) <= want || (2 << l) * d.tps <= 256) && (2 << l) * d.tps <= 512 &&
         tile_smem<T>(d, l + 1) <= cap)
    ++l;
  while (l > 0 && (total + (1 << l) - 1) >> l < 128) --l;
  if (((d.tps << l) + 31) / 32 * ((total + (1 << l) - 1) >> l) < 152 * 8 && (2 * d.tps << l) <= 512) d.tps *= 2;
  d.staged = 1;
  if (tile_smem<T>(d, l) > cap) d.staged = 0;
  if (d.log2L > 0) {
    // FP64: the largest radix whose butterflies still give each sub-partition a warp (an FP64
    // radix-8 pass on two of four warps takes longer than the passes that it saves: 64 x 96
    // FFT-CN 26.7 -> 22.7 us a step)
    int top = 8, passes = 0;
    if (sizeof(T) == 8)
      while (top > 2 && ((d.L / top) << l) < 128) top >>= 1;
    d.rad = tile_pow2_radices(d.log2L, top, &passes);
    d.odd = passes & 1;
    if (sizeof(T) == 8 && d.tps << l < 128) d.tps = 128 >> l;
  }
  return l;
}

template <typename T>
inline int tile_threads(const Dft<T>& d, int l) {
  const int t = ((d.tps << l) + 31) & ~31;
  return t < 64 ? 64 : (t > 512 ? 512 : t);
}

}  // namespace mjx
