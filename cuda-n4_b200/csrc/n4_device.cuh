// Device helpers shared by every n4b200 kernel (sm_100a).
//
// * per-axis cubic B-spline tables (span index, weights, fit weights),
//   computed in FP64 with the reference's formulas (N4.py:174-181,
//   N4.py:210-222) and stored in FP32;
// * a CTA-level Stockham radix-4/2 FFT in shared memory and the Gaussian
//   Wiener-deconvolution sharpening map built on it (N4.py:32-101,
//   cudaN4.cu:733-817);
// * fractional-histogram binning and the piecewise-linear remap
//   (N4.py:14-29, N4.py:103-113);
// * warp/CTA reductions and a bounded software grid barrier.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/n4b200.h"

namespace n4 {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kHistCopies = 8;                   // shared histogram copies per CTA
constexpr int kHistMaxShift = 24;                // fixed-point weight 2^shift, shift <= 24
constexpr unsigned long long kSpinLimit = 1ull << 23;   // bounded waits (a few seconds)

// ---------------------------------------------------------------- tables
// One axis of the fitting grid at one level.  Arrays live in shared or
// global memory; all pointers are generic.
struct Axis {
  int n;        // voxels along the axis
  int nc;       // control points (= spans + 3)
  int nsp;      // spans
  int *s;       // [n]   span index of each voxel
  float4 *w;    // [n]   cubic weights B0..B3
  float *p;     // [4][n] fit numerator weights  w_j^3 / sum_k w_k^2
  float *q;     // [4][n] fit denominator weights w_j^2
  float4 *p4;   // [n]   the same numerator weights, packed per voxel
  float4 *q4;   // [n]   the same denominator weights, packed per voxel
  int *lo, *hi; // [nsp] voxel range of each span
};

// Byte size of an axis table with `n` voxels and `nsp` spans (16-B multiple).
__host__ __device__ inline size_t axis_bytes(int n, int nsp) {
  size_t b = 0;
  b += ((size_t)n * 4 + 15) / 16 * 16;          // s
  b += (size_t)n * 16;                           // w
  b += (size_t)n * 16 * 2;                       // p, q
  b += (size_t)n * 16 * 2;                       // p4, q4
  b += ((size_t)nsp * 8 + 15) / 16 * 16;         // lo, hi
  return b;
}

__host__ __device__ inline Axis axis_at(char *base, int n, int nc) {
  Axis a;
  a.n = n; a.nc = nc; a.nsp = nc - 3;
  char *p = base;
  a.s = (int *)p;    p += ((size_t)n * 4 + 15) / 16 * 16;
  a.w = (float4 *)p; p += (size_t)n * 16;
  a.p = (float *)p;  p += (size_t)n * 16;
  a.q = (float *)p;  p += (size_t)n * 16;
  a.p4 = (float4 *)p; p += (size_t)n * 16;
  a.q4 = (float4 *)p; p += (size_t)n * 16;
  a.lo = (int *)p;   a.hi = a.lo + a.nsp;
  return a;
}

// Span index of voxel i, as N4.py:210 computes it: floor((i + 0.5) / span)
// with span = n / nspans, all in IEEE FP64 (no contraction).
__device__ __forceinline__ int span_of(int i, double span, int nsp) {
  double u = __dadd_rn((double)i, 0.5);
  int s = (int)floor(__ddiv_rn(u, span));
  return s < 0 ? 0 : (s >= nsp ? nsp - 1 : s);
}

// Weights of voxel i along an axis of `nsp` spans of `span` voxels: the cubic
// weights w = B0..B3, the fit's numerator weights p = w^3 / sum w^2 and
// denominator weights q = w^2, formed in FP64.  Returns the span index.
__device__ __forceinline__ int axis_voxel(int i, double span, int nsp, float4 &w, float4 &p, float4 &q) {
  const int s = span_of(i, span, nsp);
  const double u = __dadd_rn((double)i, 0.5);
  const double t = __ddiv_rn(__dsub_rn(u, __dmul_rn((double)s, span)), span);
  const double t2 = t * t, t3 = t * t * t, tm = 1.0 - t;
  const double w0 = tm * tm * tm / 6.0;
  const double w1 = (3.0 * t3 - 6.0 * t2 + 4.0) / 6.0;
  const double w2 = (-3.0 * t3 + 3.0 * t2 + 3.0 * t + 1.0) / 6.0;
  const double w3 = t3 / 6.0;
  const double S = w0 * w0 + w1 * w1 + w2 * w2 + w3 * w3;
  w = make_float4((float)w0, (float)w1, (float)w2, (float)w3);
  p = make_float4((float)(w0 * w0 * w0 / S), (float)(w1 * w1 * w1 / S), (float)(w2 * w2 * w2 / S),
                  (float)(w3 * w3 * w3 / S));
  q = make_float4((float)(w0 * w0), (float)(w1 * w1), (float)(w2 * w2), (float)(w3 * w3));
  return s;
}

// Voxel i's part of the spans' voxel ranges: lo[sp] is the first voxel of a
// span >= sp (n if there is none) and hi[sp] = lo[sp + 1], so the voxel where
// the span index s changes writes the spans up to its own.  (A binary search
// per span took two FP64 divisions a step one after the other.)
__device__ __forceinline__ void axis_range(int i, int s, int n, int nsp, double span, int *lo, int *hi) {
  const int before = i > 0 ? span_of(i - 1, span, nsp) : -1;
  for (int sp = before + 1; sp <= s; ++sp) {
    lo[sp] = i;
    if (sp > 0) hi[sp - 1] = i;
  }
  if (i == n - 1) {
    hi[s] = n;
    for (int sp = s + 1; sp < nsp; ++sp) lo[sp] = hi[sp] = n;
  }
}

// Fill voxels first, first + step, ... of one axis table (caller synchronises).
__device__ __forceinline__ void build_axis(const Axis &a, int first, int step) {
  const double span = __ddiv_rn((double)a.n, (double)a.nsp);
  for (int i = first; i < a.n; i += step) {
    float4 w, p, q;
    const int s = axis_voxel(i, span, a.nsp, w, p, q);
    a.s[i] = s;
    a.w[i] = w;
    a.p4[i] = p;
    a.q4[i] = q;
    a.p[0 * a.n + i] = p.x; a.p[1 * a.n + i] = p.y; a.p[2 * a.n + i] = p.z; a.p[3 * a.n + i] = p.w;
    a.q[0 * a.n + i] = q.x; a.q[1 * a.n + i] = q.y; a.q[2 * a.n + i] = q.z; a.q[3 * a.n + i] = q.w;
    axis_range(i, s, a.n, a.nsp, span, a.lo, a.hi);
  }
}

// b = sum_j w_j g[j] with a fixed association (identical in every pass).
__device__ __forceinline__ float dot4(float4 w, const float *g) {
  float b = __fmul_rn(w.x, g[0]);
  b = __fmaf_rn(w.y, g[1], b);
  b = __fmaf_rn(w.z, g[2], b);
  b = __fmaf_rn(w.w, g[3], b);
  return b;
}

// GPU global timer (ns) and the SM this thread runs on.
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ int sm_id() {
  unsigned r;
  asm volatile("mov.u32 %0, %%smid;" : "=r"(r));
  return (int)r;
}

// ---------------------------------------------------------------- reductions
__device__ __forceinline__ float warp_min(float v) {
  for (int o = 16; o; o >>= 1) v = fminf(v, __shfl_xor_sync(kFull, v, o));
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
  for (int o = 16; o; o >>= 1) v = fmaxf(v, __shfl_xor_sync(kFull, v, o));
  return v;
}
__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}

// Kahan-compensated FP32 sum (Kahan, CACM 8(1), 1965): `s` is the running
// sum and `c` the part of the last addition that `s` could not hold, fed
// back into the next term.  The error of a compensated sum of n terms is
// bounded by ~2u sum|x_i| independently of n (u = 2^-24), instead of the
// ~n u sum|x_i| of a plain recursive sum.  The intrinsics keep the compiler
// from contracting or reassociating the steps.
struct KahanSum {
  float s = 0.0f, c = 0.0f;
  __device__ __forceinline__ void add(float x) {
    const float y = __fsub_rn(x, c);
    const float t = __fadd_rn(s, y);
    c = __fsub_rn(__fsub_rn(t, s), y);
    s = t;
  }
  // adds w * x (the product rounded once, inside the first step)
  __device__ __forceinline__ void add_prod(float w, float x) {
    const float y = __fmaf_rn(w, x, -c);
    const float t = __fadd_rn(s, y);
    c = __fsub_rn(__fsub_rn(t, s), y);
    s = t;
  }
  __device__ __forceinline__ float value() const { return __fsub_rn(s, c); }
  // adds another compensated sum
  __device__ __forceinline__ void merge(const KahanSum &o) { add(o.value()); }
};

// CTA-wide reduction of four values (min, max, sum, sum) into out[0..3] of
// thread 0; `scratch` holds 4 * 32 doubles.  Deterministic order.
__device__ void block_reduce4(float vmin, float vmax, double s0, double s1,
                              double *scratch, double out[4]) {
  vmin = warp_min(vmin); vmax = warp_max(vmax); s0 = warp_sum(s0); s1 = warp_sum(s1);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (lane == 0) {
    scratch[wid] = vmin; scratch[32 + wid] = vmax; scratch[64 + wid] = s0; scratch[96 + wid] = s1;
  }
  __syncthreads();
  if (wid == 0) {
    float a = lane < nw ? (float)scratch[lane] : INFINITY;
    float b = lane < nw ? (float)scratch[32 + lane] : -INFINITY;
    double c = lane < nw ? scratch[64 + lane] : 0.0;
    double d = lane < nw ? scratch[96 + lane] : 0.0;
    a = warp_min(a); b = warp_max(b); c = warp_sum(c); d = warp_sum(d);
    if (lane == 0) { out[0] = a; out[1] = b; out[2] = c; out[3] = d; }
  }
  __syncthreads();
}

// ---------------------------------------------------------------- FFT (FP64)
// The sharpening map is computed in double precision: N4 accumulates the
// residual logU - E(logU), a small difference of O(1) values, so a relative
// error of 1e-6 in E moves the fitted lattice by ~2e-4 after a few dozen
// iterations.  The map is O(bins) work per iteration; every volume-sized
// quantity stays in FP32.
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 mul_mi(double2 a) { return make_double2(a.y, -a.x); }  // a * (-i)

__device__ __forceinline__ void dft2(double2 *v) {
  double2 a = v[0], b = v[1];
  v[0] = cadd(a, b); v[1] = csub(a, b);
}
__device__ __forceinline__ void dft4(double2 &v0, double2 &v1, double2 &v2, double2 &v3) {
  double2 t0 = cadd(v0, v2), t1 = csub(v0, v2), t2 = cadd(v1, v3), t3 = mul_mi(csub(v1, v3));
  v0 = cadd(t0, t2); v2 = csub(t0, t2); v1 = cadd(t1, t3); v3 = csub(t1, t3);
}
// FFT buffers keep value i at sw(i): a radix-4 pass stores every fourth value,
// which in order would lie in two of the eight 16-byte banks.
__device__ __forceinline__ int sw(int i) { return i ^ ((i >> 3) & 7); }

// Twiddles exp(-2 pi i m / N): m in [0, N) in order, or, for N = 512, the passes'
// own sequences one after the other, so that a warp's loads are consecutive
// (in the table of all m a pass's stride put eight of them into one bank: 410
// cycles per pass): radix-4 passes of Ns = 4, 16, 64 at 0, 12 and 60 as
// [r - 1][k], the radix-2 pass of Ns = 256 at 252.
__device__ void fft_twiddles(double2 *tw, int N) {
  for (int t = threadIdx.x; t < N; t += blockDim.x) {
    int m = t;
    if (N == 512) {
      const int Ns = t < 12 ? 4 : (t < 60 ? 16 : (t < 252 ? 64 : 256)), u = t - (t < 12 ? 0 : (t < 60 ? 12 : (t < 252 ? 60 : 252)));
      if (Ns == 256) m = u & 255;
      else m = (u / Ns + 1) * (u % Ns) * (N / (Ns * 4));
    }
    double s, c;
    sincospi(-2.0 * (double)m / (double)N, &s, &c);
    tw[t] = make_double2(c, s);
  }
}

template <int R> __device__ __forceinline__ void dft_r(double2 *v);
template <> __device__ __forceinline__ void dft_r<2>(double2 *v) { dft2(v); }
template <> __device__ __forceinline__ void dft_r<4>(double2 *v) { dft4(v[0], v[1], v[2], v[3]); }

// One Stockham pass of radix R (Govindaraju et al., SC'08, "High performance
// discrete Fourier transforms on graphics processors"): in(0..N) -> y, with
// twiddle(r, k) for r in [1, R), k in [0, Ns).  The input is a function, so that
// an elementwise step before an FFT can be part of its first pass (Ns = 1, where
// every twiddle is 1).
template <int R, class In, class Tw>
__device__ __forceinline__ void stockham_pass(const In &in, double2 *y, int N, int Ns, const Tw &twiddle) {
  const int T = N / R;
  for (int j = threadIdx.x; j < T; j += blockDim.x) {
    const int k = j & (Ns - 1);
    double2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      v[r] = in(j + r * T);
      if (r && Ns > 1) v[r] = cmul(v[r], twiddle(r, k));
    }
    dft_r<R>(v);
    const int base = (j - k) * R + k;
#pragma unroll
    for (int r = 0; r < R; ++r) y[sw(base + r * Ns)] = v[r];
  }
  __syncthreads();
}

// Forward FFT (length N = 2^m, 4 <= N <= 4096) of in(0..N): radix 4, the last
// pass radix 2 where N is no power of 4; the first pass goes to a, the others
// ping-pong a and b, each ending with a CTA barrier.  Returns the buffer that
// holds the result (value i at sw(i)).  NC: N where it is known at compile time
// (512, up to 256 bins: the passes' strides become constants), else 0.
// (Three radix-8 passes of 64 threads round differently, and N4 on a small
// volume follows every bit; the last two passes in one of 64 threads, the
// values in registers between them, took as long as the two.)
template <int NC, class In>
__device__ __forceinline__ double2 *fft_from(const In &in, double2 *a, double2 *b, int N, const double2 *tw) {
  auto from = [](const double2 *x) { return [x](int i) { return x[sw(i)]; }; };
  if constexpr (NC == 512) {
    auto packed = [tw](int at, int Ns) { return [=](int r, int k) { return tw[at + (r - 1) * Ns + k]; }; };
    stockham_pass<4>(in, a, 512, 1, packed(0, 1));
    stockham_pass<4>(from(a), b, 512, 4, packed(0, 4));
    stockham_pass<4>(from(b), a, 512, 16, packed(12, 16));
    stockham_pass<4>(from(a), b, 512, 64, packed(60, 64));
    stockham_pass<2>(from(b), a, 512, 256, packed(252, 256));
    return a;
  } else {
    auto plain = [=](int step) { return [=](int r, int k) { return tw[(r * k * step) & (N - 1)]; }; };
    const int R0 = N % 4 == 0 ? 4 : 2;
    if (R0 == 4) stockham_pass<4>(in, a, N, 1, plain(0));
    else stockham_pass<2>(in, a, N, 1, plain(0));
    for (int Ns = R0, rem = N / R0; rem > 1;) {
      const int R = rem % 4 == 0 ? 4 : 2;
      if (R == 4) stockham_pass<4>(from(a), b, N, Ns, plain(N / (Ns * 4)));
      else stockham_pass<2>(from(a), b, N, Ns, plain(N / (Ns * 2)));
      double2 *t = a; a = b; b = t;
      Ns *= R;
      rem /= R;
    }
    return a;
  }
}

// ---------------------------------------------------------------- sharpening
struct SharpenBufs {
  double2 *a, *b;    // [N] work buffers
  double2 *tw;       // [N] twiddles (filled by the caller once)
  double *Ff;        // [N/2 + 1] the Gaussian, then its real Fourier transform
};

// The Gaussian's height and exponent per squared bin for a bin width `slope`.
struct Gauss {
  double scale, exponent;
};
__device__ __forceinline__ Gauss gauss_of(double slope, double fwhm) {
  const double ln2 = 0.69314718055994530942;
  const double scaledFWHM = fwhm / slope;
  return Gauss{2.0 * sqrt(ln2 / 3.14159265358979323846) / scaledFWHM, 4.0 * ln2 / (scaledFWHM * scaledFWHM)};
}

// E[0..bins) from the fractional histogram (bin b's weight hv(b)) (N4.py:32-101,
// cudaN4.cu:733-817), all in FP64; all threads of the CTA call it.  Four FFTs.
// The steps with an exponential or a division go over all threads of the CTA,
// one value each, and use the symmetry of real inputs (index k stands for
// N - k too): inside an FFT's first pass, on its N/4 threads, four of them
// would follow one another in every thread.  R2 (optional): the residual table
// of residual_lin, R2[b] for b < bins - 1.
template <int NC, class HistF>
__device__ __forceinline__ void sharpen_map_n(const HistF &hv, int bins, int N, int off, double binMin, double slope,
                                              double wiener, const Gauss &ga, const SharpenBufs &sb, double *E,
                                              float2 *R2) {
  const double invN = 1.0 / (double)N;
  // the periodic Gaussian's N/2 + 1 distinct values, held in sb.Ff until the
  // transform takes their place
  for (int d = threadIdx.x; d <= N / 2; d += blockDim.x)
    sb.Ff[d] = ga.scale * exp(-(double)d * (double)d * ga.exponent);
  __syncthreads();
  // z = V + i F : the padded histogram and the periodic Gaussian in one FFT
  double2 *Z = fft_from<NC>(
      [&](int i) {
        const double F = sb.Ff[i <= N / 2 ? i : N - i];
        const double V = (i >= off && i < off + bins) ? hv(i - off) : 0.0;
        return make_double2(V, F);
      },
      sb.a, sb.b, N, sb.tw);
  double2 *W = (Z == sb.a) ? sb.b : sb.a;
  // split the packed transform; Wiener filter Re(conj(Ff)/(|Ff|^2 + w)) with
  // Ff real; conj(Uf), so that the forward FFT inverts
  for (int k = threadIdx.x; k <= N / 2; k += blockDim.x) {
    const int kn = (N - k) & (N - 1);
    const double2 zk = Z[sw(k)], zn = Z[sw(kn)];
    const double2 Vf = make_double2(0.5 * (zk.x + zn.x), 0.5 * (zk.y - zn.y));
    const double Ff = 0.5 * (zk.y + zn.y);
    const double g = Ff / (Ff * Ff + wiener);
    sb.Ff[k] = Ff;
    W[sw(kn)] = make_double2(Vf.x * g, Vf.y * g);
    W[sw(k)] = make_double2(Vf.x * g, -Vf.y * g);
  }
  __syncthreads();
  double2 *Y = fft_from<NC>([&](int k) { return W[sw(k)]; }, Z, W, N, sb.tw);
  double2 *Y2 = (Y == W) ? Z : W;
  // U = max(Re(ifft(Uf)), 0); pack the numerator c_i U_i (real) and U (imaginary)
  double2 *P = fft_from<NC>(
      [&](int i) {
        const double U = fmax(Y[sw(i)].x * invN, 0.0);
        const double c = binMin + (double)(i - off) * slope;
        return make_double2(c * U, U);
      },
      Y2, Y, N, sb.tw);
  double2 *P2 = (P == Y2) ? Y : Y2;
  // Gaussian smoothing of both: multiply by the (real) Ff, inverse transform
  double2 *S = fft_from<NC>(
      [&](int k) {
        const double2 v = P[sw(k)];
        const double f = sb.Ff[k <= N / 2 ? k : N - k];
        return make_double2(v.x * f, -v.y * f);
      },
      P2, P, N, sb.tw);
  for (int b = threadIdx.x; b < bins; b += blockDim.x) {
    const double2 v = S[sw(off + b)];
    const double nu = v.x * invN, de = -v.y * invN;
    E[b] = (de != 0.0) ? nu / de : 0.0;
  }
  __syncthreads();
  if (R2) {
    for (int b = threadIdx.x; b + 1 < bins; b += blockDim.x) {
      const double e = E[b];
      R2[b] = make_float2((float)(binMin + (double)b * slope - e), (float)(slope - (E[b + 1] - e)));
    }
    __syncthreads();
  }
}

template <class HistF>
__device__ __forceinline__ void sharpen_map(const HistF &hv, int bins, int N, int off, double binMin, double slope,
                                            double wiener, const Gauss &ga, const SharpenBufs &sb, double *E,
                                            float2 *R2 = nullptr) {
  if (N == 512) sharpen_map_n<512>(hv, bins, 512, off, binMin, slope, wiener, ga, sb, E, R2);
  else sharpen_map_n<0>(hv, bins, N, off, binMin, slope, wiener, ga, sb, E, R2);
}

// Float-float arithmetic (a value as the unevaluated sum of two floats, ~48
// significant bits): Knuth's TwoSum and the FMA form of Dekker's TwoProduct
// are error-free, so x - binMin and products keep their rounding errors
// exactly.  The _rn intrinsics keep the compiler from contracting or
// reassociating these sequences.
__device__ __forceinline__ float two_sum(float a, float b, float &err) {
  const float s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  err = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
  return s;
}

// Bin coordinate of a value, (x - binMin) / slope, in FP64.  The reciprocal
// product is within an ulp of the quotient; near the last bin the quotient
// itself is taken, because there one ulp decides whether the reference
// counts or drops the maximum voxel (N4.py:27).
//
// coord_split (below) gives the same coordinate from float-float arithmetic
// as a bin k and a fraction f (|error| < 2^-24, the resolution of the
// histogram's fixed point): d = x - binMin exactly by TwoSum (binMin is the
// minimum of FP32 values, a float), times 1/slope held as a float-float.  It
// declines values within two bins of the top, which take the FP64 path.
struct BinMap {
  double binMin, slope, inv_slope, top;
  float fmin, ih, il, ff_limit;
  BinMap() = default;
  __device__ BinMap(double mn, double sl, int bins)
      : binMin(mn), slope(sl), inv_slope(1.0 / sl), top((double)bins - 1.5), fmin((float)mn),
        ih((float)inv_slope), il((float)(inv_slope - (double)ih)), ff_limit((float)(bins - 2)) {}
  __device__ __forceinline__ double coord(float x) const {
    const double d = (double)x - binMin;
    const double c = d * inv_slope;
    return c > top ? d / slope : c;
  }
};

// The same coordinate in float-float arithmetic, from the map's fields fmin,
// ih + il and ff_limit: the bin k and the fraction f of x, or false within
// two bins of the top and for a NaN (then k = 0, in range of every table, and
// f is of no use).  Branch-free, so that several voxels' chains overlap, and
// without conversions, which go at a quarter of the rate: adding 2^23 rounded
// down leaves floor(p) in the low bits.
__device__ __forceinline__ bool coord_split(float x, float fmin, float ih, float il, float limit, int &k, float &f) {
  constexpr float kMagic = 8388608.0f;   // 2^23
  float dl;
  const float dh = two_sum(x, -fmin, dl);                  // x - binMin = dh + dl exactly
  const float p = __fmul_rn(dh, ih);
  const float pe = __fmaf_rn(dh, ih, -p);                  // p + pe = dh * ih exactly
  const float cl = __fadd_rn(pe, __fmaf_rn(dh, il, __fmul_rn(dl, ih)));
  const bool in = p < limit;                               // not near the top bin (or NaN)
  const float t = __fadd_rd(p, kMagic);                    // 2^23 + floor(p), for 0 <= p < 2^22
  const float fr = __fadd_rn(__fsub_rn(p, __fsub_rn(t, kMagic)), cl);   // p - floor(p) is exact
  const float step = fr < 0.0f ? 1.0f : (fr >= 1.0f ? -1.0f : 0.0f);
  f = __fadd_rn(fr, step);
  k = in ? max(__float_as_int(__fsub_rn(t, step)) - __float_as_int(kMagic), 0) : 0;   // x >= binMin: never below 0
  return in;
}

// exp(x) - 1 of a convergence term (N4.py:121-126): for |x| < 1/4 its Taylor
// series through x^7 / 7! in Horner form, x + x^2 (1/2! + x (1/3! + ...)),
// whose truncation is below x^7 / 8! < 2^-28 relative and whose last step
// is one fused multiply-add (0.65 ulp at most against FP64 over 2^21 samples
// of the interval); expm1f beyond (first iterations of a level).
__device__ __forceinline__ float expm1_conv(float x) {
  if (fabsf(x) < 0.25f) {
    float p = __fmaf_rn(x, 1.0f / 5040.0f, 1.0f / 720.0f);
    p = __fmaf_rn(p, x, 1.0f / 120.0f);
    p = __fmaf_rn(p, x, 1.0f / 24.0f);
    p = __fmaf_rn(p, x, 1.0f / 6.0f);
    p = __fmaf_rn(p, x, 0.5f);
    return __fmaf_rn(__fmul_rn(x, x), p, x);
  }
  return expm1f(x);
}

// Fractional histogram contribution of one value (N4.py:21-29) from its
// FP64 bin coordinate, as fixed-point weights of 2^shift per voxel (the two
// parts of a split add up to exactly one voxel).  Returns the bin or -1 when
// the value adds nothing.
__device__ __forceinline__ int hist_bin(double c, int bins, double scale, unsigned &qlo, unsigned &qhi) {
  if (!(c >= 0.0) || !(c < (double)bins)) return -1;   // NaN / out of range (defensive)
  const double fc = floor(c);
  const double off = c - fc;
  const int idx = (int)fc;
  const unsigned one = (unsigned)scale;
  if (off == 0.0) { qlo = one; qhi = 0u; return idx; }
  if (idx < bins - 1) {
    qhi = (unsigned)__double2uint_rn(off * scale);
    qlo = one - qhi;
    return idx;
  }
  return -1;                                             // the reference drops it
}

// The FP64 path of a value near the top bin, out of line: inlined, the
// compiler may evaluate it for every value under a predicate.  `bm` is in
// shared memory.
__device__ __noinline__ int hist_bin_top(const BinMap *bm, float x, int bins, double scale, unsigned &qlo,
                                         unsigned &qhi) {
  return hist_bin(bm->coord(x), bins, scale, qlo, qhi);
}

// Largest shift <= 24 for which `n` voxels cannot overflow a 32-bit bin.
__host__ __device__ inline int hist_shift_for(long long n) {
  int s = kHistMaxShift;
  while (s > 0 && (unsigned long long)n << s > 0xffffffffull) --s;
  return s;
}

// Piecewise-linear remap through E (N4.py:107-113) from the FP64 bin
// coordinate c of the value.
__device__ __forceinline__ double sharpened_value(double c, const double *E, int bins) {
  const double fc = floor(c);
  int idx = (int)fc;
  if (!(c >= 0.0)) idx = 0;   // unreachable for values >= binMin; keeps the access in range
  if (idx < bins - 1) {
    const double e0 = E[idx], e1 = E[idx + 1];
    return e0 + (e1 - e0) * (c - fc);
  }
  return E[bins - 1];
}

// Residual x - E(x) of the piecewise-linear remap for a value in bin
// k < bins - 1 at fraction f.  With x = binMin + (k + f) slope and
// E(x) = E[k] + f (E[k+1] - E[k]) (N4.py:107-113) the residual is linear in f
// within a bin: x - E(x) = R2[k].x + f R2[k].y, R2[k] = (binMin + k slope -
// E[k], slope - (E[k+1] - E[k])) formed in FP64 by sharpen_map, so the
// cancellation of the O(1) terms happens in FP64.  The fraction's own error
// (~2^-24) moves the result by ~2^-24 |R2[k].y| <= 2^-24 slope.
__device__ __forceinline__ float residual_lin(int k, float f, const float2 *R2) {
  const float2 t = R2[k];
  return __fmaf_rn(f, t.y, t.x);
}

// The FP64 residual of a value near the top bin, out of line as above.  (An
// FP32 coordinate for the others, error ~2^-24 c, moved the lattice of a
// 32x32x24 volume after 2 x 4 iterations by 1.4e-4 relative, measured with
// the oracle: the bound is 1e-4.)
__device__ __noinline__ float residual_top(const BinMap *bm, float x, const double *E, int bins) {
  return (float)((double)x - sharpened_value(bm->coord(x), E, bins));
}

// Refined lattice value at output index (ox, oy, oz) (array indices), from
// the (n+3)-point lattice `L` (Lee, Wolberg, Shin 1997 section 4.2;
// cudaN4.cu:257-339 with its clamped boundary).
__device__ __forceinline__ void refine_taps(int o, int n, int idx[3], float w[3]) {
  const int oi = o - 1;                      // lattice coordinate, from -1
  const int i = (oi >= 0) ? (oi >> 1) : -1;  // floor(oi / 2) for oi >= -1
  const int par = oi - 2 * i;
  for (int k = 0; k < 3; ++k) {
    int c = i - 1 + k;
    c = c < -1 ? -1 : (c > n + 1 ? n + 1 : c);
    idx[k] = c + 1;
  }
  if (par == 0) { w[0] = 0.125f; w[1] = 0.75f; w[2] = 0.125f; }
  else          { w[0] = 0.0f;   w[1] = 0.5f;  w[2] = 0.5f; }
}

__device__ void refine_lattice(const float *L, int ncx, int ncy, int ncz, float *out) {
  const int nx = ncx - 3, ny = ncy - 3, nz = ncz - 3;
  const int mx = 2 * nx + 3, my = 2 * ny + 3, mz = 2 * nz + 3;
  for (int t = threadIdx.x; t < mx * my * mz; t += blockDim.x) {
    int oz = t % mz, oy = (t / mz) % my, ox = t / (mz * my);
    int ix[3], iy[3], iz[3];
    float wx[3], wy[3], wz[3];
    refine_taps(ox, nx, ix, wx);
    refine_taps(oy, ny, iy, wy);
    refine_taps(oz, nz, iz, wz);
    float acc = 0.0f;
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b)
#pragma unroll
        for (int c = 0; c < 3; ++c)
          acc += wx[a] * wy[b] * wz[c] * L[(ix[a] * ncy + iy[b]) * ncz + iz[c]];
    out[t] = acc;
  }
}

// ---------------------------------------------------------------- grid barrier
// Barrier over all CTAs of a cooperative launch: arrivals are counted up
// from zero, and a CTA waits until the count reaches the end of its round
// (counted by thread 0).  One release-add and one acquire-poll per CTA and
// round: the CTA's barriers on both sides extend them to its other threads,
// which read what other CTAs wrote past L1 (__ldcg).  Every wait is bounded:
// on timeout (or when another CTA already failed) it records N4_ERR_TIMEOUT in
// *err and returns false.
struct GridBarrier {
  unsigned *count;
  int *err;
  unsigned nblocks;
  unsigned target;   // arrivals at the end of this CTA's last round; starts at 0

  __device__ bool sync() {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
      target += nblocks;
      unsigned long long spins = 0;
      int ok = 1;
      for (;;) {
        unsigned c;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(count) : "memory");
        if ((int)(c - target) >= 0) break;
        ++spins;
        if ((spins & 255u) == 0 && *(volatile int *)err != 0) { ok = 0; break; }
        if (spins > kSpinLimit) { atomicExch(err, (int)N4_ERR_TIMEOUT); ok = 0; break; }
      }
      s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
  }
};

}  // namespace n4
