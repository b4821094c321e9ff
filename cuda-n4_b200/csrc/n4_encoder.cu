// Warm-start encoder: a small 3-D convolutional network that predicts the
// first-level 4x4x4 log-bias lattice of N4 from the masked log fitting grid
// average-pooled to 32x32x24.  No counterpart in the reference.
//
//   input 1x32x32x24 -> conv3x3x3/2 16 -> ReLU -> conv 32 -> ReLU -> conv 64
//   -> ReLU -> conv 64 -> ReLU -> (64x2x2x2 = 512) -> linear 64
//
// Every contraction (forward, data gradient, weight gradient) runs on the
// BF16 tensor cores through one implicit-GEMM kernel (mma.sync m16n8k16,
// FP32 accumulate) whose operand tiles are gathered from the activation
// tensors by small index functors.  Activations and weights are BF16, master
// weights, gradients and Adam moments FP32.  Weight gradients reduce over the
// batch with a fixed split-K and a deterministic second pass.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/n4b200.h"

namespace enc {

typedef __nv_bfloat16 bf16;

constexpr int kLayers = 4;
constexpr int kCh[kLayers + 1] = {1, 16, 32, 64, 64};
constexpr int kIn[3] = {32, 32, 24};
constexpr int kOut = 64;          // 4x4x4 lattice
constexpr int kFeat = 64 * 8;     // 64 channels x 2x2x2

__host__ __device__ inline int out_dim(int d) { return (d - 1) / 2 + 1; }   // k3, s2, p1

// ------------------------------------------------------------------ mma
__device__ __forceinline__ void mma_bf16(float c[4], const unsigned a[4], const unsigned b[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

constexpr int BM = 64, BN = 64, BK = 32, PAD = 8;

// Exact floor(k / d) for 0 <= k < 2^24 and 1 <= d < 2^16: with
// M = ceil(2^40 / d), k*M / 2^40 exceeds k/d by less than 2^-16 < 1/d.
struct Div {
  unsigned d;
  unsigned long long M;
  Div() : d(1), M(1ull << 40) {}
  explicit Div(unsigned dd) : d(dd), M(((1ull << 40) + dd - 1) / dd) {}
  __device__ __forceinline__ int q(int k) const { return (int)(((unsigned long long)(unsigned)k * M) >> 40); }
};

// Sixteen consecutive k of one operand row, as bf16 pairs (low half first).
struct Vals {
  unsigned v[8];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = 0u;
  }
  __device__ __forceinline__ void put(int j, bf16 x) {   // j a constant after unrolling, the word clear before
    v[j >> 1] |= (unsigned)__bfloat16_as_ushort(x) << (16 * (j & 1));
  }
  __device__ __forceinline__ void half(int h, const uint4 &q) {
    v[4 * h] = q.x; v[4 * h + 1] = q.y; v[4 * h + 2] = q.z; v[4 * h + 3] = q.w;
  }
};

// p[j], j < min(nv, 16), the others 0; `vec`: p is 16-byte aligned.
__device__ __forceinline__ void load_run(Vals &o, const bf16 *p, int nv, bool vec) {
  o.clear();
  if (vec && nv >= 16) {
    o.half(0, *(const uint4 *)p);
    o.half(1, *(const uint4 *)(p + 8));
  } else {
#pragma unroll
    for (int j = 0; j < 16; ++j)
      if (j < nv) o.put(j, p[j]);
  }
}
// p[j * stride], j < min(nv, 16).
__device__ __forceinline__ void load_strided(Vals &o, const bf16 *p, size_t stride, int nv) {
  o.clear();
#pragma unroll
  for (int j = 0; j < 16; ++j)
    if (j < nv) o.put(j, p[j * stride]);
}

// One row of a gather over the 27 taps of a 3x3x3 window: k = 27 c + t reads
// p[c * stride + tap[t]] when bit t of `mask` is set (the tap meets a voxel),
// 0 otherwise.  The window's bounds are in the mask, once per row.
struct TapRow {
  const bf16 *p;
  unsigned mask;
};
__device__ __forceinline__ void load_taps(Vals &o, const TapRow &r, const int *tap, int stride, int k, int nv) {
  o.clear();
  int c = k / 27, t = k - c * 27;
  const bf16 *q = r.p + (ptrdiff_t)c * stride;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    if (j < nv && (r.mask >> t & 1u)) o.put(j, q[tap[t]]);
    if (++t == 27) { t = 0; q += stride; }
  }
}

// C[m][n] = sum_k A(m,k) B(k,n) over this block's K range; P supplies the
// sizes, the loads of 16 consecutive k of a row (load_a, load_b; the row's
// index decomposition once per block in a_row, b_row), tap offsets of window
// gathers (tap, in shared memory) and the store.  128 threads, a 64 x NT tile
// (NT = 16, 32, 64: the smallest that holds N, so that a layer of 16 channels
// does not stage and multiply 48 columns of zeros): 4 warps of 16x16, 32x16 or
// 32x32.  A thread stages half a row of the A tile and, up to 2 NT threads,
// of the B tile; the next tile is loaded into registers while this one is
// multiplied.  The sums' order over k does not depend on the tile.
template <class P, int NT>
__global__ void __launch_bounds__(128) k_igemm(const P p) {
  __shared__ __align__(16) bf16 As[BM][BK + PAD];
  __shared__ __align__(16) bf16 Bs[NT][BK + PAD];
  __shared__ int tap[27];
  constexpr int WX = NT == 16 ? 1 : 2;             // warps along n
  constexpr int WM = BM / (4 / WX), WN = NT / WX;  // a warp's tile
  constexpr int MI = WM / 16, NJ = WN / 8;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * NT;
  const int kper = ((p.K + gridDim.z - 1) / gridDim.z + BK - 1) / BK * BK;
  const int kb = blockIdx.z * kper, ke = min(p.K, kb + kper);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, tig = lane & 3;
  const int wm = (warp / WX) * WM, wn = (warp % WX) * WN;
  const int sr = threadIdx.x >> 1, sc = (threadIdx.x & 1) * 16;   // staged row, first column
  if (threadIdx.x < 27) tap[threadIdx.x] = p.tap(threadIdx.x);
  __syncthreads();
  const bool a_ok = m0 + sr < p.M, b_ok = sr < NT && n0 + sr < p.N;
  const typename P::ARow ar = p.a_row(a_ok ? m0 + sr : 0);
  const typename P::BRow br = p.b_row(b_ok ? n0 + sr : 0);
  float acc[MI][NJ][4] = {};
  Vals va, vb;
  va.clear();
  vb.clear();
  const auto load = [&](int k0) {
    const int k = k0 + sc, nv = ke - k;
    if (a_ok && nv > 0) p.load_a(va, ar, tap, k, nv);
    else va.clear();
    if (sr < NT) {
      if (b_ok && nv > 0) p.load_b(vb, br, tap, k, nv);
      else vb.clear();
    }
  };
  if (kb < ke) load(kb);
  for (int k0 = kb; k0 < ke; k0 += BK) {
    *(uint4 *)&As[sr][sc] = make_uint4(va.v[0], va.v[1], va.v[2], va.v[3]);
    *(uint4 *)&As[sr][sc + 8] = make_uint4(va.v[4], va.v[5], va.v[6], va.v[7]);
    if (sr < NT) {
      *(uint4 *)&Bs[sr][sc] = make_uint4(vb.v[0], vb.v[1], vb.v[2], vb.v[3]);
      *(uint4 *)&Bs[sr][sc + 8] = make_uint4(vb.v[4], vb.v[5], vb.v[6], vb.v[7]);
    }
    __syncthreads();
    if (k0 + BK < ke) load(k0 + BK);
#pragma unroll
    for (int kk = 0; kk < BK; kk += 16) {
      unsigned af[MI][4], bfr[NJ][2];
#pragma unroll
      for (int i = 0; i < MI; ++i) {
        const int r = wm + 16 * i + g;
        af[i][0] = *(const unsigned *)&As[r][kk + 2 * tig];
        af[i][1] = *(const unsigned *)&As[r + 8][kk + 2 * tig];
        af[i][2] = *(const unsigned *)&As[r][kk + 2 * tig + 8];
        af[i][3] = *(const unsigned *)&As[r + 8][kk + 2 * tig + 8];
      }
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int c = wn + 8 * j + g;
        bfr[j][0] = *(const unsigned *)&Bs[c][kk + 2 * tig];
        bfr[j][1] = *(const unsigned *)&Bs[c][kk + 2 * tig + 8];
      }
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) mma_bf16(acc[i][j], af[i], bfr[j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int m = m0 + wm + 16 * i + g + (e >= 2 ? 8 : 0);
        const int n = n0 + wn + 8 * j + 2 * tig + (e & 1);
        if (m < p.M && n < p.N) p.store(m, n, blockIdx.z, acc[i][j][e]);
      }
}

// ------------------------------------------------------------------ problems
struct Shape {
  int B, Ci, D, H, W, Co, Do, Ho, Wo;
  __host__ __device__ int in_pos() const { return D * H * W; }
  __host__ __device__ int out_pos() const { return Do * Ho * Wo; }
};

// Output position decomposition (b, od, oh, ow) of a flat index.
struct PosDiv {
  Div op, hw, w;
  PosDiv() {}
  PosDiv(int out_pos, int hwo, int wo) : op(out_pos), hw(hwo), w(wo) {}
};

// y = relu(conv(x, w) + bias): M = B*outpos, N = Co, K = Ci*27
struct ConvFwd {
  int M, N, K;
  Shape s;
  const bf16 *x, *w;
  const float *bias;
  bf16 *y;
  int relu;
  using ARow = TapRow;                 // the corner of the window; taps inside the image
  struct BRow { const bf16 *wn; };
  __device__ int tap(int t) const { return (t / 9 * s.H + t / 3 % 3) * s.W + t % 3; }
  __device__ ARow a_row(int m) const {
    const int op = s.out_pos();
    const int b = m / op, r = m - b * op;
    const int id = 2 * (r / (s.Ho * s.Wo)) - 1, ih = 2 * (r / s.Wo % s.Ho) - 1, iw = 2 * (r % s.Wo) - 1;
    unsigned mask = 0;
    for (int t = 0; t < 27; ++t) {
      const int d = id + t / 9, h = ih + t / 3 % 3, w2 = iw + t % 3;
      if (d >= 0 && d < s.D && h >= 0 && h < s.H && w2 >= 0 && w2 < s.W) mask |= 1u << t;
    }
    return ARow{x + (ptrdiff_t)b * s.Ci * s.in_pos() + ((ptrdiff_t)id * s.H + ih) * s.W + iw, mask};
  }
  __device__ void load_a(Vals &o, const ARow &R, const int *tp, int k, int nv) const {
    load_taps(o, R, tp, s.in_pos(), k, nv);
  }
  __device__ BRow b_row(int n) const { return BRow{w + (size_t)n * K}; }
  __device__ void load_b(Vals &o, const BRow &R, const int *, int k, int nv) const {
    load_run(o, R.wn + k, nv, (((uintptr_t)w | (unsigned)K * 2u) & 15u) == 0);
  }
  __device__ void store(int m, int n, int, float v) const {
    const int op = s.out_pos();
    const int b = m / op, r = m - b * op;
    v += bias[n];
    if (relu) v = fmaxf(v, 0.0f);
    y[((size_t)b * s.Co + n) * op + r] = __float2bfloat16(v);
  }
};

// The gradient of a ReLU's input: g where its output `y` is positive.
__device__ __forceinline__ bf16 relu_grad(float g, bf16 y) {
  return __bfloat162float(y) <= 0.0f ? __float2bfloat16(0.0f) : __float2bfloat16(g);
}

// dx = conv_transpose(dy, w) masked by the ReLU that made x: a GEMM of the
// input positions (rows) by Ci, over K = Co*27.  Input position i meets output
// (i + 1 - kd) / 2 where that is whole: with f = floor((i + 1) / 2) it is
// f - (kd >> 1), for kd = 1 when i is even and kd = 0, 2 when it is odd.  So of
// the 27 taps of a channel only 1, 2, 4 or 8 meet an output, the same ones for
// all positions of one parity class (8 classes).
struct ConvDgrad {
  Shape s;
  const bf16 *dy, *x, *w;
  bf16 *dx;
  int first[8];   // first block of a class
  // positions of one axis with parity p, and rows of class c (parities of d,
  // h, w in bits 2, 1, 0) over the batch
  static __host__ __device__ int axis_count(int n, int p) { return (n + 1 - p) >> 1; }
  __host__ __device__ int rows(int c) const {
    return s.B * axis_count(s.D, c >> 2) * axis_count(s.H, c >> 1 & 1) * axis_count(s.W, c & 1);
  }
};

// 64 rows of one parity class by NT columns; 256 threads, 8 warps of 16 x NT/2.
// Sixteen channels are staged at a time: 432 dense columns k = 27 c + t, which
// are 27 whole K steps of 16.  A class meets the same columns of every group,
// so the others are cleared once per block, a group's loads are only those of
// the class's T taps (all in flight while the group before is multiplied), the
// fragments come by ldmatrix and nothing is synchronised between the 27 steps;
// steps without a tap are not multiplied.  Terms, their order and their
// grouping by 16 are those of the dense GEMM over all 27 taps.  The row stride
// of 440 puts the eight rows of a matrix on different banks, and a warp stages
// 8 rows of 4 channels for the same reason.  Bound by the instructions of the
// gathers (one per value) and, where a layer has few rows, by the latency of
// its groups.  The three layers of a batch of 64 take 19, 37 and 70 us; 29, 49
// and 88 us when every thread divided its rows' indices and read the taps from
// shared memory at each load, 98, 105 and 142 us when each step of 32 dense
// columns loaded its own few columns between two barriers.
constexpr int kDgCols = 432, kDgLd = kDgCols + 8;
constexpr size_t dgrad_smem(int NT) { return (size_t)(BM + NT) * kDgLd * sizeof(bf16); }

template <int T, int NT>
__device__ __forceinline__ void dgrad_rows(const ConvDgrad &p, bf16 *As, bf16 *Bs, const int *tap, int at, unsigned amask,
                                           int n0, unsigned long long period, float (&acc)[NT / 16][4]) {
  constexpr int NJ = NT / 16, PARTS = 256 / NT, NA = 4 * T, NB = 16 * T / PARTS;
  const Shape &s = p.s;
  const int op = s.out_pos(), cw = s.Ci * 27;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = lane >> 3;
  const int bn = (lane & 7) + 8 * (warp % (NT / 8)), bpart = sub + 4 * (warp / (NT / 8));
  bf16 *const ato = As + ((lane & 7) + 8 * warp) * kDgLd + 27 * sub;
  bf16 *const bto = Bs + bn * kDgLd + 27 * bpart;
  // the taps, their offsets in dy, and a bit per tap that meets an output of the row
  int tp[T], of[T];
  unsigned ok = 0;
#pragma unroll
  for (int t = 0; t < T; ++t) {
    tp[t] = tap[t];
    of[t] = -((((tp[t] / 9) >> 1) * s.Ho + ((tp[t] / 3 % 3) >> 1)) * s.Wo + ((tp[t] % 3) >> 1));
    ok |= (amask >> tp[t] & 1u) << t;
  }
  const bf16 zero = __float2bfloat16(0.0f);
  bf16 va[NA], vb[NB];
  at += sub * op;
  int wat = min(n0 + bn, s.Ci - 1) * 27 + bpart * cw;   // a column past Ci repeats the last and is not stored
  const auto load = [&]() {   // the next 16 channels
#pragma unroll
    for (int i = 0; i < NA; ++i) {
      va[i] = zero;
      if (ok & 1u << i % T) va[i] = p.dy[at + i / T * 4 * op + of[i % T]];
    }
#pragma unroll
    for (int i = 0; i < NB; ++i) vb[i] = p.w[wat + i / T * PARTS * cw + tp[i % T]];
    at += 16 * op;
    wat += 16 * cw;
  };
  const unsigned a_at = (unsigned)__cvta_generic_to_shared(As + ((warp >> 1) * 16 + (lane & 15)) * kDgLd + (lane >> 4) * 8);
  const unsigned b_at = (unsigned)__cvta_generic_to_shared(
      Bs + ((warp & 1) * (NT / 2) + (NJ == 2 ? (lane >> 4) * 8 : 0) + (lane & 7)) * kDgLd + (lane >> 3 & 1) * 8);
  load();
  for (int c0 = 0; c0 < s.Co; c0 += 16) {
    if (c0 > 0) __syncthreads();
#pragma unroll
    for (int i = 0; i < NA; ++i) ato[i / T * 4 * 27 + tp[i % T]] = va[i];
#pragma unroll
    for (int i = 0; i < NB; ++i) bto[i / T * PARTS * 27 + tp[i % T]] = vb[i];
    __syncthreads();
    if (c0 + 16 < s.Co) load();
#pragma unroll
    for (int k = 0; k < 27; ++k) {
      if (!((unsigned)(period >> (16 * k % 27)) & 0xffffu)) continue;
      unsigned af[4], bfr[2 * NJ];
      asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                   : "=r"(af[0]), "=r"(af[1]), "=r"(af[2]), "=r"(af[3]) : "r"(a_at + 32 * k) : "memory");
      if constexpr (NJ == 2)
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(bfr[0]), "=r"(bfr[1]), "=r"(bfr[2]), "=r"(bfr[3]) : "r"(b_at + 32 * k) : "memory");
      else
        asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];"
                     : "=r"(bfr[0]), "=r"(bfr[1]) : "r"(b_at + 32 * k) : "memory");
#pragma unroll
      for (int j = 0; j < NJ; ++j) mma_bf16(acc[j], af, bfr + 2 * j);
    }
  }
}

template <int NT>
__global__ void __launch_bounds__(256) k_dgrad(const ConvDgrad p) {
  constexpr int NJ = NT / 16;
  extern __shared__ __align__(16) bf16 stage[];
  bf16 *As = stage, *Bs = stage + BM * kDgLd;
  __shared__ int tap[8];                    // the class's taps, ascending
  __shared__ int row_dy[BM], row_dx[BM];    // a row's element of channel 0 in dy and dx (-1: no row)
  __shared__ unsigned row_taps[BM];         // the taps that meet an output of it
  const Shape &s = p.s;
  int cls = 0, first = 0;
#pragma unroll
  for (int c = 1; c < 8; ++c)
    if ((int)blockIdx.x >= p.first[c]) cls = c, first = p.first[c];
  const int row0 = ((int)blockIdx.x - first) * BM, n0 = blockIdx.y * NT;
  const int pd = cls >> 2, ph = cls >> 1 & 1, pw = cls & 1;
  const int ip = s.in_pos();
  // a bit per tap (kd, kh, kw) from the axes' bits, and two periods of the class's
  const auto taps = [](unsigned md, unsigned mh, unsigned mw) {
    return mw * ((mh & 1u) | (mh & 2u) << 2 | (mh & 4u) << 4) * ((md & 1u) | (md & 2u) << 8 | (md & 4u) << 16);
  };
  const unsigned cmask = taps(pd ? 5u : 2u, ph ? 5u : 2u, pw ? 5u : 2u);
  const unsigned long long period = cmask | (unsigned long long)cmask << 27;
  if (threadIdx.x < 27 && (cmask >> threadIdx.x & 1u)) tap[__popc(cmask & ((1u << threadIdx.x) - 1u))] = threadIdx.x;
  if (threadIdx.x >= 64 && threadIdx.x < 64 + BM) {
    const int r = threadIdx.x - 64, q = row0 + r;
    const int nd = ConvDgrad::axis_count(s.D, pd), nh = ConvDgrad::axis_count(s.H, ph), nw = ConvDgrad::axis_count(s.W, pw);
    const int qh = q / nw, qd = qh / nh, b = qd / nd;
    const int jw = q - qh * nw, jh = qh - qd * nh, jd = qd - b * nd;
    const int fd = jd + pd, fh = jh + ph, fw = jw + pw;
    const auto axis = [](int par, int f, int n) { return par ? (f < n ? 5u : 4u) : 2u; };
    const bool in = b < s.B;
    row_taps[r] = in ? taps(axis(pd, fd, s.Do), axis(ph, fh, s.Ho), axis(pw, fw, s.Wo)) : 0u;
    row_dy[r] = b * s.Co * s.out_pos() + (fd * s.Ho + fh) * s.Wo + fw;
    row_dx[r] = in ? b * s.Ci * ip + ((2 * jd + pd) * s.H + 2 * jh + ph) * s.W + 2 * jw + pw : -1;
  }
  for (int i = threadIdx.x; i < (BM + NT) * kDgLd / 8; i += 256) ((uint4 *)stage)[i] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  float acc[NJ][4] = {};
  const int mine = (threadIdx.x & 7) + 8 * (threadIdx.x >> 5), at = row_dy[mine];
  const unsigned amask = row_taps[mine];
  switch (__popc(cmask)) {
    case 8: dgrad_rows<8, NT>(p, As, Bs, tap, at, amask, n0, period, acc); break;
    case 4: dgrad_rows<4, NT>(p, As, Bs, tap, at, amask, n0, period, acc); break;
    case 2: dgrad_rows<2, NT>(p, As, Bs, tap, at, amask, n0, period, acc); break;
    default: dgrad_rows<1, NT>(p, As, Bs, tap, at, amask, n0, period, acc); break;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, tig = lane & 3;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int dx0 = row_dx[(warp >> 1) * 16 + g + 8 * h];
    if (dx0 < 0) continue;
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int n = n0 + (warp & 1) * (NT / 2) + 8 * j + 2 * tig + e;
        if (n >= s.Ci) continue;
        const int o = dx0 + n * ip;
        p.dx[o] = relu_grad(acc[j][2 * h + e], p.x[o]);
      }
  }
}

// dw partials, and the bias gradient as one more column of ones: M = Co,
// N = Ci*27 + 1, K = B*outpos (split over blockIdx.z)
struct ConvWgrad {
  int M, N, K;
  Shape s;
  const bf16 *x, *dy;
  float *part;   // [splits][Co][Ci*27 + 1]
  PosDiv pd;     // decomposition of a position index k into (b, od, oh, ow)
  struct ARow { int m; };
  struct BRow { int ci, kd, kh, kw; };   // ci = Ci: the column of ones
  __device__ int tap(int) const { return 0; }
  __device__ ARow a_row(int m) const { return ARow{m}; }
  // an image's positions are a multiple of 8 (checked where the layers are
  // laid out), so each half of a run lies in one image
  __device__ void load_a(Vals &o, const ARow &R, const int *, int k, int nv) const {
    const int op = s.out_pos();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int kk = k + 8 * h;
      uint4 q = make_uint4(0u, 0u, 0u, 0u);
      if (8 * h < nv) {
        const int b = pd.op.q(kk);
        q = *(const uint4 *)(dy + ((size_t)b * s.Co + R.m) * op + (kk - b * op));
      }
      o.half(h, q);
    }
  }
  __device__ BRow b_row(int n) const {
    const int ci = n / 27, t = n - ci * 27;
    return BRow{ci, t / 9 - 1, (t / 3) % 3 - 1, t % 3 - 1};
  }
  __device__ void load_b(Vals &o, const BRow &R, const int *, int k, int nv) const {
    o.clear();
    if (R.ci == s.Ci) {
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (j < nv) o.put(j, __float2bfloat16(1.0f));
      return;
    }
    const int op = s.out_pos();
    const int b = pd.op.q(k), r = k - b * op;
    int od = pd.hw.q(r);
    const int r2 = r - od * s.Ho * s.Wo;
    int oh = pd.w.q(r2), ow = r2 - oh * s.Wo;
    const bf16 *img = x + ((size_t)b * s.Ci + R.ci) * s.in_pos();
    const bf16 *row = img + ((2 * od + R.kd) * s.H + 2 * oh + R.kh) * s.W + R.kw;
    bool in = (unsigned)(2 * od + R.kd) < (unsigned)s.D && (unsigned)(2 * oh + R.kh) < (unsigned)s.H;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      if (j < nv && in && (unsigned)(2 * ow + R.kw) < (unsigned)s.W) o.put(j, row[2 * ow]);
      if (++ow == s.Wo) {
        ow = 0;
        if (++oh == s.Ho) {
          oh = 0;
          if (++od == s.Do) { od = 0; img += (size_t)s.Ci * s.in_pos(); }
        }
        row = img + ((2 * od + R.kd) * s.H + 2 * oh + R.kh) * s.W + R.kw;
        in = (unsigned)(2 * od + R.kd) < (unsigned)s.D && (unsigned)(2 * oh + R.kh) < (unsigned)s.H;
      }
    }
  }
  __device__ void store(int m, int n, int z, float v) const { part[((size_t)z * M + m) * N + n] = v; }
};

// linear y = x W^T + bias: M = B, N = out, K = in
struct LinFwd {
  int M, N, K;
  const bf16 *x, *w;
  const float *bias;
  float *y;
  struct ARow { const bf16 *r; };
  struct BRow { const bf16 *r; };
  __device__ int tap(int) const { return 0; }
  __device__ ARow a_row(int m) const { return ARow{x + (size_t)m * K}; }
  __device__ void load_a(Vals &o, const ARow &R, const int *, int k, int nv) const {
    load_run(o, R.r + k, nv, (((uintptr_t)x | (unsigned)K * 2u) & 15u) == 0);
  }
  __device__ BRow b_row(int n) const { return BRow{w + (size_t)n * K}; }
  __device__ void load_b(Vals &o, const BRow &R, const int *, int k, int nv) const {
    load_run(o, R.r + k, nv, (((uintptr_t)w | (unsigned)K * 2u) & 15u) == 0);
  }
  __device__ void store(int m, int n, int, float v) const { y[(size_t)m * N + n] = v + bias[n]; }
};
// dx = dy W masked by the ReLU that made x: M = B, N = in, K = out
struct LinDgrad {
  int M, N, K;
  const bf16 *dy, *x, *w;
  bf16 *dx;
  struct ARow { const bf16 *r; };
  struct BRow { int n; };
  __device__ int tap(int) const { return 0; }
  __device__ ARow a_row(int m) const { return ARow{dy + (size_t)m * K}; }
  __device__ void load_a(Vals &o, const ARow &R, const int *, int k, int nv) const {
    load_run(o, R.r + k, nv, (((uintptr_t)dy | (unsigned)K * 2u) & 15u) == 0);
  }
  __device__ BRow b_row(int n) const { return BRow{n}; }
  __device__ void load_b(Vals &o, const BRow &R, const int *, int k, int nv) const {
    load_strided(o, w + (size_t)k * N + R.n, N, nv);
  }
  __device__ void store(int m, int n, int, float v) const {
    const size_t i = (size_t)m * N + n;
    dx[i] = relu_grad(v, x[i]);
  }
};
// dW = dy^T x, and the bias gradient as one more column of ones: M = out,
// N = in + 1, K = B
struct LinWgrad {
  int M, N, K;
  const bf16 *dy, *x;
  float *part;
  struct ARow { int m; };
  struct BRow { int n; };
  __device__ int tap(int) const { return 0; }
  __device__ ARow a_row(int m) const { return ARow{m}; }
  __device__ void load_a(Vals &o, const ARow &R, const int *, int k, int nv) const {
    load_strided(o, dy + (size_t)k * M + R.m, M, nv);
  }
  __device__ BRow b_row(int n) const { return BRow{n}; }
  __device__ void load_b(Vals &o, const BRow &R, const int *, int k, int nv) const {
    if (R.n < N - 1) {
      load_strided(o, x + (size_t)k * (N - 1) + R.n, N - 1, nv);
    } else {
      o.clear();
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (j < nv) o.put(j, __float2bfloat16(1.0f));
    }
  }
  __device__ void store(int m, int n, int z, float v) const { part[((size_t)z * M + m) * N + n] = v; }
};

// ------------------------------------------------------------------ small kernels
// Weight and bias gradients from the partials of [M][N] sums, the last column
// the bias: one warp per 32 entries, its lanes of a block's 8 warps taking every
// eighth split in order, the eight sums added in order.
__global__ void __launch_bounds__(256) k_sum_splits(const float *part, int splits, int M, int N, float *dw, float *db) {
  __shared__ float red[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n = M * N;
  for (int i0 = blockIdx.x * 32; i0 < n; i0 += gridDim.x * 32) {
    const int i = i0 + lane;
    float s = 0.0f;
    if (i < n)
      for (int z = warp; z < splits; z += 8) s += part[(size_t)z * n + i];
    red[warp][lane] = s;
    __syncthreads();
    if (warp == 0 && i < n) {
#pragma unroll
      for (int w = 1; w < 8; ++w) s += red[w][lane];
      const int m = i / N, c = i - m * N;
      if (c < N - 1) dw[(size_t)m * (N - 1) + c] = s;
      else db[m] = s;
    }
    __syncthreads();
  }
}

// A forward GEMM split over K: each block stores its partial sums (the
// wrapper's store), then k_finish adds the splits in order and applies the
// layer's own store (bias, ReLU, BF16 for the convolutions).  The forward's
// small layers (conv3, conv4, the linear head: 1 to 6 blocks of 64x64) would
// otherwise walk 16-54 K steps in one block each.
template <class P>
struct Partial : P {
  float *part;   // [splits][M][N]
  __device__ void store(int m, int n, int z, float v) const { part[((size_t)z * this->M + m) * this->N + n] = v; }
};

template <class P>
__global__ void k_finish(const P p, const float *part, int splits) {
  const long long mn = (long long)p.M * p.N;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < mn; i += (long long)gridDim.x * blockDim.x) {
    float s = 0.0f;
    for (int z = 0; z < splits; ++z) s += part[z * mn + i];
    p.store((int)(i / p.N), (int)(i % p.N), 0, s);
  }
}

// loss = mean((y - t)^2); dy = 2 (y - t) / n (bf16); one block
__global__ void k_mse(const float *y, const float *t, int n, float *loss, bf16 *dy) {
  float s = 0.0f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const float d = y[i] - t[i];
    s += d * d;
    dy[i] = __float2bfloat16(2.0f * d / (float)n);
  }
  __shared__ float red[32];
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float u = 0.0f;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) u += red[w];
    *loss = u / (float)n;
  }
}

__global__ void k_adam(float *p, const float *gr, float *m, float *v, int n, float lr, float b1, float b2, float eps,
                       float c1, float c2, bf16 *pb) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float g = gr[i];
    const float mi = b1 * m[i] + (1.0f - b1) * g;
    const float vi = b2 * v[i] + (1.0f - b2) * g * g;
    m[i] = mi;
    v[i] = vi;
    const float w = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    p[i] = w;
    pb[i] = __float2bfloat16(w);
  }
}

__global__ void k_to_bf16(const float *a, int n, bf16 *b) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) b[i] = __float2bfloat16(a[i]);
}

// ------------------------------------------------------------------ host side
template <class P>
cudaError_t run_gemm(const P &p, int splits, cudaStream_t st) {
  const int mb = (p.M + BM - 1) / BM;
  if (p.N <= 16) k_igemm<P, 16><<<dim3(mb, 1, splits), 128, 0, st>>>(p);
  // 32 columns also where 64-column tiles would leave most SMs without a block
  else if (p.N <= 32 || (long long)mb * ((p.N + 63) / 64) * splits < 128)
    k_igemm<P, 32><<<dim3(mb, (p.N + 31) / 32, splits), 128, 0, st>>>(p);
  else k_igemm<P, 64><<<dim3(mb, (p.N + 63) / 64, splits), 128, 0, st>>>(p);
  return cudaGetLastError();
}

template <int NT>
cudaError_t run_dgrad_nt(const ConvDgrad &p, int tiles, cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(k_dgrad<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dgrad_smem(NT));
  if (e != cudaSuccess) return e;
  k_dgrad<NT><<<dim3(tiles, (p.s.Ci + NT - 1) / NT), 256, dgrad_smem(NT), st>>>(p);
  return cudaGetLastError();
}
// whole groups of channels, and 32-bit element offsets at every batch size
static_assert(kCh[2] % 16 == 0 && kCh[3] % 16 == 0 && kCh[4] % 16 == 0 &&
              4096ll * 16 * 16 * 16 * 12 < (1ll << 31), "k_dgrad");
inline cudaError_t run_dgrad(ConvDgrad p, cudaStream_t st) {
  int tiles = 0;
  for (int c = 0; c < 8; ++c) {
    p.first[c] = tiles;
    tiles += (p.rows(c) + BM - 1) / BM;
  }
  return p.s.Ci <= 16 ? run_dgrad_nt<16>(p, tiles, st) : run_dgrad_nt<32>(p, tiles, st);
}

// Splits of a forward GEMM: enough blocks for about two per SM, at least two
// K steps per split, within the partials buffer (cap floats).
inline int fwd_splits(int M, int N, int K, size_t cap) {
  const long long tiles = (long long)((M + BM - 1) / BM) * ((N + BN - 1) / BN);
  const int steps = (K + BK - 1) / BK;
  long long s = std::max<long long>(1, 296 / tiles);
  s = std::min<long long>(s, std::max(1, steps / 2));
  while (s > 1 && (size_t)s * M * N > cap) --s;
  return (int)s;
}

// A forward layer: one pass, or split over K into `part` and finished in order.
template <class P>
cudaError_t run_forward(const P &p, float *part, size_t cap, cudaStream_t st) {
  const int splits = fwd_splits(p.M, p.N, p.K, cap);
  if (splits == 1) return run_gemm(p, 1, st);
  Partial<P> q;
  static_cast<P &>(q) = p;
  q.part = part;
  cudaError_t e = run_gemm(q, splits, st);
  if (e != cudaSuccess) return e;
  const long long mn = (long long)p.M * p.N;
  k_finish<P><<<(int)std::min<long long>((mn + 255) / 256, 1024), 256, 0, st>>>(p, part, splits);
  return cudaGetLastError();
}

struct Layout {
  // parameter offsets (floats) in the flat parameter vector
  size_t w[kLayers + 1], b[kLayers + 1], total;
  Shape s[kLayers];
  Layout(int B) {
    int d = kIn[0], h = kIn[1], wd = kIn[2];
    size_t o = 0;
    for (int l = 0; l < kLayers; ++l) {
      s[l] = Shape{B, kCh[l], d, h, wd, kCh[l + 1], out_dim(d), out_dim(h), out_dim(wd)};
      w[l] = o; o += (size_t)kCh[l + 1] * kCh[l] * 27;
      b[l] = o; o += kCh[l + 1];
      d = out_dim(d); h = out_dim(h); wd = out_dim(wd);
    }
    static_assert(kIn[0] % 32 == 0 && kIn[1] % 32 == 0 && kIn[2] % 24 == 0,
                  "every layer's output positions are a multiple of 8 (ConvWgrad)");
    w[kLayers] = o; o += (size_t)kOut * kFeat;
    b[kLayers] = o; o += kOut;
    total = o;
  }
};

}  // namespace enc

using namespace enc;

struct n4_encoder {
  int device = 0;
  int max_batch = 0;
  size_t nparam = 0;
  float *p = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;   // FP32 master, grad, moments
  bf16 *pb = nullptr;                                             // BF16 weights
  bf16 *act[kLayers + 1] = {};                                    // activations (act[0] = input copy)
  bf16 *dact_[kLayers + 1] = {};                                  // activation gradients
  float *out = nullptr, *tgt = nullptr, *loss = nullptr;
  bf16 *dout = nullptr;
  float *part = nullptr;
  size_t part_cap = 0;
  long long step = 0;
};

// records the message returned by n4_last_error_string (n4_api.cu)
n4_status_t n4_record_error(n4_status_t s, const char *msg);

// largest batch one n4_encoder_predict call takes (used by n4_api.cu)
int n4_encoder_capacity(const n4_encoder_t *enc) { return enc ? enc->max_batch : 0; }

// kernels one n4_encoder_predict call of batch B launches (used by n4_api.cu):
// a GEMM per layer and the head, and a finishing pass for each split one
int n4_encoder_predict_launches(const n4_encoder_t *enc, int B) {
  if (!enc || B < 1) return 0;
  const enc::Layout L(B);
  int n = enc::kLayers + 1;
  for (int l = 0; l < enc::kLayers; ++l)
    n += enc::fwd_splits(B * L.s[l].out_pos(), L.s[l].Co, L.s[l].Ci * 27, enc->part_cap) > 1 ? 1 : 0;
  n += enc::fwd_splits(B, enc::kOut, enc::kFeat, enc->part_cap) > 1 ? 1 : 0;
  return n;
}

namespace {
n4_status_t efail(n4_status_t s, const std::string &m) { return n4_record_error(s, m.c_str()); }
#define ECK(x)                                                                              \
  do {                                                                                      \
    cudaError_t e_ = (x);                                                                   \
    if (e_ != cudaSuccess) { cudaGetLastError(); return efail(N4_ERR_CUDA, std::string(#x) + ": " + cudaGetErrorString(e_)); } \
  } while (0)
// Splits of a weight gradient's sum over K positions: about four blocks per SM
// (592) of at least four K steps each.
int wgrad_splits(int M, int N, long long K) {
  const long long tiles = (long long)((M + BM - 1) / BM) * ((N + BN - 1) / BN);
  return (int)std::max<long long>(1, std::min<long long>(592 / tiles, K / (4 * BK)));
}
}  // namespace

extern "C" {

size_t n4_encoder_num_params(void) { return Layout(1).total; }

n4_status_t n4_encoder_create(n4_encoder_t **out, int device, int max_batch) {
  if (!out || max_batch < 1 || max_batch > 4096) return efail(N4_ERR_INVALID_ARG, "bad arguments");
  *out = nullptr;
  ECK(cudaSetDevice(device));
  n4_encoder *e = new n4_encoder();
  e->device = device;
  e->max_batch = max_batch;
  Layout L(max_batch);
  e->nparam = L.total;
  size_t n = L.total;
  auto fail_free = [&](cudaError_t err) {
    n4_encoder_destroy(e);
    return efail(err == cudaErrorMemoryAllocation ? N4_ERR_OOM : N4_ERR_CUDA, cudaGetErrorString(err));
  };
  cudaError_t err;
  if ((err = cudaMalloc(&e->p, n * 4)) || (err = cudaMalloc(&e->g, n * 4)) || (err = cudaMalloc(&e->m, n * 4)) ||
      (err = cudaMalloc(&e->v, n * 4)) || (err = cudaMalloc(&e->pb, n * 2)))
    return fail_free(err);
  cudaMemset(e->m, 0, n * 4);
  cudaMemset(e->v, 0, n * 4);
  cudaMemset(e->p, 0, n * 4);
  cudaMemset(e->pb, 0, n * 2);
  for (int l = 0; l <= kLayers; ++l) {
    const size_t sz = l == 0 ? (size_t)max_batch * L.s[0].in_pos() : (size_t)max_batch * L.s[l - 1].Co * L.s[l - 1].out_pos();
    if ((err = cudaMalloc(&e->act[l], sz * 2))) return fail_free(err);
    if (l > 0 && (err = cudaMalloc(&e->dact_[l], sz * 2))) return fail_free(err);   // the input has no gradient
  }
  if ((err = cudaMalloc(&e->out, (size_t)max_batch * kOut * 4)) || (err = cudaMalloc(&e->tgt, (size_t)max_batch * kOut * 4)) ||
      (err = cudaMalloc(&e->loss, 16)) || (err = cudaMalloc(&e->dout, (size_t)max_batch * kOut * 2)))
    return fail_free(err);
  // split-K partials: the largest weight gradient times the splits
  size_t need = 0;
  for (int l = 0; l < kLayers; ++l) {
    const int M = L.s[l].Co, N = L.s[l].Ci * 27 + 1;
    need = std::max(need, (size_t)wgrad_splits(M, N, (long long)max_batch * L.s[l].out_pos()) * M * N);
  }
  need = std::max(need, (size_t)wgrad_splits(kOut, kFeat + 1, max_batch) * kOut * (kFeat + 1));
  // and the forward's split layers at every batch size up to max_batch
  const size_t unbounded = ~(size_t)0;
  for (int b = 1; b <= max_batch; ++b) {
    const Layout Lb(b);
    for (int l = 0; l < kLayers; ++l) {
      const int M = b * Lb.s[l].out_pos(), N = Lb.s[l].Co;
      need = std::max(need, (size_t)fwd_splits(M, N, Lb.s[l].Ci * 27, unbounded) * M * N);
    }
    need = std::max(need, (size_t)fwd_splits(b, kOut, kFeat, unbounded) * b * kOut);
  }
  if ((err = cudaMalloc(&e->part, need * 4))) return fail_free(err);
  e->part_cap = need;
  *out = e;
  return N4_OK;
}

n4_status_t n4_encoder_destroy(n4_encoder_t *e) {
  if (!e) return N4_OK;
  cudaSetDevice(e->device);
  cudaDeviceSynchronize();
  for (void *q : {(void *)e->p, (void *)e->g, (void *)e->m, (void *)e->v, (void *)e->pb, (void *)e->out, (void *)e->tgt,
                  (void *)e->loss, (void *)e->dout, (void *)e->part})
    if (q) cudaFree(q);
  for (int l = 0; l <= kLayers; ++l) {
    if (e->act[l]) cudaFree(e->act[l]);
    if (e->dact_[l]) cudaFree(e->dact_[l]);
  }
  delete e;
  return N4_OK;
}

n4_status_t n4_encoder_set_params(n4_encoder_t *e, const float *h_params, size_t n) {
  if (!e || !h_params || n != e->nparam) return efail(N4_ERR_INVALID_ARG, "parameter count mismatch");
  ECK(cudaSetDevice(e->device));
  ECK(cudaMemcpy(e->p, h_params, n * 4, cudaMemcpyHostToDevice));
  ECK(cudaMemset(e->m, 0, n * 4));
  ECK(cudaMemset(e->v, 0, n * 4));
  k_to_bf16<<<256, 256>>>(e->p, (int)n, e->pb);
  ECK(cudaGetLastError());
  e->step = 0;
  ECK(cudaDeviceSynchronize());
  return N4_OK;
}

n4_status_t n4_encoder_get_params(n4_encoder_t *e, float *h_params, float *h_grads, size_t n) {
  if (!e || n != e->nparam) return efail(N4_ERR_INVALID_ARG, "parameter count mismatch");
  ECK(cudaSetDevice(e->device));
  ECK(cudaDeviceSynchronize());
  if (h_params) ECK(cudaMemcpy(h_params, e->p, n * 4, cudaMemcpyDeviceToHost));
  if (h_grads) ECK(cudaMemcpy(h_grads, e->g, n * 4, cudaMemcpyDeviceToHost));
  return N4_OK;
}

static n4_status_t forward(n4_encoder *e, const void *d_x, int B, cudaStream_t st) {
  Layout L(B);
  ECK(cudaMemcpyAsync(e->act[0], d_x, (size_t)B * L.s[0].in_pos() * 2, cudaMemcpyDeviceToDevice, st));
  for (int l = 0; l < kLayers; ++l) {
    const Shape &s = L.s[l];
    ConvFwd p{B * s.out_pos(), s.Co, s.Ci * 27, s, e->act[l], e->pb + L.w[l], e->p + L.b[l], e->act[l + 1], 1};
    ECK(run_forward(p, e->part, e->part_cap, st));
  }
  LinFwd lf{B, kOut, kFeat, e->act[kLayers], e->pb + L.w[kLayers], e->p + L.b[kLayers], e->out};
  ECK(run_forward(lf, e->part, e->part_cap, st));
  return N4_OK;
}

n4_status_t n4_encoder_predict(n4_encoder_t *e, const void *d_x, int B, float *d_out, void *stream) {
  if (!e || !d_x || !d_out || B < 1 || B > e->max_batch) return efail(N4_ERR_INVALID_ARG, "bad arguments");
  cudaStream_t st = (cudaStream_t)stream;
  ECK(cudaSetDevice(e->device));
  n4_status_t s = forward(e, d_x, B, st);
  if (s != N4_OK) return s;
  ECK(cudaMemcpyAsync(d_out, e->out, (size_t)B * kOut * 4, cudaMemcpyDeviceToDevice, st));
  return N4_OK;
}

// Forward + backward on one batch; gradients in the encoder; optionally an
// Adam step (lr > 0).  *h_loss (nullable) receives the batch MSE.
n4_status_t n4_encoder_train_step(n4_encoder_t *e, const void *d_x, const float *d_target, int B, float lr,
                                  float *h_loss, void *stream) {
  if (!e || !d_x || !d_target || B < 1 || B > e->max_batch) return efail(N4_ERR_INVALID_ARG, "bad arguments");
  cudaStream_t st = (cudaStream_t)stream;
  ECK(cudaSetDevice(e->device));
  n4_status_t s = forward(e, d_x, B, st);
  if (s != N4_OK) return s;
  Layout L(B);
  k_mse<<<1, 1024, 0, st>>>(e->out, d_target, B * kOut, e->loss, e->dout);
  ECK(cudaGetLastError());
  // linear head
  {
    const int N = kFeat + 1, splits = wgrad_splits(kOut, N, B);
    LinWgrad wg{kOut, N, B, e->dout, e->act[kLayers], e->part};
    ECK(run_gemm(wg, splits, st));
    k_sum_splits<<<(kOut * N + 31) / 32, 256, 0, st>>>(e->part, splits, kOut, N, e->g + L.w[kLayers], e->g + L.b[kLayers]);
    LinDgrad dg{B, kFeat, kOut, e->dout, e->act[kLayers], e->pb + L.w[kLayers], e->dact_[kLayers]};
    ECK(run_gemm(dg, 1, st));
  }
  for (int l = kLayers - 1; l >= 0; --l) {
    const Shape &sh = L.s[l];
    const long long K = (long long)B * sh.out_pos();
    const int N = sh.Ci * 27 + 1, splits = wgrad_splits(sh.Co, N, K);
    ConvWgrad wg{sh.Co, N, (int)K, sh, e->act[l], e->dact_[l + 1], e->part, PosDiv(sh.out_pos(), sh.Ho * sh.Wo, sh.Wo)};
    ECK(run_gemm(wg, splits, st));
    k_sum_splits<<<(sh.Co * N + 31) / 32, 256, 0, st>>>(e->part, splits, sh.Co, N, e->g + L.w[l], e->g + L.b[l]);
    if (l > 0) {
      ECK(run_dgrad(ConvDgrad{sh, e->dact_[l + 1], e->act[l], e->pb + L.w[l], e->dact_[l]}, st));
    }
  }
  ECK(cudaGetLastError());
  if (lr > 0.0f) {
    ++e->step;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.0f - powf(b1, (float)e->step), c2 = 1.0f - powf(b2, (float)e->step);
    k_adam<<<256, 256, 0, st>>>(e->p, e->g, e->m, e->v, (int)e->nparam, lr, b1, b2, 1e-8f, c1, c2, e->pb);
    ECK(cudaGetLastError());
  }
  if (h_loss) {
    ECK(cudaMemcpyAsync(h_loss, e->loss, 4, cudaMemcpyDeviceToHost, st));
    ECK(cudaStreamSynchronize(st));
  }
  return N4_OK;
}

// Network input for one volume: [32][32][24] BF16 written to d_x.
}  // extern "C"
