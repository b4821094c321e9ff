// The N4 iteration for one volume, executed by a group of CTAs that share
// the volume's rows (cudaN4.cu:1418-1747, N4.py:276-332).
//
// A group is either a thread-block cluster (the volume lives in the
// cluster's distributed shared memory; partials are exchanged through DSMEM;
// hardware cluster barriers) or the whole grid of a cooperative launch (the
// masked part of the volume lives in the SMs' shared memory as far as it
// fits, the rest in global memory/L2; partials are exchanged by integer
// atomics in global memory; a bounded software barrier).  The algorithm below
// is written once for both.
//
// Per level, with L the control lattice, D its last update and Gd = rows(D)
// the per-row partial evaluation of D (x/y contracted, one value per z
// control point), the slab holds logU, one float per fitting voxel:
//   reset   logU = im_log - eval(rows(L))    (level start, warm-start trial)
//   pass A  logU -= eval(Gd): the previous update applied, its convergence
//           value, masked min/max of logU                   (group reduce)
//   pass B  fractional histogram of logU                        (group reduce)
//           Wiener sharpening map E (every CTA, in shared memory)
//   pass C  residual R = logU - remap(logU)
//   fit     separable contraction of R with the fit weights     (group reduce)
//   update  D = num / (den + eps), L += D, Gd = rows(D)
// logU follows L by the same updates, applied per voxel: eval is linear, so
// logU = im_log - eval(rows(L)) up to FP32 rounding, which the reset at every
// level start clears.
//
// Rows.  A row of the fitting grid is kept as the range [z0, z1) from its
// first to its last masked voxel; a CTA works on the list of its rows that
// have one (an ellipsoid mask leaves 36 % of the rows out and fills 60 % of
// the others).  2^sg lanes share a row; in the passes that follow the
// lattice's spans along z, a lane takes one span of the row or, with fewer
// spans than lanes, a part of it, so that a row's voxels are taken a few per
// lane instead of one after the other in one thread: an equal piece (pass A on
// the cluster path), or every 2^szh-th voxel (whole-GPU path, whose rows are
// long and may lie in global memory).
#pragma once
#include <cooperative_groups.h>
#include <new>

#include "n4_device.cuh"

namespace cg = cooperative_groups;

namespace n4 {

#define kNaN __int_as_float(0x7fc00000)

// Work of one row in the whole-GPU path's partition: its voxels and what it
// costs beside them (its entries of the row tables, its share of the y
// contraction).  Half a row of voxels: with an eighth the CTAs of the short
// rows at the volume's ends took 66k cycles for the contractions of an
// iteration where the others took 49k (512x512x320 at half resolution, 148
// CTAs: 162k cycles an iteration with Z/8, 154k with Z/4 and Z/2, when pass A
// took pieces of rows; 142k with Z/2 now; 181x217x181: 128k, 124k and 121k).
// The floor keeps a CTA of many short rows within the
// row buffers (grid_rows_bound).
__host__ __device__ inline int grid_row_overhead(int Z) { return Z / 2 > 16 ? Z / 2 : 16; }
// Most rows, and most voxels, the partition gives one of K CTAs.
__host__ __device__ inline long long grid_rows_bound(long long rows, int Z, int K) {
  const int c = grid_row_overhead(Z);
  return (rows * (Z + c) / K + Z + c) / (1 + c) + 2;
}
__host__ __device__ inline long long grid_voxels_bound(long long rows, int Z, int K) {
  const int c = grid_row_overhead(Z);
  return rows * (Z + c) / K + 2ll * (Z + c);
}
// log2 of the lanes that share a row outside the span passes (the histogram)
__host__ __device__ inline int row_lanes_log2(int Z) { return Z <= 64 ? 3 : (Z <= 256 ? 4 : 5); }

// ------------------------------------------------------------------ layout
// One axis of the fitting grid at one level, in the CTA's dynamic shared
// memory: byte offsets of the span index and the weights of every voxel
// (B0..B3, the fit's numerator weights w^3 / sum w^2 and denominator weights
// w^2) and of the spans' voxel ranges.  The z contraction's lanes step over
// several voxels at once and read weights up to 7 entries past the row's last
// voxel, for terms that are zero: `tail` zero entries after the last table keep
// those reads in memory that has been written (zero times a NaN left there by
// an earlier kernel is a NaN).
struct EAxis {
  int n, nc, nsp;
  int o_s, o_w, o_p, o_q, o_tail, o_lo, o_hi;
};
constexpr int kWeightTail = 8;   // of the z axis
__host__ __device__ inline size_t eaxis_bytes(int n, int nsp, int tail = 0) {
  return ((size_t)n * 4 + 15) / 16 * 16 + (size_t)n * 48 + (size_t)tail * 16 + ((size_t)nsp * 8 + 15) / 16 * 16;
}
__host__ __device__ inline EAxis eaxis_at(int off, int n, int nc, int tail = 0) {
  EAxis a;
  a.n = n; a.nc = nc; a.nsp = nc - 3;
  a.o_w = off;
  a.o_p = a.o_w + n * 16;
  a.o_q = a.o_p + n * 16;
  a.o_tail = a.o_q + n * 16;
  a.o_s = a.o_tail + tail * 16;
  a.o_lo = a.o_s + (n * 4 + 15) / 16 * 16;
  a.o_hi = a.o_lo + a.nsp * 4;
  return a;
}

// Byte offsets of one CTA's workspace: "o_" offsets in dynamic shared memory;
// "b_" offsets in dynamic shared memory behind sm_bytes (cluster path) or in
// a per-CTA slice of global memory (whole-GPU path).
struct Plan {
  int whole_rows;      // cluster path without row lists
  // limits
  int levels, nc0x, nc0y, nc0z, NCX, NCY, NCZ, NLAT;
  int Xmax, Ymax, Zmax, slab_floats, rows_max, nvxl;
  int bins, npad, hoff;
  // shared
  int o_ax, o_ay, o_az, o_L, o_D, o_den, o_tmp, o_aux, o_H64, o_R2, o_E;
  int o_tw, o_red, o_rows, o_ytab;
  // whole-GPU path: the shared homes of Gd (also the FFT's), of T2 and of the
  // row list and slab, used as far as a volume fits them
  int o_gd, gd_bytes, o_t2, t2_bytes, o_pool, pool_bytes;
  int sm_bytes;
  // big
  int b_imlog, b_Gd, b_T2, b_ytab, b_rows, b_slotA, b_slotB, b_slotC, big_bytes;
  // the FFT work buffers, the histogram copies and the Gaussian's transform
  // (which the sharpening writes after the copies are merged, over them) live
  // in the Gd region, dead from the end of pass A until the fit, at these offsets
  int a_fa, a_fb, a_hist, a_ff;
};

// The whole-GPU path adds the CTAs' parts of a lattice sum as integers: one
// word, whose unit is 2^-60 of a bound on the level's sums (sum_shift).  That
// is an absolute unit, nothing beside FitEpsilon's default; without an epsilon
// of that size (or with N4_FLAG_FIT_ZERO_DEN) a control point that few voxels
// reach is the quotient of two sums far below the largest, and each part takes
// kSumWords words, each of 2^-40 of the unit before it: 120 bits more, every
// digit of a float at any size.  With one word such a lattice was 3e-5 off the
// FP64 oracle where sums of floats are 1e-6 off.
constexpr int kSumWords = 4;
constexpr double kSumWordUnit = 1.0 / 1099511627776.0;   // 2^-40
inline int sum_words(float eps, int zero_den) { return zero_den || eps < 1e-3f ? kSumWords : 1; }

struct Params {
  int bins;
  double wiener, fwhm, thr;   // decimal values of the float parameters
  float eps;
  int zero_den, ddof1;
  int sum_words;              // whole-GPU path: words of a lattice sum (kSumWords)
  int iters[N4_MAX_LEVELS];
};

struct VolJob {
  int X, Y, Z;                  // fitting-resolution dimensions
  const float *imlog;           // [X*Y*Z] log intensity, NaN outside the mask
  const float *warm;            // first-level lattice or nullptr
  float *lattice_out;           // final lattice
  n4_report_t *report;
};

// Statistics exchanged after pass A: min, max, sum y, sum y^2.
struct Stats { double v[4]; };

// What the passes of one iteration need from the statistics, in the CTA's
// shared memory (o_red, after 144 words of reduction scratch).
struct Iter {
  double st[4];     // group min, max, sum y, sum y^2
  BinMap bm;
  double scale;     // 2^hshift
  Gauss gauss;
  int degenerate;   // no bin range: nothing to fit
  float cv;
  float rmax;       // whole-GPU path: bound on the residuals of the map
};
static_assert(sizeof(Iter) <= (160 - 144) * 8, "Iter lies in the o_red words behind the scratch");

// ------------------------------------------------------------------ groups
// kListed: the CTA's rows are listed in shared memory; else it works on all rows
// of its planes from end to end (volumes of short rows whose list would not fit,
// where the caller asks for the cluster path).
template <bool kListed>
struct ClusterGroup {
  __device__ int rank() const { return (int)cg::this_cluster().block_rank(); }
  __device__ int size() const { return (int)cg::this_cluster().num_blocks(); }
  __device__ bool sync() const { cg::this_cluster().sync(); return true; }
  template <class T> __device__ const T *peer(const T *p, int r) const {
    return cg::this_cluster().map_shared_rank(const_cast<T *>(p), r);
  }
  static constexpr bool kGrid = false, kRowList = kListed;
};

// Accumulators of the whole-GPU path in global memory, zero at launch: three
// sets used in turn (one is cleared while the next is in use), each `len`
// words for the range, the histogram or the lattice sums (word k of entry c at
// k NLAT + c), the last word a count of partials that are not numbers.
struct GridGroup {
  GridBarrier bar;
  char *big_base;      // per-CTA big regions, stride big_stride
  size_t big_stride;
  unsigned long long *acc;   // [3][len]
  int len;
  unsigned *ext;       // [X*Y] row ranges z0 | z1 << 16 (0: no masked voxel)
  __device__ int rank() const { return (int)blockIdx.x; }
  __device__ int size() const { return (int)gridDim.x; }
  __device__ bool sync() { return bar.sync(); }
  template <class T> __device__ const T *peer(const T *p, int r) const {
    const char *mine = big_base + (size_t)blockIdx.x * big_stride;
    return (const T *)(big_base + (size_t)r * big_stride + ((const char *)p - mine));
  }
  static constexpr bool kGrid = true, kRowList = true;
};

// ------------------------------------------------------------------ phase timers
// Compile with -DN4_PHASE_TIMERS to print, per volume, the cycles thread 0 of
// the first and of the middle CTA spends between phase marks (measurement
// builds only).  The counters live in shared memory, so that the timed build
// allocates the kernel's registers as the product build does.
#ifdef N4_PHASE_TIMERS
#define N4_MARK(k)                                                     \
  do {                                                                 \
    if (threadIdx.x == 0) {                                            \
      const long long t_ = clock64();                                  \
      ph_acc[k] += t_ - ph_acc[PH_N];                                  \
      ph_acc[PH_N] = t_;                                               \
    }                                                                  \
  } while (0)
#else
#define N4_MARK(k) do { } while (0)
#endif
enum { PH_SETUP, PH_A, PH_SHARP, PH_UPDATE, PH_A_LOOP, PH_A_RED, PH_B_LOOP, PH_B_MERGE,
       PH_B_RED, PH_F_T1, PH_F_T2, PH_F_P, PH_F_RED, PH_N };
#ifdef N4_PHASE_TIMERS
__shared__ long long ph_acc[PH_N + 1];   // per-phase cycles, then the last mark
#endif

// ------------------------------------------------------------------ engine
// The Engine's fields are uniform over the CTA.  Whole-GPU path: one object
// per CTA in shared memory (EngineSlot), its fields written by thread 0 only
// (construction, run, set_level, each followed by a barrier); held in
// registers, the fields stay live through every pass and push the voxel loops
// into local-memory spills.  Cluster path: one object per thread, every thread
// writing its own copy (a shared object made the loops reload fields after
// every shared-memory store or atomic).
template <class Group>
struct Engine {
  static constexpr bool kShared = Group::kGrid;   // the object lives in shared memory
  // the threads that write the fields, and the barrier that publishes them
  __device__ __forceinline__ bool writer() const { return !kShared || threadIdx.x == 0; }
  __device__ __forceinline__ void publish() const { if (kShared) __syncthreads(); }
  Group g;
  const Plan &pl;
  const Params &pr;
  char *big;           // whole-GPU path: this CTA's slice of global memory
  // volume
  int X, Y, Z, rank, K;
  int nact;            // rows of this CTA with a masked voxel
  int vx0, np;         // its x-planes: cluster, vx = rank + m * K; whole-GPU path, vx = vx0 + m; m < np
  int hshift;          // fixed-point scale of this volume's histogram
  int seq;             // whole-GPU path: group sums so far
  double nfg;          // masked voxels of the volume
  float denmax;        // whole-GPU path: the level's largest fit denominator
  const float *src;    // the job's log volume (global memory), read by reset
  // level
  int ncx, ncy, ncz, nlat;
  int sg, sh;          // pass A: log2 of the lanes per row and per span of it
  int sz, szh;         // z contraction: the same
  int tp;              // x-planes T2 holds at a time
  EAxis ax, ay, az;
  // whole-GPU path: where the volume's buffers are (shared memory or the slice)
  float *gdp, *t2p, *slab_g;
  int *ytabp;
  int4 *rowsp;
  int slab_off, slab_cap;

  __device__ Engine(const Group &g_, const Plan &p, const Params &r, char *big_) : g(g_), pl(p), pr(r), big(big_) {
    seq = 0;
  }

  // ---- memory
  static __device__ __forceinline__ char *dyn() {
    extern __shared__ __align__(128) char smem[];
    return smem;
  }
  template <class T> static __device__ __forceinline__ T *at(int off) { return (T *)(dyn() + off); }
  __device__ __forceinline__ float *L() const { return at<float>(pl.o_L); }
  __device__ __forceinline__ float *D() const { return at<float>(pl.o_D); }
  __device__ __forceinline__ float *den() const { return at<float>(pl.o_den); }
  __device__ __forceinline__ float *tmp() const { return at<float>(pl.o_tmp); }
  __device__ __forceinline__ float *aux() const { return at<float>(pl.o_aux); }
  __device__ __forceinline__ double *red() const { return at<double>(pl.o_red); }
  __device__ __forceinline__ Iter &iter() const { return *at<Iter>(pl.o_red + 144 * 8); }
  __device__ __forceinline__ double *E() const { return at<double>(pl.o_E); }
  __device__ __forceinline__ float2 *R2() const { return at<float2>(pl.o_R2); }
  __device__ __forceinline__ unsigned long long *H64() const { return at<unsigned long long>(pl.o_H64); }
  __device__ __forceinline__ int alias0() const { return Group::kGrid ? pl.o_gd : pl.sm_bytes + pl.b_Gd; }
  __device__ __forceinline__ unsigned *hist() const { return at<unsigned>(alias0() + pl.a_hist); }
  __device__ __forceinline__ float *Gd() const {
    if constexpr (Group::kGrid) return gdp;
    else return at<float>(pl.sm_bytes + pl.b_Gd);
  }
  __device__ __forceinline__ float *T2() const {
    if constexpr (Group::kGrid) return t2p;
    else return at<float>(pl.sm_bytes + pl.b_T2);
  }
  __device__ __forceinline__ int *ytab() const {
    if constexpr (Group::kGrid) return ytabp;
    else return at<int>(pl.o_ytab);
  }
  __device__ __forceinline__ Stats *slotA() const {
    if constexpr (Group::kGrid) return (Stats *)(big + pl.b_slotA);
    else return at<Stats>(pl.sm_bytes + pl.b_slotA);
  }
  __device__ __forceinline__ unsigned long long *slotB() const {
    if constexpr (Group::kGrid) return (unsigned long long *)(big + pl.b_slotB);
    else return at<unsigned long long>(pl.sm_bytes + pl.b_slotB);
  }
  __device__ __forceinline__ float *slotC() const { return at<float>(pl.sm_bytes + pl.b_slotC); }   // cluster path

  // ---- rows.  Row r of the CTA: its voxels [z0, z1), voxel z at p[z]; its
  // plane m and y.  A pass takes the row map by value before its loops: read
  // through the Engine, its fields would be loaded again after every store.
  struct Row {
    int z0, z1, m, vy;
    float *p;
  };
  struct ClusterRows {
    int rows, slab, Y, Z;   // byte offsets of the list and of the slab
    __device__ __forceinline__ Row operator()(int r) const {
      const uint2 d = at<uint2>(rows)[r];
      Row o;
      o.z0 = (int)(d.x & 0xffffu); o.z1 = (int)(d.x >> 16);
      o.m = (int)(d.y >> 16); o.vy = (int)(d.y & 0xffffu);
      o.p = at<float>(slab) + (o.m * Y + o.vy) * Z;
      return o;
    }
    __device__ __forceinline__ int vy(int r) const { return (int)(at<uint2>(rows)[r].y & 0xffffu); }
  };
  struct WholeRows {
    int slab, Y, Z;         // byte offset of the slab
    __device__ __forceinline__ Row operator()(int r) const {
      Row o;
      o.z0 = 0; o.z1 = Z; o.m = r / Y; o.vy = r - o.m * Y;
      o.p = at<float>(slab) + r * Z;
      return o;
    }
    __device__ __forceinline__ int vy(int r) const { return r % Y; }
  };
  struct GridRows {
    const int4 *rows;
    int slab, cap;          // byte offset of the shared slab, its floats
    float *slab_g;          // where rows beyond it are
    __device__ __forceinline__ Row operator()(int r) const {
      const int4 d = rows[r];
      Row o;
      o.z0 = d.y & 0xffff; o.z1 = (int)((unsigned)d.y >> 16); o.m = d.z; o.vy = d.w;
      o.p = (d.x + o.z1 <= cap ? at<float>(slab) : slab_g) + d.x;
      return o;
    }
    __device__ __forceinline__ int vy(int r) const { return rows[r].w; }
  };
  __device__ __forceinline__ auto row_map() const {
    if constexpr (Group::kGrid) return GridRows{rowsp, slab_off, slab_cap, slab_g};
    else if constexpr (Group::kRowList) return ClusterRows{pl.o_rows, pl.sm_bytes + pl.b_imlog, Y, Z};
    else return WholeRows{pl.sm_bytes + pl.b_imlog, Y, Z};
  }
  __device__ __forceinline__ int plane_vx(int m) const { return Group::kGrid ? vx0 + m : rank + m * K; }
  __device__ __forceinline__ const float *src_row(const Row &r) const {
    return src + ((size_t)plane_vx(r.m) * Y + r.vy) * Z;
  }

  // The part of row `r` that lane (sp, h) takes in a span pass: its span's
  // voxels inside the row's range, cut into 2^sh equal pieces.
  static __device__ __forceinline__ void piece(const Row &r, int lo, int hi, int h, int sh, int &a, int &b) {
    a = max(lo, r.z0);
    b = min(hi, r.z1);
    const int c = (b - a + (1 << sh) - 1) >> sh;   // <= 0 when the span misses the row
    a += h * c;
    b = min(b, a + c);
  }

  // ---- level geometry
  __device__ void set_level(int level) {
    if (writer()) {
      ncx = ((pl.nc0x - 3) << level) + 3;
      ncy = ((pl.nc0y - 3) << level) + 3;
      ncz = ((pl.nc0z - 3) << level) + 3;
      nlat = ncx * ncy * ncz;
      ax = eaxis_at(pl.o_ax, X, ncx);
      ay = eaxis_at(pl.o_ay, Y, ncy);
      az = eaxis_at(pl.o_az, Z, ncz, kWeightTail);
      // lanes per row: 8, or enough for one per span (16 or 32 lanes of a
      // 160-voxel row hold too little each: the z contraction at 512x512x320
      // in equal pieces took 68k and 109k cycles per iteration against 48k)
      sg = 3;
      while (sg < 5 && (1 << sg) < az.nsp) ++sg;
      sh = 0;
      while (sh < sg && (az.nsp << (sh + 1)) <= (1 << sg)) ++sh;
      // z contraction: the whole-GPU path's long rows the same way; on the
      // cluster path a lane takes a whole span
      sz = sg;
      szh = sh;
      if constexpr (!Group::kGrid) {
        sz = szh = 0;
        while (sz < 5 && (1 << sz) < az.nsp) ++sz;
      }
      if constexpr (Group::kGrid) {
        const int slice = ncy * ncz;
        tp = pl.t2_bytes / 4 / slice;
        t2p = at<float>(pl.o_t2);
        ytabp = at<int>(pl.o_ytab);
        if (tp < 1) {
          tp = pl.nvxl;
          t2p = (float *)(big + pl.b_T2);
          ytabp = (int *)(big + pl.b_ytab);
        }
      } else {
        tp = max(np, 1);
      }
    }
    publish();
    // all three axes in one sweep: a voxel's weights are a chain of FP64
    // divisions, one per thread
    for (int t = threadIdx.x; t < X + Y + Z; t += blockDim.x) {
      if (t < X) build_voxel(ax, t);
      else if (t < X + Y) build_voxel(ay, t - X);
      else build_voxel(az, t - X - Y);
    }
    if (threadIdx.x < kWeightTail) at<float4>(az.o_tail)[threadIdx.x] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    __syncthreads();
    if constexpr (Group::kRowList)
      if (np <= tp) build_ytab(0, np);
    __syncthreads();
  }

  static __device__ __forceinline__ void build_voxel(const EAxis &a, int i) {
    const double span = __ddiv_rn((double)a.n, (double)a.nsp);
    float4 w, p, q;
    const int s = axis_voxel(i, span, a.nsp, w, p, q);
    at<int>(a.o_s)[i] = s;
    at<float4>(a.o_w)[i] = w;
    at<float4>(a.o_p)[i] = p;
    at<float4>(a.o_q)[i] = q;
    axis_range(i, s, a.n, a.nsp, span, at<int>(a.o_lo), at<int>(a.o_hi));
  }

  // ytab[m][sp]: first row of the CTA's list at or after the first voxel of
  // y-span sp in plane m0 + m (sp = nspy: after the plane), so that a span's
  // rows of a plane are ytab[m][sp] .. ytab[m][sp + 1] - 1.
  __device__ void build_ytab(int m0, int cnt) {
    const int w = ay.nsp + 1;
    const auto rm = row_map();
    for (int t = threadIdx.x; t < cnt * w; t += blockDim.x) {
      const int m = m0 + t / w, sp = t % w;
      const int vy = sp < ay.nsp ? at<int>(ay.o_lo)[sp] : Y;
      int lo = 0, hi = nact;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        const Row r = rm(mid);
        if (r.m > m || (r.m == m && r.vy >= vy)) hi = mid;
        else lo = mid + 1;
      }
      ytab()[t] = lo;
    }
  }

  // ---- rows(lat) -> Gd: x/y contraction of the lattice for every row of the list
  __device__ __forceinline__ int ncz_log2() const { return 32 - __clz(max(ncz - 1, 1)); }
  __device__ void rowtab(const float *lat) {
    const int lsh = ncz_log2();
    float *Gt = Gd();
    const auto rm = row_map();
    for (int t = threadIdx.x; t < (nact << lsh); t += blockDim.x) {
      const int r = t >> lsh, cz = t & ((1 << lsh) - 1);
      if (cz >= ncz) continue;
      const Row o = rm(r);
      const int vx = plane_vx(o.m);
      const int sx = at<int>(ax.o_s)[vx], sy = at<int>(ay.o_s)[o.vy];
      const float4 wx = at<float4>(ax.o_w)[vx], wy = at<float4>(ay.o_w)[o.vy];
      const float wxa[4] = {wx.x, wx.y, wx.z, wx.w};
      const float wya[4] = {wy.x, wy.y, wy.z, wy.w};
      float acc = 0.0f;
#pragma unroll
      for (int jx = 0; jx < 4; ++jx) {
        const float *lp = lat + ((sx + jx) * ncy + sy) * ncz + cz;
        float s = 0.0f;
#pragma unroll
        for (int jy = 0; jy < 4; ++jy) s = __fmaf_rn(wya[jy], lp[jy * ncz], s);
        acc = __fmaf_rn(wxa[jx], s, acc);
      }
      Gt[r * ncz + cz] = acc;
    }
  }

  // rowtab(lat) after a lattice update, through the x-contracted planes:
  // per local x-plane, X[cy][cz] = sum_jx wx lat[sx+jx][cy][cz] (into aux,
  // free outside the warm-start trial), then per row Gd[cz] = sum_jy wy
  // X[sy+jy][cz]: 8 loads and multiply-adds per entry instead of 32.  Falls
  // back to rowtab when the planes' slices do not fit in a lattice-sized
  // buffer.  The caller synchronises.
  __device__ void rowtab_planes(const float *lat) {
    const int slice = ncy * ncz;
    if ((long long)np * slice > pl.NLAT) { rowtab(lat); return; }
    float *Xp = aux();
    for (int t = threadIdx.x; t < np * slice; t += blockDim.x) {
      const int m = t / slice, c = t - m * slice;
      const int vx = plane_vx(m);
      const float4 wx = at<float4>(ax.o_w)[vx];
      const float *pa = lat + at<int>(ax.o_s)[vx] * slice + c;
      float a = __fmul_rn(wx.x, pa[0]);
      a = __fmaf_rn(wx.y, pa[slice], a);
      a = __fmaf_rn(wx.z, pa[2 * slice], a);
      Xp[t] = __fmaf_rn(wx.w, pa[3 * slice], a);
    }
    __syncthreads();
    const int lsh = ncz_log2(), nc = ncz, n = nact << lsh, cz = threadIdx.x & ((1 << lsh) - 1);
    float *Gt = Gd();
    const auto rm = row_map();
    const float4 *W = at<float4>(ay.o_w);
    const int *S = at<int>(ay.o_s);
    if (cz < nc) {   // blockDim is a multiple of 2^lsh: a thread keeps its cz
      for (int t = threadIdx.x; t < n; t += blockDim.x) {
        const int r = t >> lsh;
        const Row o = rm(r);
        const float4 wy = W[o.vy];
        const float *xa = Xp + o.m * slice + S[o.vy] * nc + cz;
        float a = __fmul_rn(wy.x, xa[0]);
        a = __fmaf_rn(wy.y, xa[nc], a);
        a = __fmaf_rn(wy.z, xa[2 * nc], a);
        Gt[r * nc + cz] = __fmaf_rn(wy.w, xa[3 * nc], a);
      }
    }
  }

  // Calls body(row, its index, a, b, sp) for every (row, span) piece of this
  // lane.  Rows go to warps in list order; with more spans than lanes the
  // spans are taken in rounds.
  template <class Body>
  __device__ __forceinline__ void span_pass(Body &&body) const {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int sh_ = sh, l = lane & ((1 << sg) - 1), sub = lane >> sg, rs = 5 - sg, n = nact, nsp = az.nsp;
    const int per = (1 << sg) >> sh_;   // spans per round
    const auto rm = row_map();
    const int *Lo = at<int>(az.o_lo), *Hi = at<int>(az.o_hi);
    for (int sp0 = 0; sp0 < nsp; sp0 += per) {
      const int sp = sp0 + (l >> sh_), h = l & ((1 << sh_) - 1);
      const bool on = sp < nsp;
      const int lo = on ? Lo[sp] : 0, hi = on ? Hi[sp] : 0;
      for (int r = (warp << rs) + sub; r < n; r += nw << rs) {
        const Row o = rm(r);
        int a, b;
        piece(o, lo, hi, h, sh_, a, b);
        body(o, r, a, b, sp);
      }
    }
  }

  // logU = im_log - eval(rows(lat)) for every voxel of the rows, im_log read
  // from the slab itself when `staged` (the cluster kernel's bulk copy of the
  // volume, before the first reset), else from the job's log volume in
  // global memory; rows(lat) goes through the Gd region (free at every
  // reset: level start, warm-start trial).
  __device__ void reset(const float *lat, bool staged = false) {
    rowtab(lat);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int s = row_lanes_log2(Z), l = lane & ((1 << s) - 1), sub = lane >> s, rs = 5 - s, n = nact, nc = ncz;
    const auto rm = row_map();
    const float *Gp = Gd();
    const float4 *W = at<float4>(az.o_w);
    const int *S = at<int>(az.o_s);
    for (int r = (warp << rs) + sub; r < n; r += nw << rs) {
      const Row o = rm(r);
      const float *im = staged ? o.p : src_row(o);
      const float *g0 = Gp + r * nc;
      for (int z = o.z0 + l; z < o.z1; z += 1 << s) {
        const float v = im[z];
        o.p[z] = isnan(v) ? v : __fsub_rn(v, dot4(W[z], g0 + S[z]));
      }
    }
    __syncthreads();
  }

  // ---- group reductions
  // Masked min/max and the convergence sums of the group, then what the
  // iteration takes from them (Iter), the same in every CTA.
  static __device__ __forceinline__ int fkey(float v) {   // order of floats as order of ints (an involution)
    const int k = __float_as_int(v);
    return k ^ ((k >> 31) & 0x7fffffff);
  }
  static __device__ __forceinline__ float funkey(int k) { return __int_as_float(k ^ ((k >> 31) & 0x7fffffff)); }

  // unsigned keys in the floats' order, 0 below all of them
  static __device__ __forceinline__ unsigned long long ukey(float v) { return (unsigned)fkey(v) ^ 0x80000000u; }
  static __device__ __forceinline__ float unukey(unsigned long long k) { return funkey((int)((unsigned)k ^ 0x80000000u)); }

  // Warp 0 takes the range and forms the bin map, warp 1 the sums and the
  // convergence value (chains of FP64 divisions), the others run idle().
  // Whole-GPU path: the range by atomics on the accumulator set, the sums in
  // CTA order from the CTAs' slots.
  template <class Idle>
  __device__ bool reduce_stats(float vmin, float vmax, double s0, double s1, bool need_cv, Idle &&idle) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    double *sc = red();
    vmin = funkey(__reduce_min_sync(kFull, fkey(vmin)));
    vmax = funkey(__reduce_max_sync(kFull, fkey(vmax)));
    if (need_cv) { s0 = warp_sum(s0); s1 = warp_sum(s1); }
    if (lane == 0) { sc[warp] = vmin; sc[32 + warp] = vmax; sc[64 + warp] = s0; sc[96 + warp] = s1; }
    __syncthreads();
    const bool in = lane < nw;
    if (warp == 0) {
      vmin = funkey(__reduce_min_sync(kFull, fkey(in ? (float)sc[lane] : INFINITY)));
      vmax = funkey(__reduce_max_sync(kFull, fkey(in ? (float)sc[32 + lane] : -INFINITY)));
      if (lane == 0) {
        if constexpr (Group::kGrid) {
          atomicMax(acc_set(seq), ~ukey(vmin) & 0xffffffffull);
          atomicMax(acc_set(seq) + 1, ukey(vmax));
        } else {
          slotA()->v[0] = vmin;
          slotA()->v[1] = vmax;
        }
      }
    } else if (warp == 1 && need_cv) {
      s0 = warp_sum(in ? sc[64 + lane] : 0.0);
      s1 = warp_sum(in ? sc[96 + lane] : 0.0);
      if (lane == 0) { slotA()->v[2] = s0; slotA()->v[3] = s1; }
    }
    N4_MARK(PH_A_LOOP);
    if (!g.sync()) return false;
    Iter &it = iter();
    if (warp == 0) {
      float mn = INFINITY, mx = -INFINITY;
      if constexpr (Group::kGrid) {
        mn = unukey(~__ldcg(acc_set(seq)) & 0xffffffffull);
        mx = unukey(__ldcg(acc_set(seq) + 1));
      } else if (lane < K) {
        const Stats *p = g.peer(slotA(), lane);
        mn = (float)p->v[0];
        mx = (float)p->v[1];
      }
      if constexpr (!Group::kGrid) {
        mn = funkey(__reduce_min_sync(kFull, fkey(mn)));
        mx = funkey(__reduce_max_sync(kFull, fkey(mx)));
      }
      if (lane == 0) {
        it.st[0] = mn; it.st[1] = mx;
        // bin range of the masked logU (N4.py:14-15); st holds FP32 values
        const double slope = ((double)mx - (double)mn) / (double)(pr.bins - 1);
        it.degenerate = !(slope > 0.0) || !isfinite(slope);
        it.bm = BinMap(mn, it.degenerate ? 1.0 : slope, pr.bins);
        it.scale = ldexp(1.0, hshift);
      }
    } else if (warp == 1) {
      if (need_cv) {
        s0 = s1 = 0.0;
        if constexpr (Group::kGrid) {
          // eight slots' loads in flight
          for (int k0 = lane; k0 < K; k0 += 256) {
            double a[8], b[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              const Stats *p = g.peer(slotA(), min(k0 + 32 * u, K - 1));
              a[u] = __ldcg(&p->v[2]);
              b[u] = __ldcg(&p->v[3]);
            }
#pragma unroll
            for (int u = 0; u < 8; ++u)
              if (k0 + 32 * u < K) { s0 += a[u]; s1 += b[u]; }
          }
        } else if (lane < K) {
          const Stats *p = g.peer(slotA(), lane);
          s0 = p->v[2];
          s1 = p->v[3];
        }
        s0 = warp_sum(s0);
        s1 = warp_sum(s1);
        if (lane == 0) {
          it.st[2] = s0; it.st[3] = s1;
          it.cv = cv_from(it.st);
        }
      }
    } else {
      idle();
    }
    if constexpr (Group::kGrid) acc_clear();
    acc_next();
    return true;
  }

  // Sum of every CTA's partial entries over the group; fin(c, sum) for every
  // entry c of [0, n) on one thread of each CTA, the same sum in all of them.
  // Cluster path: the partials are in `mine` (shared memory), read through
  // DSMEM in rank order, eight loads in flight; exact for the integer
  // histogram, Kahan-compensated for the fit's float partials.  A partial is
  // written again only after later barriers of the iteration, by which time
  // every peer has read it.
  template <class T, class Fin>
  __device__ __forceinline__ void peers_sum(const T *mine, int n, Fin &&fin) const {
    for (int c = threadIdx.x; c < n; c += blockDim.x) {
      SumOf<T> acc;
      for (int k0 = 0; k0 < K; k0 += 8) {
        T v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = k0 + u < K ? *(g.peer(mine, k0 + u) + c) : T(0);
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (k0 + u < K) acc.add(v[u]);
      }
      fin(c, acc.value());
    }
  }
  template <class T> struct SumOf;

  // Whole-GPU path: the accumulator set of the current sum, and, after its
  // barrier, the set that may be cleared (the one read at the previous sum).
  __device__ __forceinline__ unsigned long long *acc_set(int s) const {
    if constexpr (Group::kGrid) return g.acc + (size_t)(s % 3) * g.len;
    else return nullptr;
  }
  __device__ __forceinline__ void acc_clear() const {
    if constexpr (Group::kGrid) {
      if (rank == 0) {
        unsigned long long *a = acc_set(seq + 2);
        for (int i = threadIdx.x; i < g.len; i += blockDim.x) a[i] = 0ull;
      }
    }
  }
  // The next sum's set; read again only after further barriers of the CTA.
  __device__ __forceinline__ void acc_next() {
    __syncthreads();
    if (Group::kGrid && threadIdx.x == 0) ++seq;
  }

  // Fixed-point scale of the lattice sums of the whole-GPU path: `bound` is at
  // least the sum of the magnitudes of all terms, so that the 64-bit integer
  // sum stays below 2^62, whichever CTAs the terms are in (a mask of nearly
  // empty rows leaves most of them to one); integer sums are exact and the same
  // in any order.
  static __device__ __forceinline__ int sum_shift(double bound) {
    return min(61 - ilogb(fmin(fmax(bound, 1e-30), 1e300)), 52);
  }

  // ---- separable fit contraction of the rows into the group's lattice sums
  // num: the residuals with weights w^3/sum w^2; den: the mask with weights
  // w^2 (N4.py:224-236).
  //   T1[row][cz]   z contraction: the lane of a (row, span) part accumulates
  //                 the span's 4 targets in registers; the parts of a span
  //                 (every 2^szh-th voxel each, so that a span's lanes read
  //                 consecutive voxels and weights; equal pieces of 32 voxels
  //                 met in one shared-memory bank: 320x320x256 without a mask,
  //                 9.2M cycles over 18 iterations against 4.3M) are added by
  //                 shuffles, and target t takes its sums from spans t-3 .. t
  //                 by shuffles too
  //   T2[m][cy][cz] y contraction over the CTA's rows of each x-plane
  //   lattice       x contraction (the CTA's partial lattice)
  // then the group's sum of the partial lattices, fin(c, sum) per entry.  The
  // sums across rows (y, x and over the CTAs) are Kahan-compensated or exact:
  // a control point of the 256x256x160 grid gathers ~5e5 voxels through them.
  // The sum within a row covers one span and is plain FP32.
  template <bool Num, class Fin>
  __device__ bool contract(Fin &&fin) {
    float *T1 = Gd();   // Gd is dead between pass A and the next update
    const Iter &it = iter();
    const bool degenerate = Num && it.degenerate;
    if (!Group::kGrid && (nact << sz) <= kQuadLanes && az.nsp <= 8) {
      quad_rows<Num>(T1, degenerate);
    } else {
      const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
      const int l = lane & ((1 << sz) - 1), rs = 5 - sz, d = 1 << (Group::kGrid ? szh : 0);
      const int sub = lane >> sz, hh = Group::kGrid ? szh : 0;
      const int per = (1 << sz) >> hh;   // spans per round: all of them, up to 32
      const int n = nact, nsp = az.nsp, nc = ncz, ntask = (n + (1 << rs) - 1) >> rs;
      const auto rm = row_map();
      const int *Lo = at<int>(az.o_lo), *Hi = at<int>(az.o_hi);
      const SpanSums<Num> sums = span_sums<Num>();
      for (int sp0 = 0; sp0 < nsp; sp0 += per) {
        const int k = l >> hh, sp = sp0 + k, h = l & (d - 1);
        const bool in = sp < nsp;
        const int lo = in ? Lo[sp] : 0, hi = in ? Hi[sp] : 0;
        for (int task = warp; task < ntask; task += nw) {
          const int r = (task << rs) + sub;
          const bool on = in && r < n;
          float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          if (on && !degenerate) {
            const Row o = rm(r);
            int a, b;
            a = max(lo, o.z0);
            b = min(hi, o.z1);
            if constexpr (Group::kGrid) sums.template add<2>(o.p, a + h, b, d, s);
            else if (nsp > 2) sums.template add<3>(o.p, a, b, 1, s);
            else sums.template add<4>(o.p, a, b, 1, s);
          }
          for (int w = d >> 1; w; w >>= 1) {
            s.x += __shfl_xor_sync(kFull, s.x, w); s.y += __shfl_xor_sync(kFull, s.y, w);
            s.z += __shfl_xor_sync(kFull, s.z, w); s.w += __shfl_xor_sync(kFull, s.w, w);
          }
          // the sums of the one, two and three spans before
          const float y1 = __shfl_up_sync(kFull, s.y, d), z1 = __shfl_up_sync(kFull, s.z, d),
                      w1 = __shfl_up_sync(kFull, s.w, d), z2 = __shfl_up_sync(kFull, s.z, 2 * d),
                      w2 = __shfl_up_sync(kFull, s.w, 2 * d), w3 = __shfl_up_sync(kFull, s.w, 3 * d);
          if (on && h == 0) {
            float *t1 = T1 + r * nc + sp;
            const bool p1 = k >= 1, p2 = k >= 2, p3 = k >= 3;
            // targets in the order of span mod 4; a round finds the last
            // three targets of the one before open
            const auto put = [&](int i, float x0, float x1, float x2, float x3) {
              const float x = rotated_sum(sp & 3, x0, x1, x2, x3);
              t1[i] = sp0 > 0 && k + i < 3 ? t1[i] + x : x;
            };
            put(0, s.x, p1 ? y1 : 0.0f, p2 ? z2 : 0.0f, p3 ? w3 : 0.0f);
            if (k == per - 1 || sp == nsp - 1) {
              put(1, s.y, p1 ? z1 : 0.0f, p2 ? w2 : 0.0f, 0.0f);
              put(2, s.z, p1 ? w1 : 0.0f, 0.0f, 0.0f);
              put(3, s.w, 0.0f, 0.0f, 0.0f);
            }
          }
          __syncwarp();
        }
      }
    }
    __syncthreads();
    N4_MARK(PH_F_T1);
    double scale = 1.0;
    if constexpr (Group::kGrid) {
      // den: weights below 1.  num: with w <= 2/3 and sum w^2 >= 0.46 per axis,
      // w^3/sum w^2 <= 1.45 w^2, so an entry's terms sum to at most 3.1 times
      // its den times the largest residual.
      scale = ldexp(1.0, sum_shift(Num ? 4.0 * denmax * (degenerate ? 0.0f : it.rmax) : nfg));
    }
    const int slice = ncy * ncz;
    for (int m0 = 0; m0 < np || m0 == 0; m0 += tp) {
      const int cnt = min(tp, np - m0);
      if (np > tp) {
        build_ytab(m0, cnt);
        __syncthreads();
      }
      plane_sums<Num>(T1, cnt);
      __syncthreads();
      N4_MARK(PH_F_T2);
      // x contraction of planes m0 .. m0 + cnt - 1
      const float *T2p = T2();
      const float *PX = at<float>(Num ? ax.o_p : ax.o_q);
      for (int c = threadIdx.x; c < nlat; c += blockDim.x) {
        const int cx = c / slice, cc = c - cx * slice;
        KahanSum acc;
        bool any = false;
        for (int j = 0; j < 4; ++j) {
          const int sp = cx - j;
          if (sp < 0 || sp >= ax.nsp) continue;
          const int lo = at<int>(ax.o_lo)[sp], hi = at<int>(ax.o_hi)[sp];
          int m, vx;
          const int end = Group::kGrid ? min(hi, vx0 + m0 + cnt) : hi;
          if constexpr (Group::kGrid) {
            vx = max(lo, vx0 + m0);
            m = vx - vx0 - m0;
          } else {
            m = lo <= rank ? 0 : (lo - rank + K - 1) / K;
            vx = rank + m * K;
          }
          for (; vx < end; vx += Group::kGrid ? 1 : K, ++m) {
            acc.add_prod(PX[vx * 4 + j], T2p[m * slice + cc]);
            any = true;
          }
        }
        if constexpr (Group::kGrid) {
          if (any) {
            double v = ((double)acc.s - (double)acc.c) * scale;
            // a part beyond the bound is one of a map that is not finite
            if (!(fabs(v) < 4611686018427387904.0)) atomicAdd(acc_set(seq) + g.len - 1, 1ull);
            else if (v != 0.0) {
              atomicAdd(acc_set(seq) + c, (unsigned long long)__double2ll_rn(v));
              for (int k = 1; k < pr.sum_words; ++k) {
                v = (v - rint(v)) / kSumWordUnit;   // exact
                atomicAdd(acc_set(seq) + k * pl.NLAT + c, (unsigned long long)__double2ll_rn(v));
              }
            }
          }
        } else {
          slotC()[c] = acc.value();
        }
      }
      if (np > tp) __syncthreads();
    }
    N4_MARK(PH_F_P);
    if (!g.sync()) return false;
    if constexpr (Group::kGrid) {
      const unsigned long long *a = acc_set(seq);
      const bool nan = __ldcg(a + g.len - 1) != 0;
      const double inv = 1.0 / scale;
      for (int c = threadIdx.x; c < nlat; c += blockDim.x) {
        double s = (double)(long long)__ldcg(a + c), unit = 1.0;
        for (int k = 1; k < pr.sum_words; ++k) {
          unit *= kSumWordUnit;
          s += (double)(long long)__ldcg(a + k * pl.NLAT + c) * unit;
        }
        fin(c, nan ? kNaN : (float)(s * inv));
      }
      acc_clear();
      acc_next();
    } else {
      peers_sum(slotC(), nlat, fin);
      __syncthreads();
    }
    N4_MARK(PH_F_RED);
    return true;
  }

  // A bound on the voxels' residuals x - E(x) (whole-GPU path), which are linear
  // within a bin: the larger of the bin's ends that hold weight in the
  // histogram.  Bins without any have no voxel, and E there, a quotient of two
  // sums that are rounding errors, may be anything: with them in the bound, the
  // unit of the lattice sums grew to 2^-32 in a volume with one voxel of 1e12
  // (lattice 3e-5 off the FP64 oracle instead of 1e-6).  At an end without
  // weight a voxel lies within half a unit of the histogram of the other end;
  // the last bin's may be one that the histogram drops.  From the bins a thread
  // has just tabulated; read after the z contraction's barrier.  Every CTA has
  // the same map.  (One value per warp and a loop over them in every thread took
  // 10 of 1366 us at 181x217x181.)
  __device__ __forceinline__ void residual_max() {
    if ((int)(threadIdx.x & ~31u) + 1 >= pr.bins) return;
    const float2 *t = R2();
    const unsigned long long *h = H64();
    const float unit = __int_as_float((127 - hshift) << 23);   // 2^-hshift
    float m = 0.0f;
    for (int b = threadIdx.x; b + 1 < pr.bins; b += blockDim.x) {
      const bool lo = h[b] != 0, hi = h[b + 1] != 0 || b + 2 == pr.bins;
      const float e = fmaxf(lo ? fabsf(t[b].x) : 0.0f, hi ? fabsf(t[b].x + t[b].y) : 0.0f);
      if (lo || hi) m = fmaxf(m, lo && hi ? e : e + fabsf(t[b].y) * unit);
    }
    const int k = __reduce_max_sync(kFull, __float_as_int(m));
    if ((threadIdx.x & 31) == 0) atomicMax((int *)&iter().rmax, k);
  }

  // x0 + x1 + x2 + x3, the sums of spans s, s - 1, s - 2, s - 3, added in the
  // order of span mod 4 (m = s mod 4).
  static __device__ __forceinline__ float rotated_sum(int m, float x0, float x1, float x2, float x3) {
    const float a = m & 1 ? x1 : x0, b = m & 1 ? x0 : x3, c = m & 1 ? x3 : x2, e = m & 1 ? x2 : x1;
    const float t0 = m & 2 ? c : a, t1 = m & 2 ? e : b, t2 = m & 2 ? a : c, t3 = m & 2 ? b : e;
    return __fadd_rn(__fadd_rn(__fadd_rn(t0, t1), t2), t3);
  }

  // The four targets' sums of every d-th voxel of [a, b) of a row, in voxel
  // order: weights times the residual R = logU - E(logU) (Num), or the weights
  // of the masked voxels.  Voxels outside the mask add zeros.  The residuals of U voxels are
  // formed together, without branches: 4 on the cluster path's long spans, 3 on
  // its short ones (5 or 6 voxels: two steps, 6 slots instead of 8; 26.0k
  // against 28.3k cycles at 8 spans of 44 voxels on 6 CTAs), 2 on the whole-GPU
  // path (fewer registers: 1024 threads).
  template <bool Num>
  struct SpanSums {
    float bmin, ih, il, lim;
    const float4 *W;
    const float2 *R2;
    const BinMap *bm;
    const double *E;
    int bins;
    // the terms x of U voxels v
    template <int U>
    __device__ __forceinline__ void terms(const float (&v)[U], float (&x)[U]) const {
      unsigned top = 0;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if constexpr (Num) {
          int k;
          float f;
          const bool in = coord_split(v[u], bmin, ih, il, lim, k, f);
          x[u] = in ? residual_lin(k, f, R2) : 0.0f;
          if (!in && !isnan(v[u])) top |= 1u << u;
        } else {
          x[u] = isnan(v[u]) ? 0.0f : 1.0f;
        }
      }
      if (Num && top) {
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (top >> u & 1u) x[u] = residual_top(bm, v[u], E, bins);
      }
    }
    template <int U>
    __device__ __forceinline__ void add(const float *p, int a, int b, int d, float4 &s) const {
      for (int z = a; z < b; z += U * d) {
        float v[U], x[U];
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = z + u * d < b ? p[z + u * d] : kNaN;
        terms(v, x);
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const float4 w = W[z + u * d];   // past the row: the next table or its tail, times zero
          s.x = __fmaf_rn(w.x, x[u], s.x); s.y = __fmaf_rn(w.y, x[u], s.y);
          s.z = __fmaf_rn(w.z, x[u], s.z); s.w = __fmaf_rn(w.w, x[u], s.w);
        }
      }
    }
  };
  template <bool Num>
  __device__ __forceinline__ SpanSums<Num> span_sums() const {
    const Iter &it = iter();
    return SpanSums<Num>{it.bm.fmin, it.bm.ih, it.bm.il, it.bm.ff_limit, at<float4>(Num ? az.o_p : az.o_q), R2(), &it.bm,
                         E(), pr.bins};
  }

  // The z contraction with four lanes per (row, span): each forms the terms of
  // every fourth voxel, then, in voxel order, the sum of one of the span's four
  // targets.  The same sums as one lane per (row, span), with four times the
  // lanes, for CTAs of 256 (row, span)s or fewer, half of the cluster path's
  // default 512 threads, with which the line was drawn (16 CTAs, 64x64x48, 152
  // rows of one span: 7.8k cycles per iteration against 10.5k; 304 (row, span)s:
  // 8.3k against 7.7k).
  static constexpr int kQuadLanes = 256;
  template <bool Num>
  __device__ __forceinline__ void quad_rows(float *T1, bool degenerate) const {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int ls = sz + 2, l = lane & ((1 << ls) - 1), slot = l >> 2, j = l & 3, rs = 5 - ls;
    const int n = nact, nsp = az.nsp, nc = ncz, ntask = (n + (1 << rs) - 1) >> rs, zmax = Z - 1;
    const auto rm = row_map();
    const bool in = slot < nsp;
    const int lo = in ? at<int>(az.o_lo)[slot] : 0, hi = in ? at<int>(az.o_hi)[slot] : 0;
    const SpanSums<Num> sums = span_sums<Num>();
    const float *Wj = (const float *)sums.W + j;
    for (int task = warp; task < ntask; task += nw) {
      const int r = (task << rs) + (lane >> ls);
      const bool on = in && r < n;
      int a = 0, b = 0;
      const float *p = nullptr;
      if (on) {
        const Row o = rm(r);
        a = max(lo, o.z0);
        b = min(hi, o.z1);
        p = o.p;
      }
      const int len = __reduce_max_sync(kFull, degenerate ? 0 : b - a);
      float acc = 0.0f;
      constexpr int U = 2;
      for (int q = 0; q < len; q += 4 * U) {
        float v[U], x[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int z = a + q + 4 * u + j;
          v[u] = z < b ? p[z] : kNaN;
        }
        sums.terms(v, x);
        const float *w = Wj + 4 * min(a + q, zmax);   // past the row: the next table or its tail, times zero
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int i = 0; i < 4; ++i) acc = __fmaf_rn(w[4 * (4 * u + i)], __shfl_sync(kFull, x[u], i, 4), acc);
      }
      // target slot + j from the spans slot, slot - 1, ... (lane j + i of the
      // i-th before), for j = 0 and, at the last span, every j
      const float c1 = __shfl_up_sync(kFull, acc, 3), c2 = __shfl_up_sync(kFull, acc, 6),
                  c3 = __shfl_up_sync(kFull, acc, 9);
      if (on && (j == 0 || slot == nsp - 1))
        T1[r * nc + slot + j] = rotated_sum(slot & 3, acc, j < 3 && slot >= 1 ? c1 : 0.0f,
                                            j < 2 && slot >= 2 ? c2 : 0.0f, j < 1 && slot >= 3 ? c3 : 0.0f);
    }
  }

  // T2[m][cy][cz] of `cnt` x-planes.  Cluster path: Kahan in two chains per
  // entry (rows at even and at odd distance from the span's start); rows before
  // and after the plane's listed ones add zeros, which a chain need take only
  // once.  One thread per entry over its four spans where there are at least
  // four and the entries are no more than the default 512 threads, with which
  // the line was drawn; else one thread per (plane, cz) that walks the plane
  // once for all its entries (per iteration, 16 CTAs, 64x64x48: 1 span 4.1k
  // cycles against 6.4k, 8 spans 6.9k against 4.4k; 6 CTAs, 64x64x44: 4.7k
  // against 8.0k and 8.3k against 11.2k).  Same terms in the same order either
  // way.  Whole-GPU path, whose CTAs hold two or three planes: one lane per
  // span, the four sums added in FP64.
  template <bool Num>
  __device__ void plane_sums(const float *T1, int cnt) {
    float *T2p = T2();
    const int *yt = ytab();
    const float *PY = at<float>(Num ? ay.o_p : ay.o_q);
    const int nc = ncz, ny = ncy, nsp = ay.nsp, n = cnt * ny * nc, w = nsp + 1;
    const auto rm = row_map();
    const int *Lo = at<int>(ay.o_lo), *Hi = at<int>(ay.o_hi);
    const int yy = Y;
    const auto first_row = [=](int m, int sp) {   // of span sp in plane m
      if constexpr (Group::kRowList) return yt[m * w + sp];
      else return m * yy + (sp < nsp ? Lo[sp] : yy);
    };
    if constexpr (!Group::kGrid) {
      if (nsp < 4 || n > 512) {
      // one thread per (plane, cz): spans from the last to the first, the four
      // targets a span reaches open in registers
      for (int u = threadIdx.x; u < cnt * nc; u += blockDim.x) {
        const int m = u / nc, cz = u - m * nc;
        float *out = T2p + m * ny * nc + cz;
        KahanSum a[4], b[4];   // target sp + j: rows at even and at odd distance
        for (int sp = nsp - 1; sp >= 0; --sp) {
          const int lo = Lo[sp], hi = Hi[sp];
          const int r0 = first_row(m, sp), k = first_row(m, sp + 1) - r0;
          const int va = k > 0 ? rm.vy(r0) : hi, vb = va + k;
          if (va > lo) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              a[j].add(0.0f);
              if (va > lo + 1) b[j].add(0.0f);
            }
          }
          const float *t1 = T1 + r0 * nc + cz;
          const float4 *py = (const float4 *)PY + va;
          int i = 0;
          const auto take = [&](KahanSum (&s)[4]) {
            const float4 p = py[i];
            const float x = t1[i * nc];
            s[0].add_prod(p.x, x); s[1].add_prod(p.y, x); s[2].add_prod(p.z, x); s[3].add_prod(p.w, x);
            ++i;
          };
          if (k > 0 && ((va - lo) & 1)) take(b);
          while (i + 1 < k) { take(a); take(b); }
          if (i < k) take(a);
          if (k > 0 && vb < hi) {
            const bool odd = (vb - lo) & 1, both = vb + 1 < hi;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              if (!odd || both) a[j].add(0.0f);
              if (odd || both) b[j].add(0.0f);
            }
          }
          a[3].merge(b[3]);
          out[(sp + 3) * nc] = a[3].value();
#pragma unroll
          for (int j = 3; j > 0; --j) { a[j] = a[j - 1]; b[j] = b[j - 1]; }
          a[0] = KahanSum();
          b[0] = KahanSum();
        }
#pragma unroll
        for (int j = 1; j < 4; ++j) {   // targets 0, 1, 2
          a[j].merge(b[j]);
          out[(j - 1) * nc] = a[j].value();
        }
      }
      return;
      }
      for (int u = threadIdx.x; u < n; u += blockDim.x) {
        const int q = u / nc, cz = u - q * nc;
        const int m = q / ny, cy = q - m * ny;
        KahanSum acc, acc2;
        for (int j = 0; j < 4; ++j) {
          const int sp = cy - j;
          if (sp < 0 || sp >= nsp) continue;
          const int lo = Lo[sp], hi = Hi[sp];
          const int r0 = first_row(m, sp), r1 = first_row(m, sp + 1);
          const int va = r0 < r1 ? rm.vy(r0) : hi, vb = va + (r1 - r0);
          if (va > lo) acc.add(0.0f);
          if (va > lo + 1) acc2.add(0.0f);
          const float *t1 = T1 + r0 * nc + cz, *py = PY + va * 4 + j;
          int k = r1 - r0;
          if (k > 0 && ((va - lo) & 1)) {
            acc2.add_prod(py[0], t1[0]);
            t1 += nc;
            py += 4;
            --k;
          }
          for (; k > 1; k -= 2, t1 += 2 * nc, py += 8) {
            acc.add_prod(py[0], t1[0]);
            acc2.add_prod(py[4], t1[nc]);
          }
          if (k > 0) acc.add_prod(py[0], t1[0]);
          if (r0 < r1 && vb < hi) {
            const int even = (vb - lo) & 1 ? vb + 1 : vb, odd = (vb - lo) & 1 ? vb : vb + 1;
            if (even < hi) acc.add(0.0f);
            if (odd < hi) acc2.add(0.0f);
          }
        }
        acc.merge(acc2);
        T2p[u] = acc.value();
      }
      return;
    }
    const int nt = (n * 4 + 31) & ~31;   // whole warps: the lanes of an entry exchange their sums
    for (int t = threadIdx.x; t < nt; t += blockDim.x) {
      const int u = t >> 2, j = t & 3;
      const int q = u / nc, cz = u - q * nc;
      const int m = q / ny, cy = q - m * ny, sp = cy - j;
      double s = 0.0;
      if (u < n && sp >= 0 && sp < nsp) {
        KahanSum acc, acc2;
        int r = first_row(m, sp);
        const int end = first_row(m, sp + 1);
        for (; r + 1 < end; r += 2) {
          acc.add_prod(PY[rm.vy(r) * 4 + j], T1[r * nc + cz]);
          acc2.add_prod(PY[rm.vy(r + 1) * 4 + j], T1[(r + 1) * nc + cz]);
        }
        if (r < end) acc.add_prod(PY[rm.vy(r) * 4 + j], T1[r * nc + cz]);
        s = ((double)acc.s - (double)acc.c) + ((double)acc2.s - (double)acc2.c);
      }
      s += __shfl_xor_sync(kFull, s, 1);
      s += __shfl_xor_sync(kFull, s, 2);
      if (u < n && j == 0) T2p[u] = (float)s;
    }
  }

  // ---- pass A: the previous update's convergence sums from eval(Gd) (when
  // need_cv), applied to logU (when apply: logU -= eval(Gd)), and the masked
  // min/max of logU; clears the histogram copies
  __device__ bool pass_a(bool need_cv, bool apply) {
    float vmin = INFINITY, vmax = -INFINITY;
    double sy = 0.0, syy = 0.0;
    const float *Gp = Gd();
    const float4 *W4 = at<float4>(az.o_w);
    const int nc = ncz;
    if constexpr (Group::kGrid) {
      // a row's lanes take consecutive voxels: bound by the shared-memory reads
      // of the rows held there and by the lines of the others.  With a piece of
      // the row per lane, whose four values of Gd stay in registers, the lanes'
      // weights met in the same banks and every line of a row in global memory
      // came several times: 12.5M cycles over 18 iterations of 320x320x256
      // without a mask against 2.8M so, 1.83M against 0.85M at 256x256x160.
      const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
      const int s = row_lanes_log2(Z), l = lane & ((1 << s) - 1), sub = lane >> s, rs = 5 - s, n = nact;
      const auto rm = row_map();
      const int *S = at<int>(az.o_s);
      for (int r = (warp << rs) + sub; r < n; r += nw << rs) {
        const Row o = rm(r);
        const float *g0 = Gp + r * nc;
        constexpr int U = 2;
        for (int z0 = o.z0 + l; z0 < o.z1; z0 += U << s) {
          float v[U], ed[U];
#pragma unroll
          for (int u = 0; u < U; ++u) v[u] = z0 + (u << s) < o.z1 ? o.p[z0 + (u << s)] : kNaN;
          if (need_cv) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
              const int z = min(z0 + (u << s), o.z1 - 1);
              ed[u] = dot4(W4[z], g0 + S[z]);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
              const bool in = !isnan(v[u]);
              const double yd = in ? (double)expm1_conv(-ed[u]) : 0.0;
              sy += yd;
              syy += yd * yd;
              if (apply) {
                v[u] = __fsub_rn(v[u], ed[u]);
                if (in) o.p[z0 + (u << s)] = v[u];
              }
            }
          }
#pragma unroll
          for (int u = 0; u < U; ++u) {
            vmin = fminf(vmin, v[u]);   // a NaN operand is passed over
            vmax = fmaxf(vmax, v[u]);
          }
        }
      }
    } else {
      span_pass(
          [&](const Row &o, int r, int a, int b, int sp) {
            if (a >= b) return;
            constexpr int U = 2;
            if (need_cv) {
              const float *gp = Gp + r * nc + sp;
              const float g[4] = {gp[0], gp[1], gp[2], gp[3]};
              for (int z = a; z < b; z += U) {
                float v[U], ed[U], y[U];
#pragma unroll
                for (int u = 0; u < U; ++u) v[u] = z + u < b ? o.p[z + u] : kNaN;
#pragma unroll
                for (int u = 0; u < U; ++u) {
                  ed[u] = dot4(W4[z + u], g);   // past the row: finite, not used
                  y[u] = expm1_conv(-ed[u]);
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                  const bool in = !isnan(v[u]);
                  const double yd = in ? (double)y[u] : 0.0;
                  sy += yd;
                  syy += yd * yd;
                  if (apply) {
                    v[u] = __fsub_rn(v[u], ed[u]);
                    if (in) o.p[z + u] = v[u];
                  }
                  vmin = fminf(vmin, v[u]);   // a NaN operand is passed over
                  vmax = fmaxf(vmax, v[u]);
                }
              }
            } else {
              for (int z = a; z < b; ++z) {
                const float v = o.p[z];
                vmin = fminf(vmin, v);
                vmax = fmaxf(vmax, v);
              }
            }
          });
    }
    const bool ok = reduce_stats(vmin, vmax, sy, syy, need_cv, [&] {
      // the copies lie in the Gd region, which every thread has read by now
      unsigned *h = hist();
      for (int i = (int)threadIdx.x - 64; i < kHistCopies * pr.bins; i += (int)blockDim.x - 64) h[i] = 0u;
    });
    N4_MARK(PH_A_RED);
    return ok;
  }

  // ---- pass B + sharpening: histogram of logU over the group, then E
  __device__ bool pass_b() {
    const int bins = pr.bins;
    Iter &it = iter();
    // for the sharpening, beside the first voxels
    if (threadIdx.x == blockDim.x - 1) {
      it.gauss = gauss_of(it.bm.slope, pr.fwhm);
      it.rmax = 0.0f;
    }
    {
      const float bmin = it.bm.fmin, ih = it.bm.ih, il = it.bm.il, lim = it.bm.ff_limit;
      const float scale = (float)it.scale;
      const unsigned one = (unsigned)scale;
      const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
      const int s = row_lanes_log2(Z), l = lane & ((1 << s) - 1), sub = lane >> s, rs = 5 - s;
      unsigned *hc = hist() + (warp % kHistCopies) * bins;
      const auto rm = row_map();
      const int n = nact;
      for (int r = (warp << rs) + sub; r < n; r += nw << rs) {
        const Row o = rm(r);
        constexpr int U = Group::kGrid ? 2 : 3;   // 44 to 48 voxels on 8 lanes: two steps
        for (int z = o.z0 + l; z < o.z1; z += U << s) {
          float v[U], f[U];
          int k[U];
          bool in[U];
#pragma unroll
          for (int u = 0; u < U; ++u) v[u] = z + (u << s) < o.z1 ? o.p[z + (u << s)] : kNaN;
#pragma unroll
          for (int u = 0; u < U; ++u) in[u] = coord_split(v[u], bmin, ih, il, lim, k[u], f[u]);
#pragma unroll
          for (int u = 0; u < U; ++u) {
            if (in[u]) {
              const unsigned qhi = min(__float2uint_rn(__fmul_rn(f[u], scale)), one);
              atomicAdd(&hc[k[u]], one - qhi);
              atomicAdd(&hc[k[u] + 1], qhi);
            } else if (!isnan(v[u])) {
              unsigned qlo = 0, qhi = 0;
              const int key = hist_bin_top(&it.bm, v[u], bins, it.scale, qlo, qhi);
              if (key >= 0) {
                atomicAdd(&hc[key], qlo);
                if (qhi) atomicAdd(&hc[key + 1], qhi);
              }
            }
          }
        }
      }
    }
    __syncthreads();
    N4_MARK(PH_B_LOOP);
    for (int b = threadIdx.x; b < bins; b += blockDim.x) {
      unsigned long long s = 0;
#pragma unroll
      for (int c = 0; c < kHistCopies; ++c) s += hist()[c * bins + b];
      if constexpr (Group::kGrid) {
        if (s) atomicAdd(acc_set(seq) + b, s);
      } else {
        slotB()[b] = s;
      }
    }
    N4_MARK(PH_B_MERGE);
    if (!g.sync()) return false;
    if constexpr (Group::kGrid) {
      const unsigned long long *a = acc_set(seq);
      for (int b = threadIdx.x; b < bins; b += blockDim.x) H64()[b] = __ldcg(a + b);
      acc_clear();
      acc_next();
    } else {
      peers_sum(slotB(), bins, [&](int b, unsigned long long s) { H64()[b] = s; });
      __syncthreads();
    }
    N4_MARK(PH_B_RED);
    const double inv = 1.0 / it.scale;   // exact: a power of two
    const unsigned long long *h64 = H64();
    const int a0 = alias0();
    SharpenBufs sb{at<double2>(a0 + pl.a_fa), at<double2>(a0 + pl.a_fb), at<double2>(pl.o_tw), at<double>(a0 + pl.a_ff)};
    sharpen_map([=](int b) { return (double)h64[b] * inv; }, bins, pl.npad, pl.hoff, it.bm.binMin, it.bm.slope,
                pr.wiener, it.gauss, sb, E(), R2());
    if constexpr (Group::kGrid) residual_max();
    N4_MARK(PH_SHARP);
    return true;
  }

  // ---- one sharpen + fit step from the current logU: the update goes to D
  // and into L, and its rows to Gd (through aux with `planes`)
  __device__ bool fit_step(bool planes = true) {
    if (!iter().degenerate) { if (!pass_b()) return false; }
    float *Dp = D(), *Lp = L();
    const float *dn = den();
    const bool zd = pr.zero_den != 0;
    const float eps = pr.eps;
    if (!contract<true>([&](int c, float nu) {   // the residual is formed inside the z contraction
          const float de = dn[c];
          const float d = zd ? (de != 0.0f ? nu / de : 0.0f) : nu / (de + eps);
          Dp[c] = d;
          Lp[c] += d;
        }))
      return false;
    if (planes) rowtab_planes(Dp);
    else rowtab(Dp);
    __syncthreads();
    N4_MARK(PH_UPDATE);
    return true;
  }

  __device__ float cv_from(const double st[4]) const {
    const double mean_y = st[2] / nfg;
    double var = st[3] / nfg - mean_y * mean_y;
    if (pr.ddof1) var = nfg > 1.0 ? var * nfg / (nfg - 1.0) : 0.0;
    return (float)(sqrt(var > 0.0 ? var : 0.0) / (1.0 + mean_y));
  }

  // Range of the masked voxels of one row of Z voxels (z0 | z1 << 16, 0 when
  // there is none) and their number, by one warp.
  static __device__ unsigned row_range(const float *p, int Z, int &count) {
    const int lane = threadIdx.x & 31;
    int z0 = Z, z1 = 0;
    count = 0;
    for (int b = 0; b < Z; b += 32) {
      const unsigned m = __ballot_sync(kFull, b + lane < Z && !isnan(p[b + lane]));
      if (m) {
        z0 = min(z0, b + __ffs(m) - 1);
        z1 = b + 32 - __clz(m);
        count += __popc(m);
      }
    }
    return z1 > 0 ? (unsigned)z0 | (unsigned)z1 << 16 : 0u;
  }

  // The rows i of [0, n) with range(i) != 0, in order: put(position, voxels
  // before it, i, range).  Returns their number; all threads call it.
  template <class Range, class Put>
  __device__ int list_rows(int n, Range &&range, Put &&put) {
    int *sc = (int *)red();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int rows = 0, voxels = 0;
    for (int b = 0; b < n; b += blockDim.x) {
      const int i = b + (int)threadIdx.x;
      const unsigned e = i < n ? range(i) : 0u;
      const int len = (int)(e >> 16) - (int)(e & 0xffffu);
      const unsigned m = __ballot_sync(kFull, e != 0);
      int ps = len;
      for (int o = 1; o < 32; o <<= 1) {
        const int q = __shfl_up_sync(kFull, ps, o);
        if (lane >= o) ps += q;
      }
      if (lane == 31) { sc[warp] = __popc(m); sc[32 + warp] = ps; }
      __syncthreads();
      int pr_ = rows + __popc(m & ((1u << lane) - 1)), pv = voxels + ps - len, tr = 0, tv = 0;
      for (int w = 0; w < nw; ++w) {
        if (w < warp) { pr_ += sc[w]; pv += sc[32 + w]; }
        tr += sc[w];
        tv += sc[32 + w];
      }
      if (e) put(pr_, pv, i, e);
      rows += tr;
      voxels += tv;
      __syncthreads();
    }
    return rows;
  }

  // First row whose preceding rows weigh at least `target`: prefix[k] is the
  // weight before CTA k's even share of the rows.  One warp.
  __device__ int boundary(const long long *prefix, long long target) const {
    const int lane = threadIdx.x & 31, c = grid_row_overhead(Z);
    int k = 0;
    for (int q = lane; q < K; q += 32)
      if (prefix[q] <= target) k = max(k, q);
    k = __reduce_max_sync(kFull, k);
    const long long rows = (long long)X * Y;
    const int lo = (int)(rows * k / K), hi = (int)(rows * (k + 1) / K);
    long long run = prefix[k];
    if constexpr (Group::kGrid) {
      for (int b = lo; b < hi; b += 32) {
        const unsigned e = b + lane < hi ? __ldcg(g.ext + b + lane) : 0u;
        const int w = e ? (int)(e >> 16) - (int)(e & 0xffffu) + c : 0;
        int ps = w;
        for (int o = 1; o < 32; o <<= 1) {
          const int q = __shfl_up_sync(kFull, ps, o);
          if (lane >= o) ps += q;
        }
        const unsigned m = __ballot_sync(kFull, b + lane < hi && run + ps - w >= target);
        if (m) return b + __ffs(m) - 1;
        run += __shfl_sync(kFull, ps, 31);
      }
    }
    return hi;
  }

  // The CTA's row list, the volume's masked voxels and the histogram's scale.
  __device__ bool find_rows() {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int cnt = 0, rows = 0;   // the warp's masked voxels, the CTA's rows
    if constexpr (Group::kGrid) {
      // even shares of the rows are looked over first, then the rows are dealt
      // out in contiguous ranges of equal weight
      const long long nrows = (long long)X * Y;
      const int q0 = (int)(nrows * rank / K), q1 = (int)(nrows * (rank + 1) / K);
      const int c = grid_row_overhead(Z);
      long long weight = 0;
      for (int i = q0 + warp; i < q1; i += nw) {
        int n;
        const unsigned e = row_range(src + (size_t)i * Z, Z, n);
        if (lane == 0) g.ext[i] = e;
        cnt += n;
        if (e) weight += (int)(e >> 16) - (int)(e & 0xffffu) + c;
      }
      long long *sc = (long long *)red();
      if (lane == 0) sc[warp] = weight;
      __syncthreads();
      if (threadIdx.x == 0) {
        for (int w = 1; w < nw; ++w) weight += sc[w];
        *slotB() = (unsigned long long)weight;
      }
      if (!g.sync()) return false;
      // K + 1 words, in the five lattices (1280 bytes at least), free before the first level
      long long *prefix = at<long long>(pl.o_L);
      for (int k = threadIdx.x; k < K; k += blockDim.x) prefix[k + 1] = (long long)__ldcg(g.peer(slotB(), k));
      __syncthreads();
      if (threadIdx.x == 0) {
        prefix[0] = 0;
        for (int k = 0; k < K; ++k) prefix[k + 1] += prefix[k];
      }
      __syncthreads();
      int *bd = (int *)(red() + 120);
      if (warp < 2) {
        const int b = boundary(prefix, prefix[K] * (rank + warp) / K);
        if (lane == 0) bd[warp] = b;
      }
      __syncthreads();
      const int r0 = bd[0], r1 = rank == K - 1 ? (int)nrows : bd[1];
      const unsigned *ext = g.ext;
      auto range = [=](int i) { return __ldcg(ext + r0 + i); };
      rows = list_rows(r1 - r0, range, [](int, int, int, unsigned) {});
      if (threadIdx.x == 0) {
        nact = rows;
        const bool in = (long long)rows * 16 <= pl.pool_bytes / 4;
        const int used = in ? (rows * 16 + 127) / 128 * 128 : 0;
        rowsp = in ? at<int4>(pl.o_pool) : (int4 *)(big + pl.b_rows);
        slab_off = pl.o_pool + used;
        slab_cap = (pl.pool_bytes - used) / 4;
        slab_g = (float *)(big + pl.b_imlog);
        gdp = (long long)rows * pl.NCZ * 4 <= pl.gd_bytes ? at<float>(pl.o_gd) : (float *)(big + pl.b_Gd);
        bd[0] = 0x7fffffff;
        bd[1] = -1;
      }
      __syncthreads();
      int4 *out = rowsp;
      const int yy = Y;
      list_rows(r1 - r0, range, [=](int r, int v, int i, unsigned e) {
        const int vx = (r0 + i) / yy;
        out[r] = make_int4(v - (int)(e & 0xffffu), (int)e, vx, r0 + i - vx * yy);
        if (r == 0) bd[0] = vx;
        if (r == rows - 1) bd[1] = vx;
      });
      if (threadIdx.x == 0) {
        vx0 = rows ? bd[0] : 0;
        np = rows ? bd[1] - bd[0] + 1 : 0;
      }
      __syncthreads();
      for (int r = threadIdx.x; r < rows; r += blockDim.x) out[r].z -= vx0;
    } else {
      const int nplane = X > rank ? (X - rank + K - 1) / K : 0, nrow = nplane * Y;
      const float *slab = at<float>(pl.sm_bytes + pl.b_imlog);
      unsigned *ext = at<unsigned>(pl.sm_bytes + pl.b_Gd);   // free before the first level
      for (int i = warp; i < nrow; i += nw) {
        int n;
        const unsigned e = row_range(slab + (size_t)i * Z, Z, n);
        if (lane == 0) ext[i] = e;
        cnt += n;
      }
      rows = nrow;
      if constexpr (Group::kRowList) {
        // a plane's rows are listed from its first to its last row with a masked
        // voxel, empty ones between them as the empty range [1, 1)
        int *ya = at<int>(pl.sm_bytes + pl.b_T2), *yb = ya + nplane;
        for (int m = threadIdx.x; m < nplane; m += blockDim.x) { ya[m] = Y; yb[m] = -1; }
        __syncthreads();
        const int yy = Y;
        for (int i = threadIdx.x; i < nrow; i += blockDim.x)
          if (ext[i]) {
            atomicMin(&ya[i / yy], i % yy);
            atomicMax(&yb[i / yy], i % yy);
          }
        __syncthreads();
        uint2 *out = at<uint2>(pl.o_rows);
        auto range = [=](int i) {
          const unsigned e = ext[i];
          return e || i % yy < ya[i / yy] || i % yy > yb[i / yy] ? e : 0x10001u;
        };
        rows = list_rows(nrow, range, [=](int r, int, int i, unsigned e) {
          const int m = i / yy;
          out[r] = make_uint2(e, (unsigned)m << 16 | (unsigned)(i - m * yy));
        });
      }
      nact = rows;
      np = nplane;
      vx0 = 0;
    }
    __syncthreads();
    // most voxels one histogram copy can get: rows go to warps, and so to
    // copies, in list order (pass_b)
    int *copies = (int *)(red() + 128);
    if (threadIdx.x < kHistCopies) copies[threadIdx.x] = 0;
    __syncthreads();
    const int rs = 5 - row_lanes_log2(Z);
    const auto rm = row_map();
    for (int r = threadIdx.x; r < rows; r += blockDim.x) {
      int len;
      if constexpr (Group::kRowList) {
        const Row o = rm(r);
        len = o.z1 - o.z0;
      } else {
        const unsigned e = at<unsigned>(pl.sm_bytes + pl.b_Gd)[r];
        len = (int)(e >> 16) - (int)(e & 0xffffu);
      }
      atomicAdd(&copies[(r >> rs) % kHistCopies], len);
    }
    __syncthreads();
    int most = 0;
    for (int k = 0; k < kHistCopies; ++k) most = max(most, copies[k]);
    __syncthreads();
    // the group's masked voxels and its fullest copy; the copies' sums stay
    // below 2^32, and the scale does not depend on a batch's other volumes
    if (!reduce_stats(0.0f, (float)most, lane == 0 ? (double)cnt : 0.0, 0.0, true, [] {})) return false;
    if (writer()) {
      nfg = iter().st[2];
      // an even eighth of a CTA's voxels (its planes whole) and 160 more, or
      // the fullest copy's voxels where they are more
      const long long even = Group::kGrid ? 0 : ((long long)(X + K - 1) / K * Y * Z + 7) / 8 + 160;
      hshift = hist_shift_for(max(even, (long long)(iter().st[1] * 1.000001) + 1));
    }
    publish();
    return true;
  }

  // ---- the whole volume (im_log read from job.imlog; cluster path: the slab
  // holds the local rows of im_log on entry)
  __device__ void run(const VolJob &job) {
    if (writer()) {
      X = job.X; Y = job.Y; Z = job.Z;
      rank = g.rank(); K = g.size();
      nact = 0; np = 0; vx0 = 0; hshift = 0;
      nfg = 1.0;
      src = job.imlog;
    }
    publish();
    const bool lead = (rank == 0 && threadIdx.x == 0);
    n4_report_t *rep = job.report;
    if (lead) { rep->device_begin_ns = global_ns(); rep->device_end_ns = 0; rep->sm = sm_id(); }

#ifdef N4_PHASE_TIMERS
    if (threadIdx.x == 0) {
      for (int k = 0; k < PH_N; ++k) ph_acc[k] = 0;
      ph_acc[PH_N] = clock64();
    }
#endif
    fft_twiddles(at<double2>(pl.o_tw), pl.npad);
    if (!find_rows()) { if (lead) rep->status = N4_ERR_TIMEOUT; return; }
    if (lead) { rep->foreground = (long long)nfg; rep->levels = 0; rep->warm_start_used = 0; }
    if (nfg < 1.0) {
      if (rank == 0) {
        for (int c = threadIdx.x; c < pl.NLAT; c += blockDim.x) job.lattice_out[c] = 0.0f;
        if (threadIdx.x == 0) rep->status = N4_ERR_EMPTY_MASK;
      }
      return;
    }

    // first-level lattice
    set_level(0);
    for (int c = threadIdx.x; c < nlat; c += blockDim.x) L()[c] = job.warm ? job.warm[c] : 0.0f;
    __syncthreads();

    for (int level = 0; level < pl.levels; ++level) {
      if (level > 0) {
        const int pcx = ncx, pcy = ncy, pcz = ncz;
        refine_lattice(L(), pcx, pcy, pcz, tmp());
        __syncthreads();
        set_level(level);
        for (int c = threadIdx.x; c < nlat; c += blockDim.x) L()[c] = tmp()[c];
        __syncthreads();
      }
      // logU of this level's lattice, then the constant denominator of the fit
      reset(L(), level == 0 && !Group::kGrid);
      float *dn = den();
      float dmax = 0.0f;
      if (!contract<false>([=, &dmax](int c, float v) { dn[c] = v; dmax = fmaxf(dmax, v); })) goto timeout;
      if constexpr (Group::kGrid) {
        dmax = funkey(__reduce_max_sync(kFull, fkey(dmax)));
        float *sc = (float *)red();
        if ((threadIdx.x & 31) == 0) sc[threadIdx.x >> 5] = dmax;
        __syncthreads();
        if (threadIdx.x == 0) {
          denmax = 0.0f;
          for (int w = 0; w < (int)(blockDim.x >> 5); ++w) denmax = fmaxf(denmax, sc[w]);
        }
        __syncthreads();
      }
      const int maxIt = pr.iters[level];
      int it = 0;
      float cv = 1e10f;
      if (level == 0 && job.warm && maxIt > 0) {
        // warm start: one iteration from the warm lattice and one from zero;
        // keep the one whose first convergence value is not larger.  Each
        // arm starts from a reset and leaves logU one update (D, in Gd)
        // behind L, as the main loop expects after an iteration.
        float cvs[2];
        for (int arm = 0; arm < 2; ++arm) {
          for (int c = threadIdx.x; c < nlat; c += blockDim.x) L()[c] = arm == 0 ? job.warm[c] : 0.0f;
          __syncthreads();
          if (arm == 1) reset(L());   // arm 0 starts from the level's reset (L = warm)
          if (!pass_a(false, false)) goto timeout;
          if (!fit_step(false)) goto timeout;
          if (!pass_a(true, false)) goto timeout;   // the update's CV; logU not advanced
          cvs[arm] = iter().cv;
          // the next pass A writes the CTAs' sums again: not before every CTA
          // has read them (a CTA that read others would take the other arm)
          if (!g.sync()) goto timeout;
          if (arm == 0) {   // keep the warm result in aux, its update in tmp
            for (int c = threadIdx.x; c < nlat; c += blockDim.x) { aux()[c] = L()[c]; tmp()[c] = D()[c]; }
          }
          __syncthreads();
        }
        const bool use_warm = cvs[0] <= cvs[1];
        if (use_warm) {
          // logU back to the warm lattice, L and D to the warm arm's update
          reset(job.warm);
          for (int c = threadIdx.x; c < nlat; c += blockDim.x) { L()[c] = aux()[c]; D()[c] = tmp()[c]; }
          __syncthreads();
        }
        // pass A left the histogram copies in the Gd region
        if (use_warm) rowtab_planes(D());
        else rowtab(D());
        __syncthreads();
        cv = use_warm ? cvs[0] : cvs[1];
        it = 1;
        if (lead) {
          rep->warm_start_used = use_warm ? 1 : 0;
          rep->first_cv_warm = cvs[0];
          rep->first_cv_plain = cvs[1];
        }
      }
      N4_MARK(PH_SETUP);
      for (;;) {
        if (!pass_a(it > 0, it > 0)) goto timeout;   // applies the last update
        N4_MARK(PH_A);
        if (it > 0) cv = iter().cv;
        if (!((double)cv > pr.thr) || it >= maxIt) break;
        if (!fit_step()) goto timeout;
        ++it;
      }
      if (lead) { rep->iterations[level] = it; rep->final_cv[level] = cv; rep->levels = level + 1; }
    }
    if (rank == 0) {
      for (int c = threadIdx.x; c < nlat; c += blockDim.x) job.lattice_out[c] = L()[c];
      if (threadIdx.x == 0) { rep->status = N4_OK; rep->device_end_ns = global_ns(); }
    }
#ifdef N4_PHASE_TIMERS
    if (threadIdx.x == 0 && (rank == 0 || rank == K / 2))
      printf("N4PHASE K=%d nt=%d rank=%d rows=%d setup=%lld A=%lld Aloop=%lld Ared=%lld Bloop=%lld Bmerge=%lld Bred=%lld "
             "sharp=%lld T1=%lld T2=%lld P=%lld Fred=%lld update=%lld\n",
             K, (int)blockDim.x, rank, nact, ph_acc[PH_SETUP], ph_acc[PH_A], ph_acc[PH_A_LOOP], ph_acc[PH_A_RED],
             ph_acc[PH_B_LOOP], ph_acc[PH_B_MERGE], ph_acc[PH_B_RED], ph_acc[PH_SHARP], ph_acc[PH_F_T1],
             ph_acc[PH_F_T2], ph_acc[PH_F_P], ph_acc[PH_F_RED], ph_acc[PH_UPDATE]);
#endif
    return;
  timeout:
    if (lead) rep->status = N4_ERR_TIMEOUT;
  }
};

// Sum over a cluster's partials of one entry: exact for the integer
// histogram, Kahan-compensated for the fit's float partials.
template <class Group>
template <class T>
struct Engine<Group>::SumOf {
  T s = 0;
  KahanSum k;
  __device__ __forceinline__ void add(T x) {
    if constexpr (sizeof(T) == 4) k.add(x);
    else s += x;
  }
  __device__ __forceinline__ T value() const {
    if constexpr (sizeof(T) == 4) return k.value();
    else return s;
  }
};

// Shared-memory home of a CTA's Engine on the whole-GPU path: thread 0
// constructs it, then every thread of the CTA uses the same object.
template <class Group>
struct EngineSlot {
  static_assert(Engine<Group>::kShared, "only the whole-GPU path keeps its Engine in shared memory");
  alignas(16) unsigned char raw[sizeof(Engine<Group>)];
  __device__ Engine<Group> &make(const Group &g, const Plan &p, const Params &r, char *big) {
    if (threadIdx.x == 0) new (raw) Engine<Group>(g, p, r, big);
    __syncthreads();
    return *reinterpret_cast<Engine<Group> *>(raw);
  }
};

}  // namespace n4
