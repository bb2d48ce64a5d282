// The vlp4d_mpi step for one process (miniapps/vlp4d_mpi, Timestep.hpp:34-97
// without LAG_ORDER: cubic B-spline interpolation), FP64.
//
// Arrays are the reference's halo-extended views (RealView4D with offsets,
// Init.cpp:333-343): extents n[d] + 6 in every dimension, first index -3
// (HALO_PTS = 3), layout_left.  The step:
//   halo fill     periodic images; the outermost layer holds the sums
//                 sum_{j=1..8} alpha^j f(...) that stand in for the rest of
//                 the periodic line (Communication.hpp:756-896)
//   spline xy     cubic B-spline prefilter along x, then y (Spline.hpp:114-198)
//   advect 2D     x, y shift by dt/2 through the 4x4 spline (Advection.hpp
//                 thrust :95-226); only its velocity moment is used
//   field         rho, Poisson solve (the context's FP64 cuFFT solver)
//   spline vxvy   the prefilter along vx, then vy (Spline.hpp:429-469)
//   advect 4D     predictor-corrector foot with the field interpolated by
//                 3-point Lagrange, then the 4^4 spline interpolation
//                 (Advection.hpp thrust :228-415)
//   field, diagnostics and L2 norm of the new state.
//
// Two families of kernels:
// * the reference-facing entry points (vlp4d_mpi_halo_fill, _spline_xy,
//   _spline_vxvy, _advect_2d, _advect_4d) run the reference's arithmetic in
//   its order with every product and sum rounded separately (no contracted
//   FMA, as the reference's x86-64 build computes), so they reproduce it bit
//   for bit;
// * vlp4d_mpi_step fuses the sequence into four passes over f: the x/y pass
//   builds each (vx, vy) plane's halo in shared memory, prefilters it,
//   writes its coefficients and evaluates the 2D advection straight into
//   the velocity moment; the vx and vy passes extend and prefilter the v
//   lines; the 4D pass interpolates and accumulates the moment and the L2
//   norm of the new state.  Its arithmetic uses FMA and its own summation
//   order: equal to the reference up to rounding.
#include <cmath>
#include <cstdlib>
#include <type_traits>
#include <vector>

#include "internal.cuh"

namespace vlp4d {
namespace {

constexpr int kH = 3;     // HALO_PTS
constexpr int kMmax = 8;  // terms of a boundary sum (MMAX)

// Geometry of the halo-extended array.
struct HGrid {
  int n[4];
  long long e[4];  // n + 6
  long long s[4];  // strides: 1, e0, e0 e1, e0 e1 e2
  int is[4];       // the same strides as int (a stride of 2^31 would be an array of 270 GB)
  double minp[4], maxp[4], dx[4], inv_dx[4];
  // Admissible feet of the 4D advection (Advection.hpp thrust :249-250):
  // [min + local_min*h - h, min + local_max*h + h] with local = 0..n-1.
  double lo[4], hi[4];
  // The clamp of the v feet, min + (max - min) (Advection.hpp thrust :307-308).
  double vtop[4];
  double alpha, beta, sqrt3;
  __host__ __device__ long long at(int x, int y, int vx, int vy) const {
    return (long long)(x + kH) + s[1] * (y + kH) + s[2] * (vx + kH) + s[3] * (vy + kH);
  }
  __host__ __device__ long long total() const { return e[0] * e[1] * e[2] * e[3]; }
};

HGrid make_hgrid(const vlp4d_ctx *c) {
  HGrid h;
  for (int k = 0; k < 4; ++k) {
    h.n[k] = c->g.n[k];
    h.e[k] = c->g.n[k] + 2 * kH;
    h.minp[k] = c->g.minp[k];
    h.maxp[k] = c->g.maxp[k];
    h.dx[k] = c->g.dx[k];
    h.inv_dx[k] = 1. / c->g.dx[k];
    h.lo[k] = c->g.minp[k] + 0 * c->g.dx[k] - c->g.dx[k];
    h.hi[k] = c->g.minp[k] + (c->g.n[k] - 1) * c->g.dx[k] + c->g.dx[k];
    h.vtop[k] = c->g.minp[k] + (c->g.maxp[k] - c->g.minp[k]);
  }
  h.s[0] = 1;
  h.s[1] = h.e[0];
  h.s[2] = h.e[0] * h.e[1];
  h.s[3] = h.s[2] * h.e[2];
  for (int k = 0; k < 4; ++k) h.is[k] = (int)h.s[k];
  // Spline.hpp:21,36-37: sqrt3 = sqrt(3), alpha = sqrt3 - 2,
  // beta = sqrt3 * (1 - alpha*alpha) (host IEEE arithmetic).
  h.sqrt3 = std::sqrt(3.0);
  h.alpha = h.sqrt3 - 2.;
  h.beta = h.sqrt3 * (1. - h.alpha * h.alpha);
  return h;
}

// Equal (x, y) tiles of at most 32 columns and 256 points, a thread per point (a
// fixed 32 x 8 leaves 22 lanes of 32 idle at nx = 10).  `rows`: a warp per row
// of 32 columns where that leaves less than a fifth of the lanes idle.
struct PlaneTiles {
  int W, H, nxt, nyt, threads;
  PlaneTiles(const HGrid &h, bool rows) {
    nxt = (h.n[0] + 31) / 32;
    W = rows && 5 * h.n[0] >= 4 * 32 * nxt ? 32 : (h.n[0] + nxt - 1) / nxt;
    nyt = (h.n[1] + 256 / W - 1) / (256 / W);
    H = (h.n[1] + nyt - 1) / nyt;
    threads = (W * H + 31) / 32 * 32;
  }
};

__device__ __forceinline__ int wrapi(int i, int n) { return ((i % n) + n) % n; }
// The same for i in [-n, 2 n).
__device__ __forceinline__ int wrap1(int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); }

// Separately rounded arithmetic (the reference's x86-64 build has no FMA).
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }

// 8-byte asynchronous global-to-shared copies (through L1), one commit group
// per call site, waited for before the data is read.
__device__ __forceinline__ void cp_async8(double *dst, const double *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;" ::: "memory");
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// ---------------------------------------------------------------------------
// Halo fill of one process (Communication.hpp:713-754 through the local
// copy; boundary_condition :756-896; point lists of listBoundary :128-440).
// A halo point whose coordinates all lie in [-2, n+1] takes the periodic
// image.  A point in the outermost layer (-3 or n+2) of the dimensions B
// takes sum_{j_k=1..MMAX, k in B} alpha^(sum j_k) f(r + sum_k s_k j_k e_k),
// s_k = -1 (left layer) or +1 (right), r_k = (c_k - s_k) mod n_k for k in B
// and c_k mod n_k otherwise, with the highest dimension of B in the outer
// loop and the powers of alpha built by repeated products, as the
// reference does.  Every grid dimension is at least MMAX + 2 = 10, so the
// sums read interior points only.
// The order of a sum is the reference's, one addition after another, so a
// corner of all four dimensions is a chain of 8^4 additions.  The kernel
// gives each kind of point (the set B) its own blocks, the longest chains
// first: B of four dimensions a block per point and of three a warp per
// point, the products formed by all threads in shared memory and added by
// one; B of two and one a thread per point; B empty a copy.  One thread per
// point of any kind, in the order of memory, left whole warps and at last
// one block waiting for a corner's 4096 dependent loads: 2.58 ms on
// 48 x 44 x 40 x 36 against 0.054 ms here (0.067 before the point's coordinates
// were taken apart in 32 bits and the loads of the sums and copies ran ahead);
// a corner's chain alone is 0.031 (10^4).
constexpr int kHaloThreads = 256;

struct HaloParts {
  unsigned char mask[16];  // B as a bit mask
  int first[17];           // first block of each part
  int parts;
};

// Product weight of the term (j_0, .., j_{m-1}), by the reference's repeated
// products.
__device__ double halo_weight(int m, int idx, double alpha) {
  double w = alpha;
  for (int l = m - 1; l >= 0; --l) {
    if (l < m - 1) w = mul(alpha, w);
    for (int t = (idx >> (3 * l)) & 7; t > 0; --t) w = mul(w, alpha);
  }
  return w;
}

__global__ void __launch_bounds__(kHaloThreads) k_mpi_halo(double *__restrict__ f, HGrid h, HaloParts P) {
  __shared__ __align__(16) double prod[4096];
  int part = 0;
  while (part + 1 < P.parts && (int)blockIdx.x >= P.first[part + 1]) ++part;
  const int mask = P.mask[part];
  const unsigned blk = blockIdx.x - P.first[part];
  if (mask == 0) {
    // Periodic images: one block per (vx, vy) of [-2, n + 1]; where both are
    // grid coordinates, only the two points around the (x, y) plane.
    const int cvx = (int)(blk % (h.n[2] + 4)) - 2, cvy = (int)(blk / (h.n[2] + 4)) - 2;
    const bool vin = cvx >= 0 && cvx < h.n[2] && cvy >= 0 && cvy < h.n[3];
    const int m0 = h.n[0] + 4, m1 = h.n[1] + 4;
    const int full = vin ? 4 * m0 : m0 * m1;
    const int count = vin ? full + 4 * h.n[1] : full;
    const double *src = f + h.at(0, 0, wrap1(cvx, h.n[2]), wrap1(cvy, h.n[3]));
    double *dst = f + h.at(0, 0, cvx, cvy);
    // Four points of a thread at a time, their loads ahead of their stores.
    for (int t0 = threadIdx.x; t0 < count; t0 += 4 * kHaloThreads) {
      double v[4];
      int to[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int t = t0 + j * kHaloThreads;
        if (t >= count) break;
        int cx, cy;
        if (t < full) {  // whole rows
          const int r = t / m0;
          cx = t - r * m0 - 2;
          cy = !vin || r < 2 ? r - 2 : h.n[1] + r - 2;
        } else {  // two columns on each side of the grid's rows
          const int k = (t - full) & 3;
          cy = (t - full) >> 2;
          cx = k < 2 ? k - 2 : h.n[0] + k - 2;
        }
        to[j] = cx + h.is[1] * cy;
        v[j] = src[wrap1(cx, h.n[0]) + h.is[1] * wrap1(cy, h.n[1])];
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (t0 + j * kHaloThreads < count) dst[to[j]] = v[j];
    }
    return;
  }
  const int m = __popc(mask);
  // Point index: a block, a warp or a thread each.
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned idx = m == 4 ? blk : (m == 3 ? blk * (kHaloThreads / 32) + warp : blk * kHaloThreads + threadIdx.x);
  unsigned total = 1u << m, i = idx;  // 2^32 points of one kind would be an array of 270 GB
  int c[4], st[4] = {0, 0, 0, 0};
  long long base = 0;  // of the sums: their terms are at base + sum_l st[l] j_l
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    c[k] = 0;
    if (!((mask >> k) & 1)) {
      const unsigned ext = (unsigned)h.n[k] + 4;
      const unsigned q = i / ext;
      c[k] = (int)(i - q * ext) - 2;
      i = q;
      total *= ext;
      base += h.s[k] * (wrap1(c[k], h.n[k]) + kH);
    }
  }
  int l = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if ((mask >> k) & 1) {
      const int sg = (i >> l) & 1 ? 1 : -1;
      c[k] = sg < 0 ? -kH : h.n[k] + kH - 1;
      base += h.s[k] * (wrap1(c[k] - sg, h.n[k]) + kH);
      const int step = sg * h.is[k];
      if (l == 0) st[0] = step;
      else if (l == 1) st[1] = step;
      else if (l == 2) st[2] = step;
      else st[3] = step;
      ++l;
    }
  const bool on = idx < total;
  const double *p = f + base;
  double sum = 0.;
  if (m >= 3) {
    const int terms = 1 << (3 * m), stride = m == 4 ? kHaloThreads : 32;
    double *pr = m == 4 ? prod : prod + warp * 512;
    const int me = m == 4 ? (int)threadIdx.x : lane;
    if (on) {
#pragma unroll 4
      for (int t = me; t < terms; t += stride) {
        const double v = p[(long long)((t & 7) + 1) * st[0] + (long long)(((t >> 3) & 7) + 1) * st[1] +
                           (long long)(((t >> 6) & 7) + 1) * st[2] + (m == 4 ? (long long)((t >> 9) + 1) * st[3] : 0)];
        pr[t] = mul(v, halo_weight(m, t, h.alpha));
      }
    }
    if (m == 4) __syncthreads();
    else __syncwarp();
    if (me != 0 || !on) return;
    // The next sixteen products are on their way while sixteen are added.
    const double2 *q = (const double2 *)pr;
    double2 a[8], b[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] = q[k];
    for (int t = 0; t < terms; t += 32) {
#pragma unroll
      for (int k = 0; k < 8; ++k) b[k] = q[t / 2 + 8 + k];
#pragma unroll
      for (int k = 0; k < 8; ++k) sum = add(add(sum, a[k].x), a[k].y);
      const int n = t + 32 < terms ? t / 2 + 16 : 0;
#pragma unroll
      for (int k = 0; k < 8; ++k) a[k] = q[n + k];
#pragma unroll
      for (int k = 0; k < 8; ++k) sum = add(add(sum, b[k].x), b[k].y);
    }
  } else if (m == 2) {
    if (!on) return;
    double w1 = h.alpha;
#pragma unroll 2
    for (int j1 = 1; j1 <= kMmax; ++j1) {
      double v[kMmax], w0 = mul(h.alpha, w1);
#pragma unroll
      for (int j = 0; j < kMmax; ++j) v[j] = p[(long long)j1 * st[1] + (long long)(j + 1) * st[0]];
#pragma unroll
      for (int j = 0; j < kMmax; ++j) {
        sum = add(sum, mul(v[j], w0));
        w0 = mul(w0, h.alpha);
      }
      w1 = mul(w1, h.alpha);
    }
  } else {
    if (!on) return;
    double v[kMmax], w0 = h.alpha;
#pragma unroll
    for (int j = 0; j < kMmax; ++j) v[j] = p[(long long)(j + 1) * st[0]];
#pragma unroll
    for (int j = 0; j < kMmax; ++j) {
      sum = add(sum, mul(v[j], w0));
      w0 = mul(w0, h.alpha);
    }
  }
  f[h.at(c[0], c[1], c[2], c[3])] = sum;
}

// ---------------------------------------------------------------------------
// The prefilter of one extended line (Spline.hpp:114-198, LONG_ENOUGH_BUFFER
// form): e[0] and e[L+1] hold the boundary sums, e[1..L] the points -2..n+1
// (L = n + 4).  e[1..L] become the spline coefficients; e[0], e[L+1] stay.
//   causal:      t[0] = e[0] + e[1],  t[k] = e[1+k] + alpha t[k-1]
//   right end:   c[L] = sqrt3 (e[L+1] + sum_{k=0..L-1} alpha^k e[L-k])
//   anticausal:  c[i] = beta t[i-1] + alpha c[i+1]
// In place: t[k-1] is stored at e[k] once e[k] has been read; products and
// sums rounded separately, the right-end sum from the original values.
__device__ __forceinline__ void spline_line(double *__restrict__ e, long long st, int L, double alpha, double beta,
                                            double sqrt3) {
  double acc = add(e[(long long)(L + 1) * st], e[(long long)L * st]);
  double ak = alpha;
  for (int k = 1; k < L; ++k) {
    acc = add(acc, mul(e[(long long)(L - k) * st], ak));
    ak = mul(ak, alpha);
  }
  double t = add(e[0], e[st]);
  e[st] = t;
  for (int k = 1; k < L - 1; ++k) {
    t = add(e[(long long)(1 + k) * st], mul(alpha, t));
    e[(long long)(1 + k) * st] = t;
  }
  double c = mul(acc, sqrt3);
  e[(long long)L * st] = c;
  for (int i = L - 1; i >= 1; --i) {
    c = add(mul(beta, e[(long long)i * st]), mul(alpha, c));
    e[(long long)i * st] = c;
  }
}

// The fused step's prefilter splits a line of L = n + 4 points into segments
// of S consecutive points, each in one thread's registers: a first-order
// recursion y_k = x_k + alpha y_{k-1} over a segment needs only the last
// value c of the segment before, y_k(segment) + alpha^(k+1) c, and those
// follow from the segments' own last values with the factor alpha^S.  Equal
// to the recursion along the whole line up to rounding; the chain is S + the
// number of segments instead of 2 L.  Extension included: the points
// -2, -1, n, n+1 are read as their periodic images, the boundary sums e0, eR
// (points -3 and n+2) are formed from the line.
constexpr double kAlpha = 1.7320508075688772 - 2.;  // sqrt(3) - 2
__host__ __device__ constexpr double alpha_pow(int k) {
  double r = 1.;
  for (int i = 0; i < k; ++i) r *= kAlpha;
  return r;
}
// alpha^0 .. alpha^17 as operands from constant memory.
__constant__ double kAlphaPow[18] = {alpha_pow(0),  alpha_pow(1),  alpha_pow(2),  alpha_pow(3),  alpha_pow(4),
                                     alpha_pow(5),  alpha_pow(6),  alpha_pow(7),  alpha_pow(8),  alpha_pow(9),
                                     alpha_pow(10), alpha_pow(11), alpha_pow(12), alpha_pow(13), alpha_pow(14),
                                     alpha_pow(15), alpha_pow(16), alpha_pow(17)};

// The segments are aligned to the line's right end: position L is the last
// point of the last one.  Position 0 holds e0 / alpha (the causal pass starts
// from t_1 = x_1 + e0), positions before it 0.
template <int S>
__device__ __forceinline__ void seg_causal(double v[S]) {
#pragma unroll
  for (int j = 1; j < S; ++j) v[j] = fma(kAlphaPow[1], v[j - 1], v[j]);
}
template <int S>
__device__ __forceinline__ void seg_causal_carry(double v[S], double c) {
#pragma unroll
  for (int j = 0; j < S; ++j) v[j] = fma(kAlphaPow[j + 1], c, v[j]);
}
// Between the passes: beta t below position L; at L (the last point of the
// `last` segment) c[L] = sqrt3 (eR + the right-end sum, which is the causal
// value without e0's part; aL = alpha^(L-1)).
template <int S>
__device__ __forceinline__ void seg_turn(double v[S], bool last, double beta, double sqrt3, double e0, double eR,
                                         double aL) {
  const double cL = (eR + fma(-aL, e0, v[S - 1])) * sqrt3;
#pragma unroll
  for (int j = 0; j < S; ++j) v[j] *= beta;
  if (last) v[S - 1] = cL;
}
template <int S>
__device__ __forceinline__ void seg_anticausal(double v[S]) {
#pragma unroll
  for (int j = S - 2; j >= 0; --j) v[j] = fma(kAlphaPow[1], v[j + 1], v[j]);
}
template <int S>
__device__ __forceinline__ void seg_anticausal_carry(double v[S], double c) {
#pragma unroll
  for (int j = 0; j < S; ++j) v[j] = fma(kAlphaPow[S - j], c, v[j]);
}

// Cubic B-spline weights at fractional offset w (Advection.hpp:127-144),
// in the reference's order of operations.
template <bool EXACT>
__device__ __forceinline__ void bspline_w(double w, double eta[4]) {
  if (EXACT) {
    const double e3 = mul(mul(mul(1. / 6., w), w), w);
    const double e0 = sub(add(1. / 6., mul(mul(0.5, w), sub(w, 1.))), e3);
    const double e2 = sub(add(w, e0), mul(2., e3));
    const double e1 = sub(sub(sub(1., e0), e2), e3);
    eta[0] = e0;
    eta[1] = e1;
    eta[2] = e2;
    eta[3] = e3;
  } else {
    const double e3 = (1. / 6.) * w * w * w;
    const double e0 = (1. / 6.) + 0.5 * w * (w - 1.) - e3;
    const double e2 = w + e0 - 2. * e3;
    eta[0] = e0;
    eta[1] = 1. - e0 - e2 - e3;
    eta[2] = e2;
    eta[3] = e3;
  }
}

}  // namespace
}  // namespace vlp4d

namespace vlp4d {
namespace {

// ---------------------------------------------------------------------------
// Plane kernels.  A (vx, vy) plane of the extended array lives in shared
// memory with an odd row stride P >= nx + 6 (row r = y + 3, column c = x + 3):
// a thread walking a row and its neighbour walking the next row then hit
// different banks.

// Lines of a plane in shared memory, extended and prefiltered in place: line
// l (of `lines`) starts at pl + l * ls, position k of it (0 .. n + 5) is st * k
// further; positions 3 .. n + 2 are given, all are written.  G lanes share a
// line, S points each (G S >= n + 4).  The left boundary sum e0 enters the
// causal pass at position 0, which the segments hold where G S > n + 4; where
// they fill the line exactly (n = 36, 68, 100, 132, 268, 540) lane 0 starts at
// position 1 and adds e0 there.  Lines outside [flo, fhi] are extended only.
// aL = alpha^(n + 3).
template <int S, int G, int ST>
__device__ __noinline__ void plane_lines(double *pl, int st_, int ls, int n, int lines, int flo, int fhi, double beta,
                                         double sqrt3, double aL) {
  const int st = ST ? ST : st_;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  constexpr int kPer = 32 / G;
  const int g = lane % G, sub = lane / G;
  const int k0 = n + 5 - (G - g) * S;  // L = n + 4
  double aw = kAlpha;  // alpha^(g mod 8 + 1): this lane's term of the boundary sums
  for (int t = 0; t < (g & 7); ++t) aw *= kAlpha;
  // The image this lane copies: positions 1, 2 <- n+1, n+2; n+3, n+4 <- 3, 4.
  const int to = g < 2 ? 1 + g : n + 1 + g, from = g < 2 ? n + 1 + g : 1 + g;
  for (int l0 = warp * kPer; l0 < lines; l0 += nwarps * kPer) {
    const int l = l0 + sub;
    const bool on = l < lines;
    const bool filter = l >= flo && l <= fhi;
    double *p = pl + (on ? l : lines - 1) * ls;
    // left: sum_j alpha^j f(n-2-j) (position n+1-j); right: f(1+j) (4+j)
    double e0 = aw * p[(n - (g & 7)) * st], eR = aw * p[(5 + (g & 7)) * st];
#pragma unroll
    for (int d = 4; d > 0; d >>= 1) {
      e0 += __shfl_xor_sync(0xffffffffu, e0, d);
      eR += __shfl_xor_sync(0xffffffffu, eR, d);
    }
    if (on && g < 4) p[to * st] = p[from * st];
    if (on && g == 4) p[0] = filter ? e0 * (1. / kAlpha) : e0;
    if (on && g == 5) p[(n + 5) * st] = eR;
    __syncwarp();
    double v[S];
    double *q = p + k0 * st;
#pragma unroll
    for (int j = 0; j < S; ++j) v[j] = k0 + j >= 0 ? q[j * st] : 0.;
    if (g == 0 && k0 == 1) v[0] += e0;  // no lane holds position 0
    seg_causal<S>(v);
    // The lanes' last values, summed up with alpha^S per lane.
    double x = v[S - 1], A = alpha_pow(S);
#pragma unroll
    for (int d = 1; d < G; d <<= 1) {
      const double y = __shfl_up_sync(0xffffffffu, x, d, G);
      if (g >= d) x = fma(A, y, x);
      A *= A;
    }
    x = __shfl_up_sync(0xffffffffu, x, 1, G);
    seg_causal_carry<S>(v, g ? x : 0.);
    seg_turn<S>(v, g == G - 1, beta, sqrt3, e0, eR, aL);
    seg_anticausal<S>(v);
    x = v[0];
    A = alpha_pow(S);
#pragma unroll
    for (int d = 1; d < G; d <<= 1) {
      const double y = __shfl_down_sync(0xffffffffu, x, d, G);
      if (g + d < G) x = fma(A, y, x);
      A *= A;
    }
    x = __shfl_down_sync(0xffffffffu, x, 1, G);
    seg_anticausal_carry<S>(v, g < G - 1 ? x : 0.);
    __syncwarp();  // every lane of the line has read it
    if (on && filter) {
#pragma unroll
      for (int j = 0; j < S; ++j)
        if (k0 + j >= 1) q[j * st] = v[j];
      if (g == 0) p[0] = e0;
    }
    __syncwarp();
  }
}

// The same with one thread per line, for lines too long for 32 segments of 17.
__device__ __noinline__ void plane_lines_long(double *pl, int st, int ls, int n, int lines, int flo, int fhi,
                                              double beta, double sqrt3) {
  for (int l = threadIdx.x; l < lines; l += blockDim.x) {
    double *p = pl + l * ls;
    double w = kAlpha, e0 = 0., eR = 0.;
    for (int j = 1; j <= kMmax; ++j) {
      e0 = fma(p[(n + 1 - j) * st], w, e0);
      eR = fma(p[(4 + j) * st], w, eR);
      w *= kAlpha;
    }
    p[0] = e0;
    p[st] = p[(n + 1) * st];
    p[2 * st] = p[(n + 2) * st];
    p[(n + 3) * st] = p[3 * st];
    p[(n + 4) * st] = p[4 * st];
    p[(n + 5) * st] = eR;
    if (l >= flo && l <= fhi) spline_line(p, st, n + 4, kAlpha, beta, sqrt3);
  }
}

// S points per lane and G lanes per line for lines of n + 4 points (odd S:
// the lanes of a line fall on distinct shared-memory banks).
template <int ST>
__device__ __forceinline__ void plane_lines_any(double *pl, int st, int ls, int n, int lines, int flo, int fhi,
                                                double beta, double sqrt3, double aL) {
  const int L = n + 4;
  if (L <= 40) plane_lines<5, 8, ST>(pl, st, ls, n, lines, flo, fhi, beta, sqrt3, aL);
  else if (L <= 72) plane_lines<9, 8, ST>(pl, st, ls, n, lines, flo, fhi, beta, sqrt3, aL);
  else if (L <= 104) plane_lines<13, 8, ST>(pl, st, ls, n, lines, flo, fhi, beta, sqrt3, aL);
  else if (L <= 136) plane_lines<17, 8, ST>(pl, st, ls, n, lines, flo, fhi, beta, sqrt3, aL);
  else if (L <= 272) plane_lines<17, 16, ST>(pl, st, ls, n, lines, flo, fhi, beta, sqrt3, aL);
  else if (L <= 544) plane_lines<17, 32, ST>(pl, st, ls, n, lines, flo, fhi, beta, sqrt3, aL);
  else plane_lines_long(pl, st, ls, n, lines, flo, fhi, beta, sqrt3);
}

// Spline::computeCoeff_xy on every plane of a halo-filled array, in place,
// in the reference's arithmetic.
__global__ void __launch_bounds__(256) k_mpi_spline_xy(double *__restrict__ f, HGrid h, int P) {
  extern __shared__ __align__(16) double pl[];
  const int E0 = h.n[0] + 2 * kH, E1 = h.n[1] + 2 * kH;
  const long long planes = h.e[2] * h.e[3];
  for (long long p = blockIdx.x; p < planes; p += gridDim.x) {
    double *g = f + p * h.s[2];
    for (int r = threadIdx.y; r < E1; r += blockDim.y)
      for (int c = threadIdx.x; c < E0; c += blockDim.x) cp_async8(pl + r * P + c, g + (long long)r * E0 + c);
    cp_async_wait_all();
    __syncthreads();
    const int tid = threadIdx.y * blockDim.x + threadIdx.x, nt = blockDim.x * blockDim.y;
    for (int r = tid; r < E1; r += nt) spline_line(pl + (long long)r * P, 1, h.n[0] + 4, h.alpha, h.beta, h.sqrt3);
    __syncthreads();
    for (int c = 1 + tid; c < E0 - 1; c += nt) spline_line(pl + c, P, h.n[1] + 4, h.alpha, h.beta, h.sqrt3);
    __syncthreads();
    for (int r = threadIdx.y; r < E1; r += blockDim.y)
      for (int c = threadIdx.x; c < E0; c += blockDim.x) g[(long long)r * E0 + c] = pl[r * P + c];
    __syncthreads();
  }
}

// The fused x/y pass of vlp4d_mpi_step.  Each CTA takes the interior
// (vx, vy) planes p = blockIdx.x, blockIdx.x + gridDim.x, ...: loads the
// plane's grid points from fn, builds its halo, prefilters it, writes the
// coefficients of the whole extended plane into cxy, and evaluates the 2D
// advection by dt (Advection.hpp thrust :131-214) at every grid point,
// adding it to the thread's moment accumulators, planes in a fixed order.
// Thread t owns the CPT cells of column t % nx, rows (t / nx) * CPT ..;
// it walks them with a sliding window of four x sums, so a cell costs
// about 4 shared-memory loads instead of 16.  With the prefilter's lines
// split into segments (plane_lines) the pass takes 2.22 ms at 128^4 against
// 4.13 with one thread per line (70 of 512 threads at work at 64^2); one
// 145 KB plane per SM: the load of the plane and the barriers between the
// phases are exposed (1.9 TB/s).  The accumulators go to
// part[blockIdx.x][ix + nx*iy] at the end.  A foot outside the spline's
// range sets bit 2 of *err (the reference stops: "Time step is too
// large").
template <int CPT>
__global__ void __launch_bounds__(512) k_mpi_xy_pass(const double *__restrict__ fn, double *__restrict__ cxy,
                                                     HGrid h, int P, double dt, double aLx, double aLy,
                                                     double *__restrict__ part, int *__restrict__ err) {
  extern __shared__ __align__(16) double pl[];
  const int nx = h.n[0], ny = h.n[1], nvx = h.n[2];
  const int E0 = nx + 2 * kH, E1 = ny + 2 * kH;
  const int nxy = nx * ny;
  const long long planes = (long long)nvx * h.n[3];
  double acc[CPT];
#pragma unroll
  for (int k = 0; k < CPT; ++k) acc[k] = 0.;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  // This thread's strip of the 2D advection: column ix, rows iy0 .. iy0+CPT-1.
  const int ix = threadIdx.x % nx, iy0 = (threadIdx.x / nx) * CPT;
  const bool own = iy0 < ny;
  bool bad = false;
  for (long long p = blockIdx.x; p < planes; p += gridDim.x) {
    const int ivx = (int)(p % nvx), ivy = (int)(p / nvx);
    {
      const double *src = fn + h.at(0, 0, ivx, ivy) + (long long)warp * E0 + lane;
      double *d = pl + (warp + kH) * P + kH + lane;
      for (int iy = warp; iy < ny; iy += nwarps, src += (long long)nwarps * E0, d += nwarps * P) {
#pragma unroll 4
        for (int ix = 0; ix < nx; ix += 32)
          if (ix + lane < nx) cp_async8(d + ix, src + ix);
      }
    }
    cp_async_wait_all();
    __syncthreads();
    // x lines of the grid's rows, then y lines of every column (the first
    // and last extended only, as the reference's column update leaves them;
    // the rows above and below come out as the y sums of x lines).
    plane_lines_any<1>(pl + kH * P, 1, P, nx, ny, 0, ny - 1, h.beta, h.sqrt3, aLx);
    __syncthreads();
    plane_lines_any<0>(pl, P, 1, ny, E0, 1, E0 - 2, h.beta, h.sqrt3, aLy);
    __syncthreads();
    {
      double *dst = cxy + h.at(-kH, -kH, ivx, ivy) + (long long)warp * E0 + lane;
      const double *q = pl + warp * P + lane;
      for (int r = warp; r < E1; r += nwarps, dst += (long long)nwarps * E0, q += nwarps * P) {
#pragma unroll 4
        for (int k = 0; k < E0; k += 32)
          if (k + lane < E0) dst[k] = q[k];
      }
    }
    // 2D advection at the grid points of the plane, from the coefficients.
    // The shift (dt vx, dt vy) is the same for the whole plane: one cell
    // offset and one set of weights per direction (the reference evaluates
    // them per cell; they differ only by the rounding of x_i - dt vx).
    const double vx = h.minp[2] + ivx * h.dx[2], vy = h.minp[3] + ivy * h.dx[3];
    const double fx = -dt * vx * h.inv_dx[0], fy = -dt * vy * h.inv_dx[1];
    const int mx = (int)floor(fx), my = (int)floor(fy);
    if (mx < -1 || mx > 0 || my < -1 || my > 0) bad = true;  // i0 = ix + mx must stay in [-1, nx-1]
    double ex[4], ey[4];
    bspline_w<false>(fx - mx, ex);
    bspline_w<false>(fy - my, ey);
    if (!bad && own) {
      // x sums of rows iy0 + my - 1 + r (r = 0 .. CPT + 2), a window of four.
      const double *b = pl + (iy0 + my - 1 + kH) * P + (ix + mx - 1 + kH);
      double w0 = 0., w1 = 0., w2 = 0.;
      auto rows = [&](bool whole) {
#pragma unroll
        for (int r = 0; r < CPT + 3; ++r) {
          double w3 = 0.;
          if (whole || iy0 + r - 3 < ny) {  // row needed by some cell of the strip
            w3 = ex[0] * b[0] + ex[1] * b[1] + ex[2] * b[2] + ex[3] * b[3];
            b += P;
          }
          if (r >= 3 && (whole || iy0 + r - 3 < ny)) acc[r - 3] += ey[0] * w0 + ey[1] * w1 + ey[2] * w2 + ey[3] * w3;
          w0 = w1;
          w1 = w2;
          w2 = w3;
        }
      };
      if (iy0 + CPT <= ny) rows(true);
      else rows(false);
    }
    __syncthreads();
  }
  if (bad) atomicOr(err, 2);
  if (own) {
#pragma unroll
    for (int j = 0; j < CPT; ++j)
      if (iy0 + j < ny) part[(long long)blockIdx.x * nxy + ix + (long long)nx * (iy0 + j)] = acc[j];
  }
}

// ---------------------------------------------------------------------------
// v lines.  A warp takes a tile of 32 lines along dimension `dim` (2: vx,
// 3: vy) at 32 consecutive x positions and one (y, o) pair (o: the other v
// coordinate, in [olo, olo + no)); lane l owns the line at x = x0 + l, kept
// in shared memory as [position][lane] (conflict-free).  `in` may be `out`
// (each line is read before it is written, by its own lane).  EXTEND: the line's
// grid points (positions 0..n-1) come from `in` and its halo is built here
// (periodic images, boundary sums); otherwise all n + 6 positions come from
// `in` as they are.  Lines with o in [flo, fhi] are prefiltered (the
// reference's column update skips the outermost layer of the first v
// dimension, Spline.hpp:164).  All n + 6 positions go to `out`.
template <bool EXTEND>
__global__ void __launch_bounds__(128) k_mpi_vlines(const double *in, double *out, HGrid h,
                                                    int dim, int olo, int no, int flo, int fhi) {
  extern __shared__ __align__(16) double tiles[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int n = h.n[dim];
  const int E = n + 2 * kH;
  double *tile = tiles + (long long)warp * E * 32;
  const int odim = dim == 2 ? 3 : 2;
  const long long sl = h.s[dim], so = h.s[odim];
  const int xchunks = (int)((h.e[0] + 31) / 32);
  const long long ntiles = (long long)xchunks * h.e[1] * no;
  for (long long t = (long long)blockIdx.x * nwarps + warp; t < ntiles; t += (long long)gridDim.x * nwarps) {
    const int xc = (int)(t % xchunks);
    const long long r = t / xchunks;
    const int y = (int)(r % h.e[1]) - kH;
    const int o = (int)(r / h.e[1]) + olo;
    const int x = xc * 32 + lane - kH;
    const bool live = x < h.n[0] + kH;
    // Line base: position -3 of the line dimension.
    const long long base = (long long)(x + kH) + h.s[1] * (y + kH) + so * (o + kH);
    if (live) {
      if (EXTEND) {
        for (int i = 0; i < n; ++i) cp_async8(tile + (i + kH) * 32 + lane, in + base + (long long)(i + kH) * sl);
      } else {
        for (int i = 0; i < E; ++i) cp_async8(tile + i * 32 + lane, in + base + (long long)i * sl);
      }
    }
    cp_async_wait_all();
    __syncwarp();
    if (live) {
      double *col = tile + lane;
      if (EXTEND) {
        double wl = h.alpha, sL = 0., sR = 0.;
        for (int j = 1; j <= kMmax; ++j) {
          sL = fma(col[(n + 1 - j) * 32], wl, sL);
          sR = fma(col[(4 + j) * 32], wl, sR);
          wl *= h.alpha;
        }
        col[0] = sL;
        col[1 * 32] = col[(n + 1) * 32];
        col[2 * 32] = col[(n + 2) * 32];
        col[(n + 3) * 32] = col[3 * 32];
        col[(n + 4) * 32] = col[4 * 32];
        col[(n + 5) * 32] = sR;
      }
      if (o >= flo && o <= fhi) spline_line(col, 32, n + 4, h.alpha, h.beta, h.sqrt3);
      for (int i = 0; i < E; ++i) out[base + (long long)i * sl] = col[i * 32];
    }
    __syncwarp();
  }
}

// The fused step's v lines: a block takes 32 lines along `dim` at consecutive
// points of the extended (x, y) plane (contiguous in memory) and one o; warp w
// holds S consecutive points of its lane's line in registers,
// read and written straight from and to global memory in whole 256-byte rows,
// and the segments exchange one value per direction through shared memory.
// Bound by HBM: 0.78 ms per direction at 128^4, 5.9 TB/s (a lane per line with
// the tile in shared memory, its chain of 2 x 132 latencies: 1.49 ms).  Every point of the block's lines has been
// read at the first barrier, so `in` may be `out`.
template <int S, int NW>
__global__ void __launch_bounds__(NW * 32) k_mpi_vlines_seg(const double *in, double *out, HGrid h, int dim, int olo,
                                                            int flo, int fhi, double aL) {
  __shared__ double edge[NW][32], sum0[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int n = h.n[dim], k0 = n + 5 - (NW - w) * S;  // L = n + 4
  const long long sl = h.s[dim];
  const int o = olo + (int)blockIdx.y;
  const long long i = (long long)blockIdx.x * 32 + lane;
  const bool live = i < h.s[2];
  const long long base = i + h.s[dim == 2 ? 3 : 2] * (o + kH);
  const double *src = in + base;
  double v[S];
#pragma unroll
  for (int j = 0; j < S; ++j) {
    const int k = k0 + j;
    const int at = k < 3 ? k + n : (k >= n + 3 ? k - n : k);
    v[j] = live && k >= 1 ? src[at * sl] : 0.;
  }
  // The boundary sums: the left one by the warp that holds position 0 (or
  // whose first point is position 1), the right one by the last warp.
  const bool first = k0 <= 1 && k0 + S > 1, last = w == NW - 1;
  double e0 = 0., eR = 0.;
  if (first) {
#pragma unroll
    for (int j = 1; j <= kMmax; ++j) e0 = fma(alpha_pow(j), !live ? 0. : src[(n + 1 - j) * sl], e0);
    sum0[lane] = e0;
  }
  if (last) {
#pragma unroll
    for (int j = 1; j <= kMmax; ++j) eR = fma(alpha_pow(j), !live ? 0. : src[(4 + j) * sl], eR);
  }
  const bool filter = o >= flo && o <= fhi;
  if (filter) {
    if (first) {
#pragma unroll
      for (int j = 0; j < S; ++j)
        if (k0 + j == 1) v[j] += e0;
    }
    seg_causal<S>(v);
    edge[w][lane] = v[S - 1];
  }
  __syncthreads();
  if (filter) {
    double c = 0.;
    for (int q = 0; q < w; ++q) c = fma(alpha_pow(S), c, edge[q][lane]);
    seg_causal_carry<S>(v, c);
    seg_turn<S>(v, last, h.beta, h.sqrt3, sum0[lane], eR, aL);
    seg_anticausal<S>(v);
    __syncthreads();
    edge[w][lane] = v[0];
    __syncthreads();
    c = 0.;
    for (int q = NW - 1; q > w; --q) c = fma(alpha_pow(S), c, edge[q][lane]);
    seg_anticausal_carry<S>(v, c);
  }
  if (!live) return;
  double *dst = out + base;
#pragma unroll
  for (int j = 0; j < S; ++j)
    if (k0 + j >= 1) dst[(k0 + j) * sl] = v[j];
  if (first) dst[0] = e0;
  if (last) dst[(n + 5) * sl] = eR;
}

}  // namespace
}  // namespace vlp4d

namespace vlp4d {
namespace {

// ---------------------------------------------------------------------------
// Advection::advect_2D_xy (thrust Advection.hpp:95-226, spline branch
// :175-206) in the reference's arithmetic: fn's grid points receive the
// 4x4 spline interpolation of the coefficients in tmp at
// (x - dt vx, y - dt vy).  A foot outside [xmin-1, xmax] (in cells) sets
// bit 2 of *err and the point receives 0.
// A block is a tile of W x and H y (PlaneTiles), a thread takes the planes p = z,
// z + G, ...  With the call's copy, one box: 48 x 44 x 40 x 36 46 us, 10 x 92 x 112 x
// 23 43 (one thread per cell with its index taken apart by 64-bit divisions 63 and
// 52; blocks of 32 x 8 points 52 and 81).
__global__ void __launch_bounds__(256) k_mpi_advect_2d(const double *__restrict__ tmp, double *__restrict__ fn,
                                                       HGrid h, int W, int H, double dt, int *__restrict__ err) {
  const int ty = threadIdx.x / W, ix = blockIdx.x * W + (threadIdx.x - ty * W), iy = blockIdx.y * H + ty;
  if (ty >= H || ix >= h.n[0] || iy >= h.n[1]) return;
  const int planes = h.n[2] * h.n[3];
  const double x = add(h.minp[0], mul((double)ix, h.dx[0]));
  const double y = add(h.minp[1], mul((double)iy, h.dx[1]));
  bool bad = false;
  for (int p = blockIdx.z; p < planes; p += gridDim.z) {
    const int ivy = p / h.n[2], ivx = p - ivy * h.n[2];
    const double vx = add(h.minp[2], mul((double)ivx, h.dx[2]));
    const double vy = add(h.minp[3], mul((double)ivy, h.dx[3]));
    const double fx = mul(sub(sub(x, mul(dt, vx)), h.minp[0]), h.inv_dx[0]);
    const double fy = mul(sub(sub(y, mul(dt, vy)), h.minp[1]), h.inv_dx[1]);
    const int i0 = (int)floor(fx), i1 = (int)floor(fy);
    double v = 0.;
    if (i0 < -1 || i0 > h.n[0] - 1 || i1 < -1 || i1 > h.n[1] - 1) {
      bad = true;
    } else {
      double ex[4], ey[4], t[4][4];
      const double *row = tmp + h.at(i0 - 1, i1 - 1, ivx, ivy);
#pragma unroll
      for (int ky = 0; ky < 4; ++ky)
#pragma unroll
        for (int kx = 0; kx < 4; ++kx) t[ky][kx] = __ldg(row + ky * h.s[1] + kx);
      bspline_w<true>(sub(fx, (double)i0), ex);
      bspline_w<true>(sub(fy, (double)i1), ey);
#pragma unroll
      for (int ky = 0; ky < 4; ++ky) {
        double s = 0.;
#pragma unroll
        for (int kx = 0; kx < 4; ++kx) s = add(s, mul(ex[kx], t[ky][kx]));
        v = add(v, mul(ey[ky], s));
      }
    }
    fn[h.at(ix, iy, ivx, ivy)] = v;
  }
  if (bad) atomicOr(err, 2);
}

// 3-point Lagrange weights (Advection.hpp thrust :29-34).
template <bool EXACT>
__device__ __forceinline__ void lag3w(double p, double c[3]) {
  if (EXACT) {
    c[0] = mul(mul(.5, sub(p, 1.)), sub(p, 2.));
    c[1] = mul(mul(-1., p), sub(p, 2.));
    c[2] = mul(mul(.5, p), sub(p, 1.));
  } else {
    c[0] = .5 * (p - 1.) * (p - 2.);
    c[1] = -p * (p - 2.);
    c[2] = .5 * p * (p - 1.);
  }
}

// Whether coordinate x of a foot lies in dimension j's admissible range.  A NaN
// (of dt, the field, or f through it) does not: a test for lying outside would
// let it pass, and its cell index is INT_MIN.
__device__ __forceinline__ bool in_range(const HGrid &h, double x, int j) { return x >= h.lo[j] && x <= h.hi[j]; }

// computeFeet (thrust Advection.hpp:260-309): half-step predictor with the
// cell's own field, the field interpolated (periodic 3x3 Lagrange) at the
// predicted (x, y), then the full-step foot; vx, vy clamped to the domain.
// Returns the foot in grid units (xs - min) / h per dimension and whether
// it lies in the admissible range.
template <bool EXACT>
__device__ __forceinline__ bool foot4d(const HGrid &h, const double *__restrict__ ex, const double *__restrict__ ey,
                                       int ix, int iy, int ivx, int ivy, double dt, double g[4]) {
  const int nx = h.n[0], ny = h.n[1];
  double x, y, vx, vy, hdt = mul(0.5, dt);
  if (EXACT) {
    x = add(h.minp[0], mul((double)ix, h.dx[0]));
    y = add(h.minp[1], mul((double)iy, h.dx[1]));
    vx = add(h.minp[2], mul((double)ivx, h.dx[2]));
    vy = add(h.minp[3], mul((double)ivy, h.dx[3]));
  } else {
    x = h.minp[0] + ix * h.dx[0];
    y = h.minp[1] + iy * h.dx[1];
    vx = h.minp[2] + ivx * h.dx[2];
    vy = h.minp[3] + ivy * h.dx[3];
  }
  double t[2];
  if (EXACT) {
    t[0] = mul(h.inv_dx[0], sub(sub(x, mul(hdt, vx)), h.minp[0]));
    t[1] = mul(h.inv_dx[1], sub(sub(y, mul(hdt, vy)), h.minp[1]));
  } else {
    t[0] = h.inv_dx[0] * (x - hdt * vx - h.minp[0]);
    t[1] = h.inv_dx[1] * (y - hdt * vy - h.minp[1]);
  }
  int ip[2];
  double c[2][3];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    // The reference's (n + ipos + k) % n; a far-off predictor (a time step
    // the range check will reject) is kept inside the field by the clamp
    // and the non-negative modulo.
    ip[j] = (int)fmax(fmin(round(t[j]) - 1., 1e9), -1e9);
    lag3w<EXACT>(EXACT ? sub(t[j], (double)ip[j]) : t[j] - ip[j], c[j]);
  }
  double e1 = 0., e2 = 0.;
  const int r0 = wrapi(ip[0], nx), r1 = wrapi(ip[1], ny);
#pragma unroll
  for (int k1 = 0; k1 < 3; ++k1) {
    const int jy = r1 + k1 >= ny ? r1 + k1 - ny : r1 + k1;
#pragma unroll
    for (int k0 = 0; k0 < 3; ++k0) {
      const int jx = r0 + k0 >= nx ? r0 + k0 - nx : r0 + k0;
      const int q = jx + nx * jy;
      if (EXACT) {
        const double w = mul(c[0][k0], c[1][k1]);
        e1 = add(e1, mul(w, __ldg(ex + q)));
        e2 = add(e2, mul(w, __ldg(ey + q)));
      } else {
        const double w = c[0][k0] * c[1][k1];
        e1 = fma(w, __ldg(ex + q), e1);
        e2 = fma(w, __ldg(ey + q), e2);
      }
    }
  }
  double xs[4];
  if (EXACT) {
    const double vxh = sub(vx, mul(hdt, e1)), vyh = sub(vy, mul(hdt, e2));
    xs[0] = sub(x, mul(dt, vxh));
    xs[1] = sub(y, mul(dt, vyh));
    xs[2] = fmax(fmin(sub(vx, mul(dt, e1)), h.vtop[2]), h.minp[2]);
    xs[3] = fmax(fmin(sub(vy, mul(dt, e2)), h.vtop[3]), h.minp[3]);
  } else {
    xs[0] = x - dt * (vx - hdt * e1);
    xs[1] = y - dt * (vy - hdt * e2);
    xs[2] = fmax(fmin(vx - dt * e1, h.vtop[2]), h.minp[2]);
    xs[3] = fmax(fmin(vy - dt * e2, h.vtop[3]), h.minp[3]);
  }
  bool ok = true;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    ok &= in_range(h, xs[j], j);
    g[j] = EXACT ? mul(h.inv_dx[j], sub(xs[j], h.minp[j])) : h.inv_dx[j] * (xs[j] - h.minp[j]);
  }
  return ok;
}

// interp_4d (thrust Advection.hpp:311-385, spline branch): 4^4 tensor
// B-spline interpolation of the coefficients c at the foot g (grid units).
template <bool EXACT>
__device__ __forceinline__ double interp4d(const HGrid &h, const double *__restrict__ c, const double g[4]) {
  int ip[4];
  double eta[4][4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    ip[j] = (int)floor(g[j]);
    bspline_w<EXACT>(EXACT ? sub(g[j], (double)ip[j]) : g[j] - ip[j], eta[j]);
  }
  const double *b = c + h.at(ip[0] - 1, ip[1] - 1, ip[2] - 1, ip[3] - 1);
  double f1 = 0.;
#pragma unroll
  for (int k3 = 0; k3 < 4; ++k3) {
#pragma unroll
    for (int k2 = 0; k2 < 4; ++k2) {
      double f2 = 0.;
#pragma unroll
      for (int k1 = 0; k1 < 4; ++k1) {
        const double *row = b + k1 * h.s[1] + k2 * h.s[2] + k3 * h.s[3];
        if (EXACT) {
          double f3 = 0.;
#pragma unroll
          for (int k0 = 0; k0 < 4; ++k0) f3 = add(f3, mul(eta[0][k0], __ldg(row + k0)));
          f2 = add(f2, mul(f3, eta[1][k1]));
        } else {
          const double f3 = eta[0][0] * __ldg(row) + eta[0][1] * __ldg(row + 1) + eta[0][2] * __ldg(row + 2) +
                            eta[0][3] * __ldg(row + 3);
          f2 = fma(f3, eta[1][k1], f2);
        }
      }
      f1 = EXACT ? add(f1, mul(mul(f2, eta[2][k2]), eta[3][k3])) : fma(f2 * eta[2][k2], eta[3][k3], f1);
    }
  }
  return f1;
}

// Advection::advect_4D at the grid points: a block is a tile of W x and H y
// (PlaneTiles), blockIdx.z = plane group; a thread takes the planes p = z, z + G, ...
// (p = ivx + nvx*ivy).  MOMENT also accumulates the velocity moment
// (part[z][ix + nx*iy]) and, per block, the sum of squares of the new
// values (l2[block] as a (sum, 0) pair) for the field and the L2 norm.
template <bool EXACT, bool MOMENT>
__global__ void __launch_bounds__(256) k_mpi_advect_4d(const double *__restrict__ c, double *__restrict__ fn,
                                                       const double *__restrict__ ex, const double *__restrict__ ey,
                                                       HGrid h, int W, int H, double dt,
                                                       double *__restrict__ part, double *__restrict__ l2,
                                                       int *__restrict__ err) {
  const int ty = threadIdx.x / W, ix = blockIdx.x * W + (threadIdx.x - ty * W), iy = blockIdx.y * H + ty;
  const int G = gridDim.z;
  const bool live = ty < H && ix < h.n[0] && iy < h.n[1];
  const long long planes = (long long)h.n[2] * h.n[3];
  double acc = 0., sq = 0.;
  bool bad = false;
  if (live) {
    for (long long p = blockIdx.z; p < planes; p += G) {
      const int ivx = (int)(p % h.n[2]), ivy = (int)(p / h.n[2]);
      double g[4];
      double v = 0.;
      if (foot4d<EXACT>(h, ex, ey, ix, iy, ivx, ivy, dt, g)) {
        v = interp4d<EXACT>(h, c, g);
      } else {
        bad = true;
      }
      fn[h.at(ix, iy, ivx, ivy)] = v;
      if (MOMENT) {
        acc += v;
        sq = fma(v, v, sq);
      }
    }
  }
  if (bad) atomicOr(err, 2);
  if (MOMENT) {
    if (live) part[(long long)blockIdx.z * h.n[0] * h.n[1] + ix + (long long)h.n[0] * iy] = acc;
    // Block sum of sq in a fixed order.
    __shared__ double ws[8];
    const int tid = threadIdx.x;
    double v = sq;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((tid & 31) == 0) ws[tid >> 5] = v;
    __syncthreads();
    if (tid == 0) {
      double s = 0.;
      for (int w = 0; w < (int)blockDim.x / 32; ++w) s += ws[w];
      const long long b = blockIdx.x + (long long)gridDim.x * (blockIdx.y + (long long)gridDim.y * blockIdx.z);
      l2[2 * b] = s;
      l2[2 * b + 1] = 0.;
    }
  }
}

// ---------------------------------------------------------------------------
// The tiled 4D advection.  A CTA owns a tile of W x (4 YG) y x V vx grid
// points and marches along vy: the coefficients its feet can reach (two more
// points on each side of x, y and vx, five vy slabs) stay in a ring of six
// shared-memory slabs, the sixth arriving by cp.async while a step computes.
// A thread owns four (EXACT: two) cells at consecutive y: a coefficient row is
// read from shared memory once for all of them, 112 (160) loads per cell
// instead of 256.
//
// Tile4 (internal.cuh) is the geometry of the tiles.
// Cells of a thread (consecutive in y) and threads of a block.  Measured, us,
// four cells and 256 threads (255 registers) against two and 512 (128): fused
// 128 x 128 x 64 x 64 4343 / 5052, 64^4 1271 / 1349, 48 x 44 x 40 x 36 331 / 338;
// EXACT, with twice the FP64 instructions per load, 6530 / 5474, 1891 / 1471 and
// 443 / 366.  (Three and 384 threads: 19.9 ms at 128^4 against 16.6 for four.)
template <bool EXACT>
struct TileShape {
  static constexpr int cells = EXACT ? 2 : 4, threads = EXACT ? 512 : 256;
};
constexpr int kRing = 6;

// Weight j of the cubic B-spline at fractional offset p, for a j known at
// run time only: z^3/6 (outer) or 2/3 - z^2 + z^3/2 (inner) with z = p or
// 1 - p.  EXACT evaluates the reference's sequence and selects.
template <bool EXACT>
__device__ __forceinline__ double bspline_j(double p, int j) {
  if (EXACT) {
    double e[4];
    bspline_w<true>(p, e);
    return j <= 0 ? e[0] : (j == 1 ? e[1] : (j == 2 ? e[2] : e[3]));
  }
  const double z = (j == 0 || j == 2) ? 1. - p : p;
  const double z2 = z * z;
  return (j == 0 || j == 3) ? z2 * z * (1. / 6.) : fma(z2, fma(.5, z, -1.), 2. / 3.);
}

// The predictor's x part of a thread (it depends on x and vx only) and y part
// of a row (y and vy): the 3-point weights of the field there and the first
// of the three points, relative to the tile's field rows and columns.
constexpr int kTileX = 6;  // c0[3], x, vx, first column
constexpr int kTileY = 5;  // c1[3], y, first row

// What bounds it: FP64 (about 350 multiply-adds per cell in the sums and 100
// in the foot, at 64 per clock and SM) and the shared-memory pipe (112 loads
// of 8 bytes per cell at 128 bytes per clock and SM) take about the same
// time.  The sign of the field decides whether a cell's vx (vy) taps start
// at -2 or -1; where the cells of a thread disagree, the warp reads one
// slab more in that dimension and each cell's weight is 0 on the slab that
// is not its own (EXACT skips it), so the lines where a field component changes sign cost a quarter more
// there and not a second pass.  Cells whose x or y taps start at different
// points (only beside the planes vx = 0 and vy = 0) take one sweep each;
// feet further than one cell away interpolate one by one from global memory.
// Measured (128^4, a field whose zero lines cross the plane): 16.5 ms against
// 55 to 58 ms for two cells per thread from L1, whose warps ran both branches
// wherever the two cells' first taps differed (26 ms where they hardly ever
// did); FP64 pipe 48%, shared-memory pipe 51%, fixed-latency waits first (two
// warps per scheduler); sums along x first: 17.4 ms.
template <bool EXACT, bool MOMENT, int PXC>
__global__ void __launch_bounds__(TileShape<EXACT>::threads, 1)
    k_mpi_advect_4d_tile(const double *__restrict__ c, double *__restrict__ fn, const double *__restrict__ ex,
                         const double *__restrict__ ey, HGrid h, Tile4 T, double dt, double *__restrict__ part,
                         double *__restrict__ l2, int *__restrict__ err) {
  constexpr int kCells = TileShape<EXACT>::cells, kTileThreads = TileShape<EXACT>::threads;
  extern __shared__ __align__(16) double sm[];
  const int PX = PXC ? PXC : T.PX;
  const int RY = T.RY, slab = T.slab;
  const int rows = kCells * T.YG, lines = T.W * T.V;
  double *fex = sm + kRing * slab, *fey = fex + PX * RY;
  double *xt = fey + PX * RY;         // [kTileX][lines]
  double *yt = xt + kTileX * lines;   // [2][kTileY][rows], by the parity of vy
  int *rowoff = reinterpret_cast<int *>(yt + 2 * kTileY * rows);  // [RV][RY]: a slab's rows in c, -1 past the halo
  const int tid = threadIdx.x;
  const int tx = tid % T.W, tr = tid / T.W;
  const int yg = tr % T.YG, vl = tr / T.YG;
  const int nx = h.n[0], ny = h.n[1], nvx = h.n[2], nvy = h.n[3];
  const double hdt = mul(0.5, dt);
  double sq = 0.;
  bool bad = false;
  for (int item = blockIdx.x; item < T.nitems; item += gridDim.x) {
    int r = item;
    const int x0 = (r % T.nxt) * T.W;
    r /= T.nxt;
    const int yt0 = (r % T.nyt) * rows;
    r /= T.nyt;
    const int vx0 = (r % T.nvt) * T.V, seg = r / T.nvt, vt = r % T.nvt;
    const int vy0 = seg * T.Q, vy1 = vy0 + T.Q < nvy ? vy0 + T.Q : nvy;
    const int x = x0 + tx, y0 = yt0 + kCells * yg, ivx = vx0 + vl;
    const bool live = vl < T.V && x < nx && y0 < ny && ivx < nvx;
    __syncthreads();  // the item before has been read
    // Slab vy of the tile into ring slot `slot`; points past the halo (next
    // to cells past the grid) are left as they are.
    for (int i = tid; i < RY * T.RV; i += kTileThreads) {
      const int v = i / RY, yy = i - v * RY;
      rowoff[i] = yt0 + yy < ny + 5 && vx0 + v < nvx + 5 ? h.is[1] * yy + h.is[2] * v : -1;
    }
    __syncthreads();
    const int xlim = nx + 5 - x0;
    auto load_slab = [&](int vy, int slot) {
      const double *g = c + h.at(x0 - 2, yt0 - 2, vx0 - 2, vy);
      double *d = sm + slot * slab;
      for (int i = tid; i < slab; i += kTileThreads) {
        const int row = PXC ? i / PX : (int)__umulhi((unsigned)i, T.magic);  // i / PX
        const int xx = i - row * PX, off = rowoff[row];
        if (off >= 0 && xx < xlim) cp_async8(d + i, g + (off + xx));
      }
    };
    for (int k = 0; k < 5; ++k) load_slab(vy0 - 2 + k, k);
    // The field around the tile, periodic.
    for (int i = tid; i < PX * RY; i += kTileThreads) {
      const int q = wrapi(x0 - 2 + i % PX, nx) + nx * wrapi(yt0 - 2 + i / PX, ny);
      fex[i] = __ldg(ex + q);
      fey[i] = __ldg(ey + q);
    }
    // The predictor (foot4d) at (position i of dimension d, velocity v of it).
    auto predictor = [&](int d, int i, int v, double w[3], double &pos, double &vel) {
      pos = EXACT ? add(h.minp[d], mul((double)i, h.dx[d])) : h.minp[d] + i * h.dx[d];
      vel = EXACT ? add(h.minp[d + 2], mul((double)v, h.dx[d + 2])) : h.minp[d + 2] + v * h.dx[d + 2];
      const double t = EXACT ? mul(h.inv_dx[d], sub(sub(pos, mul(hdt, vel)), h.minp[d]))
                             : h.inv_dx[d] * (pos - hdt * vel - h.minp[d]);
      const int ip = (int)fmax(fmin(round(t) - 1., 1e9), -1e9);
      lag3w<EXACT>(EXACT ? sub(t, (double)ip) : t - ip, w);
      return ip;
    };
    for (int i = tid; i < lines; i += kTileThreads) {
      double w[3], pos, vel;
      const int ip = predictor(0, x0 + i % T.W, vx0 + i / T.W, w, pos, vel);
      xt[i] = w[0];
      xt[lines + i] = w[1];
      xt[2 * lines + i] = w[2];
      xt[3 * lines + i] = pos;
      xt[4 * lines + i] = vel;
      xt[5 * lines + i] = (double)(ip - (x0 - 2));
    }
    auto y_table = [&](int vy) {
      if (tid < rows) {
        double w[3], pos, vel, *t = yt + (vy & 1) * kTileY * rows + tid;
        const int ip = predictor(1, yt0 + tid, vy, w, pos, vel);
        t[0] = w[0];
        t[rows] = w[1];
        t[2 * rows] = w[2];
        t[3 * rows] = pos;
        t[4 * rows] = (double)(ip - (yt0 - 2));
      }
    };
    y_table(vy0);
    double racc[kCells] = {};
    int s0 = 0;  // ring slot of slab vy - 2
    for (int vy = vy0; vy < vy1; ++vy) {
      cp_async_wait_all();
      __syncthreads();
      if (vy + 1 < vy1) {
        load_slab(vy + 3, s0 == 0 ? kRing - 1 : s0 - 1);
        y_table(vy + 1);
      }
      if (live) {
        double g[kCells][4];
        bool ok[kCells];
        // The feet (foot4d, with the field from shared memory: its 3 x 3
        // points share their rows among the four cells).
        {
          const double *xl = xt + vl * T.W + tx;
          const double *yl = yt + (vy & 1) * kTileY * rows + kCells * yg;
          const int lx = (int)xl[5 * lines], ly = (int)yl[4 * rows];
          bool infield = lx >= 0 && lx + 2 < PX && ly >= 0 && ly + kCells + 2 <= RY;
#pragma unroll
          for (int q = 1; q < kCells; ++q) infield &= yl[4 * rows + q] == yl[4 * rows] + q;
          if (infield) {
            const double c0 = xl[0], c1 = xl[lines], c2 = xl[2 * lines];
            double e1[kCells] = {}, e2[kCells] = {};
            const double *p1 = fex + ly * PX + lx, *p2 = fey + ly * PX + lx;
#pragma unroll
            for (int k = 0; k < kCells + 2; ++k) {
              const double a0 = p1[k * PX], a1 = p1[k * PX + 1], a2 = p1[k * PX + 2];
              const double b0 = p2[k * PX], b1 = p2[k * PX + 1], b2 = p2[k * PX + 2];
              const double ra = EXACT ? 0. : c0 * a0 + c1 * a1 + c2 * a2;
              const double rb = EXACT ? 0. : c0 * b0 + c1 * b1 + c2 * b2;
#pragma unroll
              for (int q = 0; q < kCells; ++q) {
                const int k1 = k - q;
                if (k1 < 0 || k1 > 2) continue;
                const double w = yl[k1 * rows + q];
                if (EXACT) {
                  const double w0 = mul(c0, w), w1 = mul(c1, w), w2 = mul(c2, w);
                  e1[q] = add(add(add(e1[q], mul(w0, a0)), mul(w1, a1)), mul(w2, a2));
                  e2[q] = add(add(add(e2[q], mul(w0, b0)), mul(w1, b1)), mul(w2, b2));
                } else {
                  e1[q] = fma(w, ra, e1[q]);
                  e2[q] = fma(w, rb, e2[q]);
                }
              }
            }
            const double xc = xl[3 * lines], vxc = xl[4 * lines];
            const double vyc = EXACT ? add(h.minp[3], mul((double)vy, h.dx[3])) : h.minp[3] + vy * h.dx[3];
#pragma unroll
            for (int q = 0; q < kCells; ++q) {
              const double yc = yl[3 * rows + q];
              double xs[4];
              if (EXACT) {
                xs[0] = sub(xc, mul(dt, sub(vxc, mul(hdt, e1[q]))));
                xs[1] = sub(yc, mul(dt, sub(vyc, mul(hdt, e2[q]))));
                xs[2] = fmax(fmin(sub(vxc, mul(dt, e1[q])), h.vtop[2]), h.minp[2]);
                xs[3] = fmax(fmin(sub(vyc, mul(dt, e2[q])), h.vtop[3]), h.minp[3]);
              } else {
                xs[0] = xc - dt * (vxc - hdt * e1[q]);
                xs[1] = yc - dt * (vyc - hdt * e2[q]);
                xs[2] = fmax(fmin(vxc - dt * e1[q], h.vtop[2]), h.minp[2]);
                xs[3] = fmax(fmin(vyc - dt * e2[q], h.vtop[3]), h.minp[3]);
              }
              ok[q] = true;
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                ok[q] &= in_range(h, xs[j], j);
                g[q][j] = EXACT ? mul(h.inv_dx[j], sub(xs[j], h.minp[j])) : h.inv_dx[j] * (xs[j] - h.minp[j]);
              }
            }
          } else {
#pragma unroll
            for (int q = 0; q < kCells; ++q) {
              const int iy = y0 + q < ny ? y0 + q : ny - 1;
              ok[q] = foot4d<EXACT>(h, ex, ey, x, iy, ivx, vy, dt, g[q]);
            }
          }
        }
        // First cells of the taps relative to the grid point: -1 or 0 in every
        // dimension.  Bit q of mx, my, m2, m3: 0 for cell q.  b2, b3 = 1 (and
        // the mask 0) where all cells of the thread say 0.
        bool fast = true;
        int b2 = 0, b3 = 0;
        unsigned mx = 0, my = 0, m2 = 0, m3 = 0;
        const unsigned all = y0 + kCells <= ny ? (1u << kCells) - 1u : (1u << (ny - y0)) - 1u;
        double out[kCells] = {};
        double e0[kCells][4], e1[kCells][4], e2[kCells][4], p3[kCells];
#pragma unroll
        for (int q = 0; q < kCells; ++q) {
          const double f0 = floor(g[q][0]), f1 = floor(g[q][1]), f2 = floor(g[q][2]), f3 = floor(g[q][3]);
          const int a0 = (int)f0 - x + 1, a1 = (int)f1 - (y0 + q) + 1, a2 = (int)f2 - ivx + 1, a3 = (int)f3 - vy + 1;
          fast &= (ok[q] && (unsigned)(a0 | a1 | a2 | a3) < 2u) || y0 + q >= ny;
          mx |= (unsigned)(a0 & 1) << q;
          my |= (unsigned)(a1 & 1) << q;
          m2 |= (unsigned)(a2 & 1) << q;
          m3 |= (unsigned)(a3 & 1) << q;
          bspline_w<EXACT>(EXACT ? sub(g[q][0], f0) : g[q][0] - f0, e0[q]);
          bspline_w<EXACT>(EXACT ? sub(g[q][1], f1) : g[q][1] - f1, e1[q]);
          bspline_w<EXACT>(EXACT ? sub(g[q][2], f2) : g[q][2] - f2, e2[q]);
          p3[q] = EXACT ? sub(g[q][3], f3) : g[q][3] - f3;
        }
        m2 &= all;
        m3 &= all;
        if (m2 == all) { b2 = 1; m2 = 0; }
        if (m3 == all) { b3 = 1; m3 = 0; }
        if (fast) {
          const unsigned act = __activemask();
          const bool five2 = __any_sync(act, m2 != 0), five3 = __any_sync(act, m3 != 0);
          // Five slabs: every lane reads the same five, all of them loaded.
          if (five2 && b2) { b2 = 0; m2 = all; }
          if (five3 && b3) { b3 = 0; m3 = all; }
          // The sum over the slabs for the cells whose x and y taps start at
          // (bx, by); MIX: some lane's cells differ in their first slab.
          auto sweep = [&](auto mixed, unsigned bx, unsigned by, int n3, bool five2, double val[kCells]) {
            constexpr bool MIX = decltype(mixed)::value;
            // First tap: local x = tx + 2 - 1 + (0 or -1) and so on.
            const double *base = sm + ((vl + b2) * RY + kCells * yg + (int)by) * PX + tx + (int)bx;
            int slot = s0 + b3;
            if (slot >= kRing) slot -= kRing;
#pragma unroll
            for (int q = 0; q < kCells; ++q) val[q] = 0.;
            // The cells' vx weights on the five slabs (MIX) or the four.
            double w2[kCells][MIX ? 5 : 4];
#pragma unroll
            for (int q = 0; q < kCells; ++q) {
              const bool later = MIX && ((m2 >> q) & 1);
#pragma unroll
              for (int k = 0; k < (MIX ? 5 : 4); ++k)
                w2[q][k] = later ? (k > 0 ? e2[q][k - 1] : 0.) : (k < 4 ? e2[q][k] : 0.);
            }
#pragma unroll 1
            for (int k3 = 0; k3 < n3; ++k3) {
              const double *sl = base + slot * slab;
              if (++slot == kRing) slot = 0;
              double u[kCells] = {}, w3[kCells];
              bool in3[kCells];
#pragma unroll
              for (int q = 0; q < kCells; ++q) {
                const int j = MIX ? k3 - (int)((m3 >> q) & 1) : k3;
                in3[q] = !MIX || (j >= 0 && j < 4);
                w3[q] = bspline_j<EXACT>(p3[q], j);
                if (!EXACT && !in3[q]) w3[q] = 0.;
              }
#pragma unroll
              for (int k2 = 0; k2 < (MIX ? 5 : 4); ++k2) {
                if (MIX && k2 == 4 && !five2) break;
                const double *row = sl + k2 * RY * PX;
                // EXACT sums along x first, as the reference does; otherwise y
                // first: sixteen independent chains of four.
                double s2[kCells], t[kCells][4];
#pragma unroll
                for (int k = 0; k < kCells + 3; ++k) {
                  const double v0 = row[k * PX], v1 = row[k * PX + 1], v2 = row[k * PX + 2], v3 = row[k * PX + 3];
#pragma unroll
                  for (int q = 0; q < kCells; ++q) {
                    const int k1 = k - q;
                    if (k1 < 0 || k1 > 3) continue;
                    if (EXACT) {
                      const double f3 = add(add(add(mul(e0[q][0], v0), mul(e0[q][1], v1)), mul(e0[q][2], v2)),
                                            mul(e0[q][3], v3));
                      s2[q] = k1 == 0 ? mul(f3, e1[q][0]) : add(s2[q], mul(f3, e1[q][k1]));
                    } else {
                      const double w = e1[q][k1];
                      t[q][0] = k1 == 0 ? w * v0 : fma(w, v0, t[q][0]);
                      t[q][1] = k1 == 0 ? w * v1 : fma(w, v1, t[q][1]);
                      t[q][2] = k1 == 0 ? w * v2 : fma(w, v2, t[q][2]);
                      t[q][3] = k1 == 0 ? w * v3 : fma(w, v3, t[q][3]);
                      if (k1 == 3)
                        s2[q] = fma(e0[q][1], t[q][1], e0[q][0] * t[q][0]) + fma(e0[q][3], t[q][3], e0[q][2] * t[q][2]);
                    }
                  }
                }
#pragma unroll
                for (int q = 0; q < kCells; ++q) {
                  const bool later = MIX && ((m2 >> q) & 1);
                  const bool in2 = k2 == 0 ? !later : (k2 == 4 ? later : true);
                  if (EXACT) {
                    const double v = add(val[q], mul(mul(s2[q], w2[q][k2]), w3[q]));
                    if (in2 && in3[q]) val[q] = v;
                  } else {
                    u[q] = fma(s2[q], w2[q][k2], u[q]);
                  }
                }
              }
              if (!EXACT) {
#pragma unroll
                for (int q = 0; q < kCells; ++q) val[q] = fma(u[q], w3[q], val[q]);
              }
            }
          };
          // One sweep per pair of first x and y taps among the thread's
          // cells: one, except beside the planes vx = 0 and vy = 0.
          unsigned rem = all;
          do {
            const int q0 = rem ? __ffs(rem) - 1 : 0;
            const unsigned bx = (mx >> q0) & 1, by = (my >> q0) & 1;
            const unsigned take = rem & (bx ? mx : ~mx) & (by ? my : ~my);
            rem &= ~take;
            double val[kCells];
            if (five2 || five3) sweep(std::true_type{}, bx, by, five3 ? 5 : 4, five2, val);
            else sweep(std::false_type{}, bx, by, 4, false, val);
#pragma unroll
            for (int q = 0; q < kCells; ++q) out[q] = (take >> q) & 1 ? val[q] : out[q];
          } while (__any_sync(act, rem != 0));
        } else {
#pragma unroll
          for (int q = 0; q < kCells; ++q) {
            if (y0 + q < ny) {
              // The foot again: it is rarely needed and not kept.
              double gq[4];
              if (foot4d<EXACT>(h, ex, ey, x, y0 + q, ivx, vy, dt, gq)) out[q] = interp4d<EXACT>(h, c, gq);
              else bad = true;
            }
          }
        }
        double *o = fn + h.at(x, y0, ivx, vy);
#pragma unroll
        for (int q = 0; q < kCells; ++q) {
          if (y0 + q < ny) {
            o[q * h.s[1]] = out[q];
            if (MOMENT) {
              racc[q] += out[q];
              sq = fma(out[q], out[q], sq);
            }
          }
        }
      }
      if (++s0 == kRing) s0 = 0;
    }
    if (MOMENT) {
      // Sum over the tile's vx in order; one partial per (vx tile, segment).
      __syncthreads();
      const int cells = T.W * rows;
      if (vl < T.V) {
#pragma unroll
        for (int q = 0; q < kCells; ++q) sm[vl * cells + (kCells * yg + q) * T.W + tx] = live ? racc[q] : 0.;
      }
      __syncthreads();
      double *dst = part + (long long)(vt * T.nseg + seg) * nx * ny;
      for (int i = tid; i < cells; i += kTileThreads) {
        const int xx = x0 + i % T.W, yy = yt0 + i / T.W;
        if (xx < nx && yy < ny) {
          double s = 0.;
          for (int v = 0; v < T.V; ++v) s += sm[v * cells + i];
          dst[xx + (long long)nx * yy] = s;
        }
      }
    }
  }
  if (bad) atomicOr(err, 2);
  if (MOMENT) {
    // Block sum of sq in a fixed order.
    __shared__ double ws[kTileThreads / 32];
    double v = sq;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((tid & 31) == 0) ws[tid >> 5] = v;
    __syncthreads();
    if (tid == 0) {
      double t = 0.;
      for (int w = 0; w < kTileThreads / 32; ++w) t += ws[w];
      l2[2 * blockIdx.x] = t;
      l2[2 * blockIdx.x + 1] = 0.;
    }
  }
}

// ---------------------------------------------------------------------------
// initcase of vlp4d_mpi (Init.cpp:126-277) on a halo array: the halo is
// zero, as after init() (Init.cpp:370-372); grid points get
//   10 SLD10: (1/2pi) exp(-(vx^2+vy^2)/2) (1 + 0.05 cos(x/2) cos(y/2))
//   20 TSI20: 1/(4 pi vthx vthy) (1 - ax sin(kx x) - ay sin(ky y))
//             [exp(-((vx-vd)/vthx)^2/2 - (vy/vthy)^2/2) + (vx+vd) term],
//             vd 2.4, vthx 1, vthy 0.5, ax 0.05, ay 0.25, kx = ky = 0.2
//   2, 5 CYL02 / CYL05: AMPLI hx hv with the cosine bumps of x, vx (2) or
//             y, vy (5); case 5 leaves the last vx, y and x index at 0, as
//             the reference's loops do (Init.cpp:198-202 stop before
//             local_nxmax).
__global__ void k_mpi_init_case(double *__restrict__ f, HGrid h, int idcase) {
  const long long total = h.total();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    long long r0 = i;
    int c[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      c[k] = (int)(r0 % h.e[k]) - kH;
      r0 /= h.e[k];
    }
    bool inside = true;
#pragma unroll
    for (int k = 0; k < 4; ++k) inside &= (c[k] >= 0 && c[k] < h.n[k]);
    double v = 0.;
    if (inside) {
      const double x = h.minp[0] + c[0] * h.dx[0], y = h.minp[1] + c[1] * h.dx[1];
      const double vx = h.minp[2] + c[2] * h.dx[2], vy = h.minp[3] + c[3] * h.dx[3];
      if (idcase == 10) {
        const double sum = vx * vx + vy * vy;
        v = (1. / (2 * M_PI)) * exp(-0.5 * sum) * (1 + 0.05 * (cos(0.5 * x) * cos(0.5 * y)));
      } else if (idcase == 20) {
        const double vd = 2.4, vthx = 1.0, vthy = 0.5, ax = 0.05, ay = 0.25, kx = 0.2, ky = 0.2;
        const double a = (vx - vd) / vthx, b = (vx + vd) / vthx, q = vy / vthy;
        v = 1. / (4 * M_PI * vthx * vthy) * (1 - ax * sin(kx * x) - ay * sin(ky * y)) *
            (exp(-.5 * (a * a + q * q)) + exp(-.5 * (b * b + q * q)));
      } else if (idcase == 2 || idcase == 5) {
        const bool skip = idcase == 5 && (c[2] == h.n[2] - 1 || c[1] == h.n[1] - 1 || c[0] == h.n[0] - 1);
        if (!skip) {
          const double PERIOD = 0.5 * M_PI, AMPLI = 4, cc = 0.50 * (6. / 16.), rc = 0.50 * (4. / 16.);
          const double xx = idcase == 2 ? x : y, vv = idcase == 2 ? vx : vy;
          double hv = 0.0, hx = 0.0;
          if ((vv <= cc + rc) && (vv >= cc - rc)) hv = cos(PERIOD * ((vv - cc) / rc));
          else if ((vv <= -cc + rc) && (vv >= -cc - rc)) hv = -cos(PERIOD * ((vv + cc) / rc));
          if ((xx <= cc + rc) && (xx >= cc - rc)) hx = cos(PERIOD * ((xx - cc) / rc));
          else if ((xx <= -cc + rc) && (xx >= -cc - rc)) hx = -cos(PERIOD * ((xx + cc) / rc));
          v = AMPLI * hx * hv;
        }
      }
    }
    f[i] = v;
  }
}

// ---------------------------------------------------------------------------
// Velocity moment of the grid points of a halo array (Field.cpp:5-55):
// part[group][ixy] over the planes of the group.
__global__ void k_mpi_rho_partial(const double *__restrict__ f, double *__restrict__ part, HGrid h, int groups) {
  const long long nxy = (long long)h.n[0] * h.n[1];
  const long long ixy = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const int g = blockIdx.y;
  if (ixy >= nxy) return;
  const int ix = (int)(ixy % h.n[0]), iy = (int)(ixy / h.n[0]);
  const long long nv = (long long)h.n[2] * h.n[3];
  const long long v0 = nv * g / groups, v1 = nv * (g + 1) / groups;
  // Eight planes' loads ahead of their sums; the planes follow one another
  // without divisions.
  double s = 0.;
  int ivx = (int)(v0 % h.n[2]);
  const double *p = f + h.at(ix, iy, ivx, (int)(v0 / h.n[2]));
  const long long row = h.s[3] - (long long)(h.n[2] - 1) * h.s[2];  // from the last vx to the next vy
  auto next = [&] {
    if (++ivx == h.n[2]) {
      ivx = 0;
      p += row;
    } else {
      p += h.s[2];
    }
  };
  long long v = v0;
  for (; v + 8 <= v1; v += 8) {
    double t[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      t[k] = __ldg(p);
      next();
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) s += t[k];
  }
  for (; v < v1; ++v) {
    s += __ldg(p);
    next();
  }
  part[(long long)g * nxy + ixy] = s;
}

__device__ __forceinline__ void kahan(double &s, double &c, double x) {
  const double y = x - c;
  const double t = s + y;
  c = (t - s) - y;
  s = t;
}

// Sum of squares of the grid points of a halo array, per block as a Kahan
// (sum, compensation) pair, threads reduced in a fixed order.
__global__ void __launch_bounds__(256) k_mpi_l2_partial(const double *__restrict__ f, HGrid h,
                                                        double *__restrict__ l2) {
  // A warp walks rows (32 x positions at a time); the block's 8 warps take
  // rows r = 8 * blockIdx + warp, stepping by 8 * gridDim.
  const long long rows = (long long)h.n[1] * h.n[2] * h.n[3];  // below 2^32: such an array would be 550 GB
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  double s = 0., cp = 0.;
  // Four rows' loads at a time ahead of their sums.
  const long long step = (long long)gridDim.x * nw;
  for (long long r = (long long)blockIdx.x * nw + warp; r < rows; r += 4 * step) {
    const double *row[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const unsigned q = (unsigned)(r + k * step < rows ? r + k * step : r);
      const unsigned rv = q / (unsigned)h.n[1], ivy = rv / (unsigned)h.n[2];
      row[k] = f + h.at(0, (int)(q - rv * h.n[1]), (int)(rv - ivy * h.n[2]), (int)ivy);
    }
    const int live = rows - r > 3 * step ? 4 : (int)((rows - r + step - 1) / step);
    for (int ix = lane; ix < h.n[0]; ix += 32) {
      double v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] = __ldg(row[k] + ix);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (k < live) kahan(s, cp, v[k] * v[k]);
    }
  }
  __shared__ double ws[256];
  ws[threadIdx.x] = s - cp;
  __syncthreads();
  // The first warp: eight threads' sums per lane, then the lanes', in order.
  if (threadIdx.x < 32) {
    double a = 0., b = 0.;
#pragma unroll
    for (int t = 0; t < 8; ++t) kahan(a, b, ws[threadIdx.x * 8 + t]);
    double A = 0., B = 0.;
    for (int l = 0; l < 32; ++l) {
      kahan(A, B, __shfl_sync(0xffffffffu, a, l));
      kahan(A, B, -__shfl_sync(0xffffffffu, b, l));
    }
    if (threadIdx.x == 0) {
      l2[2 * blockIdx.x] = A;
      l2[2 * blockIdx.x + 1] = B;
    }
  }
}

// l2norm[iter] = sqrt(sum * dx dy dvx dvy) from `blocks` (sum, comp) pairs
// (Diags.cpp:50-76): lane l of the one warp adds the pairs l, l + 32, .. in
// order, lane 0 the lanes' sums in order, compensated throughout.  (One
// thread over 592 pairs: 38 us, a chain of loads and of 4 x 1184 additions.)
__global__ void k_mpi_l2_finish(const double *__restrict__ l2, long long blocks, double scale,
                                double *__restrict__ out) {
  double s = 0., c = 0.;
#pragma unroll 4
  for (long long b = threadIdx.x; b < blocks; b += 32) {
    kahan(s, c, l2[2 * b]);
    kahan(s, c, -l2[2 * b + 1]);
  }
  double a = 0., ac = 0.;
  for (int l = 0; l < 32; ++l) {
    kahan(a, ac, __shfl_sync(0xffffffffu, s, l));
    kahan(a, ac, -__shfl_sync(0xffffffffu, c, l));
  }
  if (threadIdx.x == 0) *out = sqrt(a * scale);
}

}  // namespace
}  // namespace vlp4d

// ---------------------------------------------------------------------------
// Host side.
namespace vlp4d {
namespace {

int mpi_check(const vlp4d_ctx *c, const char *what) {
  if (!c) return fail_msg(VLP4D_ERR_INVALID_ARG, std::string(what) + ": context is NULL");
  if (c->slab)
    return fail_msg(VLP4D_ERR_UNSUPPORTED, std::string(what) + ": the vlp4d_mpi arrays need an ordinary context");
  if (c->dtype != VLP4D_F64)
    return fail_msg(VLP4D_ERR_UNSUPPORTED, std::string(what) + ": the vlp4d_mpi path is FP64 (as the reference)");
  for (int k = 0; k < 4; ++k)
    if (c->g.n[k] < kMmax + 2)
      return fail_msg(VLP4D_ERR_INVALID_ARG,
                      std::string(what) + ": every grid dimension must be at least 10 (MMAX + 2, Init.cpp:85-89)");
  return VLP4D_OK;
}

int mpi_check_ptr(const void *p, const char *what) {
  if (!p) return fail_msg(VLP4D_ERR_INVALID_ARG, std::string(what) + ": array is NULL");
  if ((uintptr_t)p % 16) return fail_msg(VLP4D_ERR_INVALID_ARG, std::string(what) + ": array must be 16-byte aligned");
  return VLP4D_OK;
}

// Odd row stride of a shared-memory plane and its size in bytes.
int plane_stride(const HGrid &h) { return (int)(h.e[0] | 1); }
size_t plane_bytes(const HGrid &h) { return sizeof(double) * (size_t)h.e[1] * (size_t)plane_stride(h); }

int smem_limit(const vlp4d_ctx *c) {
  int v = 0;
  cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device);
  return v;
}

int launch_halo(vlp4d_ctx *c, const HGrid &h, double *f, cudaStream_t s) {
  (void)c;
  HaloParts P;
  P.parts = 0;
  long long blocks = 0;
  for (int m = 4; m >= 0; --m)
    for (int mask = 0; mask < 16; ++mask) {
      if (__builtin_popcount(mask) != m) continue;
      long long points = 1LL << m;
      for (int k = 0; k < 4; ++k)
        if (!((mask >> k) & 1) && (m > 0 || k >= 2)) points *= h.n[k] + 4;
      const long long per = m == 4 || m == 0 ? 1 : (m == 3 ? kHaloThreads / 32 : kHaloThreads);
      P.mask[P.parts] = (unsigned char)mask;
      P.first[P.parts++] = (int)blocks;
      blocks += (points + per - 1) / per;
      if (blocks > 0x7fffffffLL) return fail_msg(VLP4D_ERR_UNSUPPORTED, "mpi_halo_fill: too many halo points");
    }
  P.first[P.parts] = (int)blocks;
  k_mpi_halo<<<(unsigned)blocks, kHaloThreads, 0, s>>>(f, h, P);
  VLP4D_LAUNCH_CHECK();
  return VLP4D_OK;
}

int launch_spline_xy_exact(vlp4d_ctx *c, const HGrid &h, double *f, cudaStream_t s) {
  const size_t smem = plane_bytes(h);
  if (smem > (size_t)smem_limit(c))
    return fail_msg(VLP4D_ERR_UNSUPPORTED, "mpi_spline_xy: the (x, y) plane does not fit in shared memory");
  VLP4D_CUDA_TRY(cudaFuncSetAttribute(k_mpi_spline_xy, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 0;
  VLP4D_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_mpi_spline_xy, 256, smem));
  long long grid = (long long)c->num_sms * (per_sm > 0 ? per_sm : 1);
  const long long planes = h.e[2] * h.e[3];
  if (grid > planes) grid = planes;
  k_mpi_spline_xy<<<(unsigned)grid, dim3(32, 8), smem, s>>>(f, h, plane_stride(h));
  VLP4D_LAUNCH_CHECK();
  return VLP4D_OK;
}

// v lines along `dim` for o in [olo, olo + no), prefiltered for o in
// [flo, fhi].
template <bool EXTEND>
int launch_vlines(vlp4d_ctx *c, const HGrid &h, const double *in, double *out, int dim, int olo, int no, int flo,
                  int fhi, cudaStream_t s) {
  const size_t tile = sizeof(double) * 32 * (size_t)h.e[dim];
  const int lim = smem_limit(c);
  int warps = (int)(lim / tile);
  if (warps > 4) warps = 4;
  if (warps < 1) return fail_msg(VLP4D_ERR_UNSUPPORTED, "mpi v lines: a tile does not fit in shared memory");
  const size_t smem = tile * warps;
  auto k = k_mpi_vlines<EXTEND>;
  VLP4D_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 0;
  VLP4D_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, 32 * warps, smem));
  const long long tiles = (h.e[0] + 31) / 32 * h.e[1] * no;
  long long grid = (long long)c->num_sms * (per_sm > 0 ? per_sm : 1);
  const long long need = (tiles + warps - 1) / warps;
  if (grid > need) grid = need;
  k<<<(unsigned)grid, 32 * warps, smem, s>>>(in, out, h, dim, olo, no, flo, fhi);
  VLP4D_LAUNCH_CHECK();
  return VLP4D_OK;
}

// The fused step's v lines: extended and prefiltered, along dim.
int launch_vlines_fused(vlp4d_ctx *c, const HGrid &h, const double *in, double *out, int dim, int olo, int no, int flo,
                        int fhi, cudaStream_t s) {
  const int L = h.n[dim] + 4;
  const double aL = std::pow(h.alpha, L - 1);
  const dim3 grid((unsigned)((h.s[2] + 31) / 32), (unsigned)no);
#define VLP4D_SEG(S, NW) k_mpi_vlines_seg<S, NW><<<grid, NW * 32, 0, s>>>(in, out, h, dim, olo, flo, fhi, aL)
  // Longer lines than 32 segments of 17 hold: a lane per line.
  if (no > 65535 || L > 17 * 32) return launch_vlines<true>(c, h, in, out, dim, olo, no, flo, fhi, s);
  if (L <= 40) VLP4D_SEG(5, 8);
  else if (L <= 72) VLP4D_SEG(9, 8);
  else if (L <= 104) VLP4D_SEG(13, 8);
  else if (L <= 136) VLP4D_SEG(17, 8);
  else if (L <= 272) VLP4D_SEG(17, 16);
  else VLP4D_SEG(17, 32);
#undef VLP4D_SEG
  VLP4D_LAUNCH_CHECK();
  return VLP4D_OK;
}

int launch_spline_vxvy_exact(vlp4d_ctx *c, const HGrid &h, double *f, cudaStream_t s) {
  int rc = launch_vlines<false>(c, h, f, f, 2, -kH, h.n[3] + 2 * kH, -kH, h.n[3] + kH - 1, s);
  if (rc) return rc;
  return launch_vlines<false>(c, h, f, f, 3, -kH + 1, h.n[2] + 4, -kH + 1, h.n[2] + kH - 2, s);
}

template <int CPT>
int launch_xy_pass_cpt(vlp4d_ctx *c, const HGrid &h, const double *fn, double *cxy, double dt, int *groups,
                       cudaStream_t s) {
  const size_t smem = plane_bytes(h);
  auto k = k_mpi_xy_pass<CPT>;
  VLP4D_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 0;
  VLP4D_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, 512, smem));
  long long grid = (long long)c->num_sms * (per_sm > 0 ? per_sm : 1);
  const long long planes = (long long)h.n[2] * h.n[3];
  if (grid > planes) grid = planes;
  if (grid > c->rho_part_groups) grid = c->rho_part_groups;
  k<<<(unsigned)grid, 512, smem, s>>>(fn, cxy, h, plane_stride(h), dt, std::pow(h.alpha, h.n[0] + 3),
                                      std::pow(h.alpha, h.n[1] + 3), c->rho_part, c->d_err);
  VLP4D_LAUNCH_CHECK();
  *groups = (int)grid;
  return VLP4D_OK;
}

// The fused x/y pass: fn's grid points -> coefficients of the extended
// (x, y) planes in cxy (interior v planes) and the moment partials of the
// 2D advection by dt.
int launch_xy_pass(vlp4d_ctx *c, const HGrid &h, const double *fn, double *cxy, double dt, int *groups,
                   cudaStream_t s) {
  if (plane_bytes(h) > (size_t)smem_limit(c))
    return fail_msg(VLP4D_ERR_UNSUPPORTED, "mpi_step: the (x, y) plane does not fit in shared memory");
  // Cells per thread: the smallest CPT whose strips (nx columns of
  // ceil(ny / CPT) strips) fit in the 512 threads.
  const long long nx = h.n[0], ny = h.n[1];
  auto fits = [&](long long cpt) { return nx * ((ny + cpt - 1) / cpt) <= 512; };
  if (nx > 512) return fail_msg(VLP4D_ERR_UNSUPPORTED, "mpi_step: nx above 512");
  if (fits(1)) return launch_xy_pass_cpt<1>(c, h, fn, cxy, dt, groups, s);
  if (fits(2)) return launch_xy_pass_cpt<2>(c, h, fn, cxy, dt, groups, s);
  if (fits(4)) return launch_xy_pass_cpt<4>(c, h, fn, cxy, dt, groups, s);
  if (fits(8)) return launch_xy_pass_cpt<8>(c, h, fn, cxy, dt, groups, s);
  if (fits(16)) return launch_xy_pass_cpt<16>(c, h, fn, cxy, dt, groups, s);
  if (fits(32)) return launch_xy_pass_cpt<32>(c, h, fn, cxy, dt, groups, s);
  return fail_msg(VLP4D_ERR_UNSUPPORTED, "mpi_step: the x/y plane needs more than 32 cells per thread");
}

// 4D advection of the coefficients c4 into fn's grid points; MOMENT: with
// the moment partials (groups written to *groups) and per-block sums of
// squares (*blocks pairs in c->mpi_part).
template <bool EXACT, bool MOMENT>
int launch_advect_4d(vlp4d_ctx *c, const HGrid &h, const double *c4, double *fn, double dt, int *groups,
                     long long *blocks, cudaStream_t s) {
  const PlaneTiles t(h, true);
  const long long bx = t.nxt, by = t.nyt;
  const long long planes = (long long)h.n[2] * h.n[3];
  // One resident wave: every block walks the planes p = z, z + G, ... at the
  // same pace, so the blocks in flight read neighbouring (vx, vy) slabs.
  int per_sm = 0;
  VLP4D_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_mpi_advect_4d<EXACT, MOMENT>, t.threads, 0));
  long long G = ((long long)c->num_sms * (per_sm > 0 ? per_sm : 1)) / (bx * by);
  if (G < 1) G = 1;
  if (G > planes) G = planes;
  if (MOMENT) {
    if (G > c->rho_part_groups) G = c->rho_part_groups;
    if (G * bx * by > c->mpi_part_cap) G = c->mpi_part_cap / (bx * by);
    if (G < 1) return fail_msg(VLP4D_ERR_UNSUPPORTED, "mpi 4D advection: too many (x, y) blocks for the partials");
  }
  const dim3 grid((unsigned)bx, (unsigned)by, (unsigned)G);
  k_mpi_advect_4d<EXACT, MOMENT><<<grid, t.threads, 0, s>>>(c4, fn, c->ex, c->ey, h, t.W, t.H, dt, c->rho_part,
                                                             c->mpi_part, c->d_err);
  VLP4D_LAUNCH_CHECK();
  if (groups) *groups = (int)G;
  if (blocks) *blocks = G * bx * by;
  return VLP4D_OK;
}

// The ring, the field around the tile, the predictor's x and y parts.
size_t tile4_smem(const Tile4 &T) {
  return sizeof(double) * ((size_t)kRing * T.slab + 2 * (size_t)T.PX * T.RY + (size_t)kTileX * T.W * T.V +
                           2 * (size_t)kTileY * T.R * T.YG) +
         sizeof(int) * (size_t)T.RY * T.RV;
}

// Tiles of k_mpi_advect_4d_tile: x in equal tiles of at most 32, then the
// (YG, V) with YG * V threads rows of W whose ring fits and which takes the
// fewest (rounds of tiles over the SMs) x (steps of a segment): a tile past
// the grid's edge idles, and every segment starts with five slabs and their
// latency, about two steps' worth.  False: nothing fits (or more partials
// than the context holds), and the cell-per-thread kernel runs (48 x 44 x 40
// x 36 in the reference's arithmetic: 0.555 ms against 0.366 for the tiles).
bool tile4_config(const vlp4d_ctx *c, const HGrid &h, int cells, int threads, bool moment, Tile4 &T) {
  const int lim = smem_limit(c) - 1024;
  const long long nx = h.n[0], ny = h.n[1], nvx = h.n[2], nvy = h.n[3];
  Tile4 t;
  t.R = cells;
  t.nxt = (int)((nx + 31) / 32);
  t.W = (int)((nx + t.nxt - 1) / t.nxt);
  t.PX = t.W + 4;
  t.magic = (unsigned)(((1ULL << 32) + t.PX - 1) / t.PX);
  double best = 0.;
  for (int yg = 1; yg <= 16; ++yg)
    for (int v = 1; v <= 16; ++v) {
      if (t.W * yg * v > threads) continue;
      t.YG = yg;
      t.V = v;
      t.RY = cells * yg + 4;
      t.RV = v + 4;
      t.slab = t.PX * t.RY * t.RV;
      if ((long long)tile4_smem(t) > lim) continue;
      const long long nyt = (ny + cells * yg - 1) / (cells * yg), nvt = (nvx + v - 1) / v;
      if (nyt * nvt * t.nxt > (1 << 24)) continue;
      for (long long nseg = 1; nseg <= nvy && nseg <= 64; ++nseg) {
        const long long Q = (nvy + nseg - 1) / nseg;
        if ((nvy + Q - 1) / Q != nseg) continue;
        if (moment && nvt * nseg > c->rho_part_groups) continue;
        const long long items = t.nxt * nyt * nvt * nseg;
        // A step of a tile: its warps share the SM's FP64 pipe on top of the
        // latency of one warp's own chain.
        const int warps = (t.W * yg * v + 31) / 32;
        const double cost = (double)((items + c->num_sms - 1) / c->num_sms) * (Q + 2) * (warps + 8);
        if (best > 0. && cost >= best) continue;
        best = cost;
        T = t;
        T.nyt = (int)nyt;
        T.nvt = (int)nvt;
        T.Q = (int)Q;
        T.nseg = (int)nseg;
        T.nitems = (int)items;
      }
    }
  return best > 0.;
}

// Whether the tiles beat one thread per cell in the reference's arithmetic.  The
// tiles pay for idle rims, for the slabs that mixed first taps add and, in one
// round, for the slowest tile; a thread per cell reads all 256 taps through L1.
// Both times are estimates, in us on 148 SMs, fitted to 460 grids of 10 to 96
// points a side in fields of four modes (11 and 12% off, rms): tiles Q + 0.5
// steps of 4.8 + 0.66 per warp, a quarter (a tenth) more where a vx (vy) grid line
// has no velocity and its feet lie on either side; threads 0.12 ns per cell of
// whole rows, up to 0.21 in tiles of short rows.  Over those grids the choice
// gains 1.20 against tiles everywhere and 1.28 against one thread per cell in
// blocks of 32 x 8 everywhere.  Tiles / threads: 26 x 16 x 16 x 14 40 / 20, 16^4
// 31 / 18; 48 x 44 x 40 x 36 336 / 520, 38 x 55 x 72 x 64 1330 / 2230.
bool tile4_faster(const vlp4d_ctx *c, const HGrid &h, const Tile4 &T) {
  auto still = [&](int d) {  // a grid line of no velocity
    const double k = std::round(-h.minp[d] / h.dx[d]);
    return k >= 0. && k < h.n[d] && std::fabs(h.minp[d] + k * h.dx[d]) < 1e-9 * h.dx[d];
  };
  const int rounds = (T.nitems + c->num_sms - 1) / c->num_sms, warps = (T.W * T.YG * T.V + 31) / 32;
  const double tiles = 5.6 + (rounds == 1 ? 1. : 0.8 * rounds) * (T.Q + 0.52) * (4.8 + 0.66 * warps) *
                                 (1. + (still(2) ? 0.24 : 0.) + (still(3) ? 0.1 : 0.));
  const PlaneTiles p(h, true);
  const double kcells = 1e-3 * p.nxt * p.nyt * p.threads * h.n[2] * h.n[3];
  const double threads = 8.7 + kcells * (p.W == 32 ? 0.1215 : 0.206 - 0.092 * h.n[0] / (32. * p.nxt));
  return tiles < threads;
}

template <bool EXACT, bool MOMENT, int PXC>
int run_advect_4d_tile(vlp4d_ctx *c, const HGrid &h, const Tile4 &T, const double *c4, double *fn, double dt,
                       long long *blocks, cudaStream_t s) {
  auto k = k_mpi_advect_4d_tile<EXACT, MOMENT, PXC>;
  const size_t smem = tile4_smem(T);
  VLP4D_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int grid = T.nitems < c->num_sms ? T.nitems : c->num_sms;
  k<<<grid, TileShape<EXACT>::threads, smem, s>>>(c4, fn, c->ex, c->ey, h, T, dt, c->rho_part, c->mpi_part, c->d_err);
  VLP4D_LAUNCH_CHECK();
  if (blocks) *blocks = grid;
  return VLP4D_OK;
}

// The 4D advection of the coefficients c4 into fn's grid points, with the
// moment partials (groups written to *groups) and per-block sums of squares
// (*blocks pairs in c->mpi_part) when MOMENT.
template <bool EXACT, bool MOMENT>
int launch_advect_4d_any(vlp4d_ctx *c, const HGrid &h, const double *c4, double *fn, double dt, int *groups,
                         long long *blocks, cudaStream_t s) {
  // Sought once per context: up to 60 us of host time (10 x 10 x 100 x 300).
  MpiTiles &tiles = c->mpi_tiles[EXACT];
  std::call_once(tiles.once, [&] {
    tiles.use = c->fused && tile4_config(c, h, TileShape<EXACT>::cells, TileShape<EXACT>::threads, MOMENT, tiles.T) &&
                (!EXACT || c->fused_only || tile4_faster(c, h, tiles.T));
  });
  if (!tiles.use) return launch_advect_4d<EXACT, MOMENT>(c, h, c4, fn, dt, groups, blocks, s);
  const Tile4 &T = tiles.T;
  if (groups) *groups = T.nvt * T.nseg;
  if (T.PX == 36) return run_advect_4d_tile<EXACT, MOMENT, 36>(c, h, T, c4, fn, dt, blocks, s);
  return run_advect_4d_tile<EXACT, MOMENT, 0>(c, h, T, c4, fn, dt, blocks, s);
}

int launch_rho_halo(vlp4d_ctx *c, const HGrid &h, const double *f, cudaStream_t s) {
  const long long nxy = (long long)h.n[0] * h.n[1];
  const int groups = c->rho_groups;
  k_mpi_rho_partial<<<dim3((unsigned)((nxy + 255) / 256), groups), 256, 0, s>>>(f, c->rho_part, h, groups);
  VLP4D_LAUNCH_CHECK();
  return launch_rho_finish(c, groups, s);
}

int launch_l2_halo(vlp4d_ctx *c, const HGrid &h, const double *f, int iter, cudaStream_t s) {
  long long blocks = (long long)c->num_sms * 4;
  if (blocks > c->mpi_part_cap) blocks = c->mpi_part_cap;
  k_mpi_l2_partial<<<(unsigned)blocks, 256, 0, s>>>(f, h, c->mpi_part);
  VLP4D_LAUNCH_CHECK();
  const double scale = h.dx[0] * h.dx[1] * h.dx[2] * h.dx[3];
  k_mpi_l2_finish<<<1, 32, 0, s>>>(c->mpi_part, blocks, scale, c->l2norm + iter);
  VLP4D_LAUNCH_CHECK();
  return VLP4D_OK;
}

}  // namespace
}  // namespace vlp4d

using namespace vlp4d;

extern "C" {

size_t vlp4d_mpi_size(const vlp4d_ctx *ctx) {
  if (!ctx) return 0;
  size_t n = 1;
  for (int k = 0; k < 4; ++k) n *= (size_t)(ctx->g.n[k] + 2 * kH);
  return n;
}

int vlp4d_mpi_init_case(vlp4d_ctx *ctx, void *fn, void *stream) {
  int rc = mpi_check(ctx, "mpi_init_case");
  if (rc || (rc = mpi_check_ptr(fn, "mpi_init_case"))) return rc;
  const int ic = ctx->dom.idcase;
  if (ic != 2 && ic != 5 && ic != 10 && ic != 20)
    return fail_msg(VLP4D_ERR_INVALID_ARG, "mpi_init_case: unknown test case (the reference aborts, Init.cpp:142-145)");
  k_mpi_init_case<<<ctx->num_sms * 8, 256, 0, (cudaStream_t)stream>>>((double *)fn, make_hgrid(ctx), ic);
  VLP4D_LAUNCH_CHECK();
  return VLP4D_OK;
}

int vlp4d_mpi_halo_fill(vlp4d_ctx *ctx, void *fn, void *stream) {
  int rc = mpi_check(ctx, "mpi_halo_fill");
  if (rc || (rc = mpi_check_ptr(fn, "mpi_halo_fill"))) return rc;
  return launch_halo(ctx, make_hgrid(ctx), (double *)fn, (cudaStream_t)stream);
}

int vlp4d_mpi_spline_xy(vlp4d_ctx *ctx, void *fn, void *stream) {
  int rc = mpi_check(ctx, "mpi_spline_xy");
  if (rc || (rc = mpi_check_ptr(fn, "mpi_spline_xy"))) return rc;
  return launch_spline_xy_exact(ctx, make_hgrid(ctx), (double *)fn, (cudaStream_t)stream);
}

int vlp4d_mpi_spline_vxvy(vlp4d_ctx *ctx, void *fn, void *stream) {
  int rc = mpi_check(ctx, "mpi_spline_vxvy");
  if (rc || (rc = mpi_check_ptr(fn, "mpi_spline_vxvy"))) return rc;
  return launch_spline_vxvy_exact(ctx, make_hgrid(ctx), (double *)fn, (cudaStream_t)stream);
}

int vlp4d_mpi_advect_2d(vlp4d_ctx *ctx, void *fn, void *fn_tmp, double dt, void *stream) {
  int rc = mpi_check(ctx, "mpi_advect_2d");
  if (rc || (rc = mpi_check_ptr(fn, "mpi_advect_2d")) || (rc = mpi_check_ptr(fn_tmp, "mpi_advect_2d"))) return rc;
  if (fn == fn_tmp) return fail_msg(VLP4D_ERR_INVALID_ARG, "mpi_advect_2d: fn and fn_tmp must differ");
  const HGrid h = make_hgrid(ctx);
  cudaStream_t s = (cudaStream_t)stream;
  VLP4D_CUDA_TRY(cudaMemcpyAsync(fn_tmp, fn, sizeof(double) * (size_t)h.total(), cudaMemcpyDeviceToDevice, s));
  const PlaneTiles t(h, false);
  // Sixteen blocks of 256 threads per SM.
  const long long tiles = (long long)t.nxt * t.nyt, planes = (long long)h.n[2] * h.n[3];
  long long G = ((long long)ctx->num_sms * 16 * 256 + tiles * t.threads - 1) / (tiles * t.threads);
  if (G > planes) G = planes;
  k_mpi_advect_2d<<<dim3((unsigned)t.nxt, (unsigned)t.nyt, (unsigned)G), t.threads, 0, s>>>(
      (const double *)fn_tmp, (double *)fn, h, t.W, t.H, dt, ctx->d_err);
  VLP4D_LAUNCH_CHECK();
  return VLP4D_OK;
}

int vlp4d_mpi_advect_4d(vlp4d_ctx *ctx, void *fn, void *tmp_fn, double dt, void *stream) {
  int rc = mpi_check(ctx, "mpi_advect_4d");
  if (rc || (rc = mpi_check_ptr(fn, "mpi_advect_4d")) || (rc = mpi_check_ptr(tmp_fn, "mpi_advect_4d"))) return rc;
  if (fn == tmp_fn) return fail_msg(VLP4D_ERR_INVALID_ARG, "mpi_advect_4d: fn and tmp_fn must differ");
  const HGrid h = make_hgrid(ctx);
  cudaStream_t s = (cudaStream_t)stream;
  VLP4D_CUDA_TRY(cudaMemcpyAsync(tmp_fn, fn, sizeof(double) * (size_t)h.total(), cudaMemcpyDeviceToDevice, s));
  return launch_advect_4d_any<true, false>(ctx, h, (const double *)tmp_fn, (double *)fn, dt, nullptr, nullptr, s);
}

int vlp4d_mpi_field(vlp4d_ctx *ctx, const void *fn, void *stream) {
  int rc = mpi_check(ctx, "mpi_field");
  if (rc || (rc = mpi_check_ptr(fn, "mpi_field"))) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  if ((rc = launch_rho_halo(ctx, make_hgrid(ctx), (const double *)fn, s))) return rc;
  return launch_field_poisson(ctx, s);
}

int vlp4d_mpi_l2norm(vlp4d_ctx *ctx, const void *fn, int iter, void *stream) {
  int rc = mpi_check(ctx, "mpi_l2norm");
  if (rc || (rc = mpi_check_ptr(fn, "mpi_l2norm"))) return rc;
  if (iter < 0 || iter >= ctx->hist_len) return fail_msg(VLP4D_ERR_INVALID_ARG, "mpi_l2norm: iter outside [0, nbiter]");
  return launch_l2_halo(ctx, make_hgrid(ctx), (const double *)fn, iter, (cudaStream_t)stream);
}

int vlp4d_mpi_step(vlp4d_ctx *ctx, void *fn, void *fnp1, int iter, void *stream) {
  int rc = mpi_check(ctx, "mpi_step");
  if (rc || (rc = mpi_check_ptr(fn, "mpi_step")) || (rc = mpi_check_ptr(fnp1, "mpi_step"))) return rc;
  if (fn == fnp1) return fail_msg(VLP4D_ERR_INVALID_ARG, "mpi_step: fn and fnp1 must differ");
  if (iter < 0 || iter >= ctx->hist_len) return fail_msg(VLP4D_ERR_INVALID_ARG, "mpi_step: iter outside [0, nbiter]");
  const HGrid h = make_hgrid(ctx);
  cudaStream_t s = (cudaStream_t)stream;
  double *f = (double *)fn, *g = (double *)fnp1;
  const double dt = ctx->dom.dt;
  int groups = 0;
  // x/y: f's grid points -> x/y coefficients of the interior v planes (in g)
  // and the moment of the half-step 2D advection.
  if ((rc = launch_xy_pass(ctx, h, f, g, 0.5 * dt, &groups, s))) return rc;
  if ((rc = launch_rho_finish(ctx, groups, s))) return rc;
  if ((rc = launch_field_poisson(ctx, s))) return rc;
  // vx lines of the interior vy planes (g -> f), then vy lines of every vx
  // position (in place in f): f holds the 4D coefficients.
  if ((rc = launch_vlines_fused(ctx, h, g, f, 2, 0, h.n[3], 0, h.n[3] - 1, s))) return rc;
  if ((rc = launch_vlines_fused(ctx, h, f, f, 3, -kH, h.n[2] + 2 * kH, -kH + 1, h.n[2] + kH - 2, s)))
    return rc;
  long long blocks = 0;
  if ((rc = launch_advect_4d_any<false, true>(ctx, h, f, g, dt, &groups, &blocks, s))) return rc;
  if ((rc = launch_rho_finish(ctx, groups, s))) return rc;
  if ((rc = launch_field_poisson(ctx, s))) return rc;
  if ((rc = launch_diags(ctx, iter, s))) return rc;
  const double scale = h.dx[0] * h.dx[1] * h.dx[2] * h.dx[3];
  k_mpi_l2_finish<<<1, 32, 0, s>>>(ctx->mpi_part, blocks, scale, ctx->l2norm + iter);
  VLP4D_LAUNCH_CHECK();
  return VLP4D_OK;
}

}  // extern "C"
