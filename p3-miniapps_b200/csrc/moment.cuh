// Second stage of the velocity moment (field_rho, miniapps/vlp4d/thrust/
// field.cpp:6-32): rho[ixy] = dvx * dvy * (sum over the plane groups of the
// FP64 partial sums part[group][ixy]).
//
// The groups are added in a fixed order that does not depend on the launch
// shape: S contiguous ranges of groups, [s*G/S, (s+1)*G/S), each summed in
// increasing group order, then the slices in a fixed order (slice_sum).  Blocks of
// some cells x S slices sum the slices of a cell in
// parallel (the partials of small grids are few cells of many groups; one
// thread per cell left most of the GPU idle and the kernel bound by the
// latency of its sequential loads).
#pragma once

namespace vlp4d {

// Cells of a block and slices of the groups: 32 x 16, or 16 x 32 for many
// groups (small planes: 1024 groups of 32 x 32 cells 3.9 us against 5.3; 74
// groups of 128 x 128 cells 9.2 against 5.8).
constexpr int kMomentThreads = 512;
inline bool moment_wide(int groups) { return groups >= 512; }

// The sum of a cell's slices: 16 in increasing order, 32 in four chains of
// eight and their pairs.  (One chain of 32 has 1.66e-16 rms error on 64 to 1024
// Maxwellian planes, of 16 1.25e-16, four of eight 0.86e-16.)
template <int CELLS, int SLICES>
__device__ __forceinline__ double slice_sum(const double (&sl)[SLICES][CELLS], int cx) {
  static_assert(SLICES == 16 || SLICES == 32, "slices");
  constexpr int chains = SLICES == 32 ? 4 : 1, len = SLICES / chains;
  double sum[chains];
#pragma unroll
  for (int q = 0; q < chains; ++q) {
    sum[q] = 0.0;
#pragma unroll
    for (int k = 0; k < len; ++k) sum[q] += sl[q * len + k][cx];
  }
  if constexpr (chains == 4) return (sum[0] + sum[1]) + (sum[2] + sum[3]);
  return sum[0];
}

template <int kMomentCells, int kMomentSlices>
__device__ __forceinline__ void moment_finish(const double *__restrict__ part, double *__restrict__ rho,
                                              long long nxy, int groups, double dvx, double dvy) {
  __shared__ double sl[kMomentSlices][kMomentCells];
  const int cx = threadIdx.x % kMomentCells, s = threadIdx.x / kMomentCells;
  const long long ixy = (long long)blockIdx.x * kMomentCells + cx;
  const int g0 = (int)((long long)groups * s / kMomentSlices);
  const int g1 = (int)((long long)groups * (s + 1) / kMomentSlices);
  double acc = 0.0;
  if (ixy < nxy) {
    int g = g0;
    // Loads of eight groups issued before their adds (fixed order).
    for (; g + 8 <= g1; g += 8) {
      double v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = __ldcg(part + (long long)(g + k) * nxy + ixy);
#pragma unroll
      for (int k = 0; k < 8; ++k) acc += v[k];
    }
    for (; g < g1; ++g) acc += __ldcg(part + (long long)g * nxy + ixy);
  }
  sl[s][cx] = acc;
  __syncthreads();
  if (s == 0 && ixy < nxy) rho[ixy] = slice_sum(sl, cx) * dvx * dvy;  // field.cpp:23 (sum * dvx * dvy)
}

// The whole moment in one launch where a cell has few planes: a block sums
// kRhoSmallCells neighbouring cells in kRhoSmallSlices contiguous ranges of
// the nv planes, then the ranges (slice_sum).  (16^4 FP64: 3.2 us against
// 1.9 + 2.3 and a launch; moment, field and diagnostic 24.3 -> 21.4 us.)  Beyond
// kRhoSmallPlanes planes, or where the cells alone fill the GPU, the two-stage
// sum has the more loads in flight.
constexpr int kRhoSmallCells = 16, kRhoSmallSlices = 32, kRhoSmallPlanes = 1024;
inline bool rho_small(long long nxy, long long nv) { return nv <= kRhoSmallPlanes && nxy <= 8192; }

template <typename T>
__device__ __forceinline__ void moment_small(const T *__restrict__ f, double *__restrict__ rho, long long nxy, int nv,
                                             double dvx, double dvy) {
  __shared__ double sl[kRhoSmallSlices][kRhoSmallCells];
  const int cx = threadIdx.x % kRhoSmallCells, s = threadIdx.x / kRhoSmallCells;
  const long long ixy = (long long)blockIdx.x * kRhoSmallCells + cx;
  const int v0 = nv * s / kRhoSmallSlices, v1 = nv * (s + 1) / kRhoSmallSlices;
  double acc = 0.0;
  if (ixy < nxy) {
    const T *p = f + ixy + v0 * nxy;
#pragma unroll 16
    for (int v = v0; v < v1; ++v, p += nxy) acc += (double)__ldg(p);
  }
  sl[s][cx] = acc;
  __syncthreads();
  if (s == 0 && ixy < nxy) rho[ixy] = slice_sum(sl, cx) * dvx * dvy;
}

}  // namespace vlp4d
