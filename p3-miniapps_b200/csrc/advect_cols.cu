// Sweeps of any shape by columns: the route of the grids that the pipelined
// plane and v-slab kernels decline (row widths that are no multiple of four,
// columns that do not fill their chunks, unaligned buffers) or serve with
// chunks of a few rows.  They replace one thread per output with all taps
// through L1, 6 loads per cell and direction or 36 for a pair of sweeps, by
// sliding windows: a thread walks its column with the last rows in registers.
//
// Reference: miniapps/vlp4d/thrust/advection.hpp:77-386.  Per output the
// arithmetic is that of the cell-per-thread kernels (interp6 of the first
// sweep, then of the second), so the results are the same bits.
#include "internal.cuh"
#include "stencil.cuh"

namespace vlp4d {

namespace {

__device__ __forceinline__ void cp_async_elem(double *dst, const double *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_elem(float *dst, const float *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}

// One output from N taps: the weights of the 6-tap line (interp6), or of the
// composed 11-tap line (FP64 plain, FP32 differences about tap 5).
template <int N>
__device__ __forceinline__ double interp_n(const double (&w)[N], const double (&f)[N]) {
  double acc = w[0] * f[0];
#pragma unroll
  for (int k = 1; k < N; ++k) acc = fma(w[k], f[k], acc);
  return acc;
}
template <int N>
__device__ __forceinline__ float interp_n(const float (&w)[N], const float (&f)[N]) {
  constexpr int mid = N == 6 ? 2 : 5;
  float acc = w[0] * (f[1] - f[0]);
#pragma unroll
  for (int k = 1; k < N - 1; ++k) acc = fmaf(w[k], f[k + 1] - f[k], acc);
  return f[mid] + acc;
}

struct XyCols {
  const void *fin;
  void *fout;
  int nx, ny, nvx, nvy;
  int W, nxt;        // columns of a tile, tiles along x
  int S, Rs, nch;    // strips of a tile, rows of a strip, tiles along y
  int G;             // plane groups
  StencilTable tx, ty;
  double *part;      // moment partials [G][nx * ny]
};
constexpr int kColsRows = 16;     // most rows of a strip
constexpr int kColsThreads = 256;
constexpr int kColsWidth = 128;   // most columns of a tile

// x and/or y sweep (TX, TY taps, 0: none) of the planes g, g + G, ... of one
// tile of W columns and S strips of Rs rows.  The plane's tile and halo are
// brought in by cp.async already shifted by the plane's x and y offsets and
// wrapped, so that tap k of output (i, j) is at (i + k, j + k); a thread owns
// a column of one strip, sweeps a row of it along x from six shared-memory
// loads and along y from its window of the last swept rows.
//
// Bound by the shared-memory pipe (six loads per swept row, (RM + 5) / Rs
// rows per output: 68% busy) and the latency of its sums.  FP64, x and y:
// 99 x 101 x 77 x 83, 332 us (3.1 TB/s); 127 x 127 x 96 x 96, 576 us (4.1);
// 45 x 39 x 51 x 43, 25 us against 76 for one thread per output.  With a
// branch per row and divisions in the loads: 461, 780 and 33 us.
template <typename T, int TX, int TY, int RM, bool RHO>
__global__ void __launch_bounds__(kColsThreads, 2) k_xy_cols(XyCols a) {
  pdl_wait();
  pdl_trigger();
  extern __shared__ __align__(16) unsigned char csm[];
  T *tile = reinterpret_cast<T *>(csm);
  constexpr int HX = TX ? TX - 1 : 0, HY = TY ? TY - 1 : 0;
  const int pitch = a.W + HX;
  int b = blockIdx.x;
  const int x0 = (b % a.nxt) * a.W;
  b /= a.nxt;
  const int y0 = (b % a.nch) * a.S * a.Rs, g = b / a.nch;
  const int cols = a.nx - x0 < a.W ? a.nx - x0 : a.W;
  const int rows = a.ny - y0 < a.S * a.Rs ? a.ny - y0 : a.S * a.Rs;
  const int ix = threadIdx.x % a.W, strip = threadIdx.x / a.W;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int nr = strip < a.S && ix < cols ? (rows - strip * a.Rs < a.Rs ? rows - strip * a.Rs : a.Rs) : 0;
  const long long nxy = (long long)a.nx * a.ny;
  const long long planes = (long long)a.nvx * a.nvy;
  double acc[RM];
  if (RHO) {
#pragma unroll
    for (int i = 0; i < RM; ++i) acc[i] = 0.;
  }
  const int slot = pitch * ((a.S - 1) * a.Rs + RM + HY);
  auto load = [&](long long p, T *dst) {
    const int ivx = (int)(p % a.nvx), ivy = (int)(p / a.nvx);
    const int gx0 = TX ? (x0 + a.tx.m[ivx]) % a.nx : x0;
    int gy = ((TY ? y0 + a.ty.m[ivy] : y0) + warp) % a.ny;
    // This lane's columns: every 32nd, wrapped (more than once where the
    // row is narrower than the stencil).
    constexpr int kCh = (kColsWidth + HX + 31) / 32;
    int at[kCh];
#pragma unroll
    for (int k = 0; k < kCh; ++k) {
      at[k] = gx0 + lane + 32 * k;
      if (lane + 32 * k < cols + HX)
        while (at[k] >= a.nx) at[k] -= a.nx;
    }
    const T *src = static_cast<const T *>(a.fin) + p * nxy;
    T *d = dst + warp * pitch + lane;
    const int step = nwarps % a.ny;
    for (int r = warp; r < rows + HY; r += nwarps, d += nwarps * pitch) {
      const T *row = src + (long long)gy * a.nx;
#pragma unroll
      for (int k = 0; k < kCh; ++k)
        if (lane + 32 * k < cols + HX) cp_async_elem(d + 32 * k, row + at[k]);
      gy += step;
      if (gy >= a.ny) gy -= a.ny;
    }
  };
  if (g < planes) load(g, tile);
  asm volatile("cp.async.commit_group;" ::: "memory");
  int buf = 0;
  for (long long p = g; p < planes; p += a.G, buf ^= 1) {
    const int ivx = (int)(p % a.nvx), ivy = (int)(p / a.nvx);
    // The next plane into the other slot while this one is swept.
    if (p + a.G < planes) load(p + a.G, tile + (buf ^ 1) * slot);
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    if (nr > 0) {
      T wx[TX ? TX : 1], wy[TY ? TY : 1];
      if (TX) {
#pragma unroll
        for (int k = 0; k < TX; ++k) wx[k] = __ldg(WeightsOf<T>::get(a.tx) + TX * ivx + k);
      }
      if (TY) {
#pragma unroll
        for (int k = 0; k < TY; ++k) wy[k] = __ldg(WeightsOf<T>::get(a.ty) + TY * ivy + k);
      }
      const T *q = tile + buf * slot + strip * a.Rs * pitch + ix;
      T *out = static_cast<T *>(a.fout) + p * nxy + (long long)(y0 + strip * a.Rs) * a.nx + x0 + ix;
      T win[TY ? TY : 1];
      // All RM rows, with no branch between them (rows past the strip's are
      // read from the tile's spare rows and not stored): the sweeps of
      // several rows are in flight together.
#pragma unroll
      for (int r = 0; r < RM + HY; ++r) {
        T v;
        if constexpr (TX != 0) {
          T t[TX];
#pragma unroll
          for (int k = 0; k < TX; ++k) t[k] = q[k];
          v = interp_n<TX>(wx, t);
        } else {
          v = q[0];
        }
        q += pitch;
        if constexpr (TY != 0) {
          win[r % (TY ? TY : 1)] = v;
          if (r >= HY) {
            T t[TY];
#pragma unroll
            for (int k = 0; k < TY; ++k) t[k] = win[(r + 1 + k) % (TY ? TY : 1)];
            v = interp_n<TY>(wy, t);
          }
        }
        if (r >= HY) {
          if (r - HY < nr) *out = v;
          out += a.nx;
          if (RHO) acc[r - HY] += (double)v;
        }
      }
    }
    __syncthreads();
  }
  if (RHO && nr > 0) {
    double *d = a.part + (long long)g * nxy + (long long)(y0 + strip * a.Rs) * a.nx + x0 + ix;
#pragma unroll
    for (int i = 0; i < RM; ++i)
      if (i < nr) d[(long long)i * a.nx] = acc[i];
  }
}

struct VCols {
  const void *fin;
  void *fout;
  int nxy, nvx, nvy;
  int ngx;      // groups of V vx
  int Q;        // output rows of a segment
  StencilTable tvx, tvy;
};
constexpr int kVColsThreads = 128;

// vx and/or vy sweep: a thread owns V consecutive vx of one (x, y) column and
// walks a segment of Q output rows along vy: per row it loads the V + 5 taps
// of its vx outputs (one row ahead, consecutive columns in consecutive
// lanes), sweeps them along vx and keeps the last six swept rows for vy.
//
// Bound by L2 where the arrays lie in it ((V + 5) / V x (Q + 5) / Q loads per
// cell), else by HBM: the vx taps that neighbouring groups share are L2 hits.
// FP64, vx and vy: 45 x 39 x 51 x 43, 15 us (4.1 TB/s of f) against 114 for
// one thread per output; 127 x 127 x 96 x 96, 626 us (3.8 TB/s).
template <typename T, bool DVX, bool DVY, int V>
__global__ void __launch_bounds__(kVColsThreads, 4) k_v_cols(VCols a) {
  pdl_wait();
  pdl_trigger();
  const unsigned gid = blockIdx.x * kVColsThreads + threadIdx.x;
  if (gid >= (unsigned)a.nxy * (unsigned)a.ngx) return;
  const int col = (int)(gid % (unsigned)a.nxy), ivx0 = (int)(gid / (unsigned)a.nxy) * V;
  constexpr int NT = DVX ? V + 5 : V, HY = DVY ? 5 : 0;
  const int iv0 = blockIdx.y * a.Q;
  const int rows = (a.nvy - iv0 < a.Q ? a.nvy - iv0 : a.Q) + HY;
  T wx[6], wy[6];
  int jx = ivx0, jy = iv0;
  if (DVX) {
    load_weights_dep(WeightsOf<T>::get(a.tvx), col, wx);
    jx += a.tvx.m[col];
  }
  if (DVY) {
    load_weights_dep(WeightsOf<T>::get(a.tvy), col, wy);
    jy = (iv0 + a.tvy.m[col]) % a.nvy;
  }
  int off[NT];
  jx %= a.nvx;
#pragma unroll
  for (int j = 0; j < NT; ++j) {
    off[j] = jx * a.nxy;
    if (++jx == a.nvx) jx = 0;
  }
  const long long ystride = (long long)a.nxy * a.nvx;
  const T *fin = static_cast<const T *>(a.fin) + col;
  T *out = static_cast<T *>(a.fout) + col + (long long)ivx0 * a.nxy + (long long)iv0 * ystride;
  T cur[NT], win[6][V];
  auto load = [&](int j, T (&t)[NT]) {
    const T *row = fin + (long long)j * ystride;
#pragma unroll
    for (int k = 0; k < NT; ++k) t[k] = row[off[k]];
  };
  load(jy, cur);
  for (int r0 = 0; r0 < rows; r0 += 6) {
#pragma unroll
    for (int u = 0; u < 6; ++u) {
      const int r = r0 + u;
      if (r < rows) {
        T nxt[NT];
        if (++jy == a.nvy) jy = 0;
        if (r + 1 < rows) load(jy, nxt);
#pragma unroll
        for (int v = 0; v < V; ++v)
          win[u][v] = DVX ? interp6(wx, cur[v], cur[(v + 1) % NT], cur[(v + 2) % NT], cur[(v + 3) % NT],
                                    cur[(v + 4) % NT], cur[(v + 5) % NT])
                          : cur[v];
        if (r >= HY) {
#pragma unroll
          for (int v = 0; v < V; ++v) {
            const T o = DVY ? interp6(wy, win[(u + 1) % 6][v], win[(u + 2) % 6][v], win[(u + 3) % 6][v],
                                      win[(u + 4) % 6][v], win[(u + 5) % 6][v], win[u][v])
                            : win[u][v];
            if (ivx0 + v < a.nvx) out[(long long)v * a.nxy] = o;
          }
          out += ystride;
        }
#pragma unroll
        for (int k = 0; k < NT; ++k) cur[k] = nxt[k];
      }
    }
  }
}

template <typename T, int TX, int TY, int RM, bool RHO>
int run_xy_cols(vlp4d_ctx *c, XyCols &a, cudaStream_t s) {
  auto k = k_xy_cols<T, TX, TY, RM, RHO>;
  const int threads = (a.W * a.S + 31) / 32 * 32;
  const size_t smem =
      2 * sizeof(T) * (size_t)(a.W + (TX ? TX - 1 : 0)) * ((a.S - 1) * a.Rs + RM + (TY ? TY - 1 : 0));
  if (smem > 200 * 1024) return VLP4D_ERR_UNSUPPORTED;
  VLP4D_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 0;
  VLP4D_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, threads, smem));
  if (per_sm < 1) return VLP4D_ERR_UNSUPPORTED;
  const long long tiles = (long long)a.nxt * a.nch, planes = (long long)a.nvx * a.nvy;
  long long G = (long long)per_sm * c->num_sms / tiles;
  if (G < 1) G = 1;
  if (G > planes) G = planes;
  if (RHO && G > c->rho_part_groups) G = c->rho_part_groups;
  // Equal numbers of planes per group, as far as they go.
  const long long per = (planes + G - 1) / G;
  G = (planes + per - 1) / per;
  if (G * tiles > 0x7fffffffLL) return VLP4D_ERR_UNSUPPORTED;
  a.G = (int)G;
  VLP4D_CUDA_TRY(launch_dep(c, k, dim3((unsigned)(G * tiles)), dim3(threads), smem, s, a));
  VLP4D_LAUNCH_CHECK();
  return VLP4D_OK;
}

// Tiles: columns in equal tiles of at most 128; strips of at most 16 rows
// (their moment sums are registers), as many of them in a block as 256
// threads hold, the rows spread evenly.
void xy_cols_tiles(const vlp4d_ctx *c, XyCols &a) {
  a.nx = c->g.n[0];
  a.ny = c->g.n[1];
  a.nvx = c->g.n[2];
  a.nvy = c->g.n[3];
  a.nxt = (a.nx + kColsWidth - 1) / kColsWidth;
  a.W = (a.nx + a.nxt - 1) / a.nxt;
  const int strips = (a.ny + kColsRows - 1) / kColsRows;
  int S = kColsThreads / a.W;
  if (S > strips) S = strips;
  a.nch = (strips + S - 1) / S;
  a.S = (strips + a.nch - 1) / a.nch;
  a.Rs = (a.ny + a.nch * a.S - 1) / (a.nch * a.S);
  // The last tile may be left without rows.
  a.nch = (a.ny + a.S * a.Rs - 1) / (a.S * a.Rs);
}

// RM: the rows of a strip rounded up to 8, 12 or 16.
template <typename T, int TX, int TY, bool RHO>
int run_xy_cols_rm(vlp4d_ctx *c, XyCols &a, cudaStream_t s) {
  if (a.Rs <= 8) return run_xy_cols<T, TX, TY, 8, RHO>(c, a, s);
  if (a.Rs <= 12) return run_xy_cols<T, TX, TY, 12, RHO>(c, a, s);
  return run_xy_cols<T, TX, TY, 16, RHO>(c, a, s);
}

template <typename T>
int dispatch_xy_cols(vlp4d_ctx *c, XyCols &a, int tx, int ty, bool rho, cudaStream_t s) {
  if (tx == 11) {  // the FP32 time loop's joined half steps
    if constexpr (sizeof(T) == 4) return run_xy_cols_rm<T, 11, 11, true>(c, a, s);
    else return VLP4D_ERR_UNSUPPORTED;
  }
  if (tx && ty) return rho ? run_xy_cols_rm<T, 6, 6, true>(c, a, s) : run_xy_cols_rm<T, 6, 6, false>(c, a, s);
  if (tx) return run_xy_cols_rm<T, 6, 0, false>(c, a, s);
  return run_xy_cols_rm<T, 0, 6, false>(c, a, s);
}

template <typename T, bool DVX, bool DVY, int V>
int run_v_cols(vlp4d_ctx *c, VCols &a, cudaStream_t s) {
  a.ngx = (a.nvx + V - 1) / V;
  const long long threads = (long long)a.nxy * a.ngx;
  if (threads > 0x7fffffffLL - kVColsThreads || (long long)a.nxy * a.nvx > 0x7fffffffLL) return VLP4D_ERR_UNSUPPORTED;
  const long long blocks = (threads + kVColsThreads - 1) / kVColsThreads;
  // Segments: rounds of resident blocks (four per SM) x rows walked.
  const long long slots = 4LL * c->num_sms;
  long long best = -1;
  for (int nseg = 1; nseg <= a.nvy && nseg <= 64; ++nseg) {
    const int Q = (a.nvy + nseg - 1) / nseg;
    if ((a.nvy + Q - 1) / Q != nseg) continue;
    const long long cost = (blocks * nseg + slots - 1) / slots * (Q + (DVY ? 5 : 0) + 2);
    if (best < 0 || cost < best) {
      best = cost;
      a.Q = Q;
    }
  }
  VLP4D_CUDA_TRY(launch_dep(c, k_v_cols<T, DVX, DVY, V>, dim3((unsigned)blocks, (unsigned)((a.nvy + a.Q - 1) / a.Q)),
                            dim3(kVColsThreads), 0, s, a));
  VLP4D_LAUNCH_CHECK();
  return VLP4D_OK;
}

}  // namespace

// Narrow planes leave most lanes of a tile's loads and sweeps idle, and planes
// of few cells most threads of a block: there one thread per output is faster
// (us, columns against threads: x, 11 x 38 x 88 x 48 FP32 18.3 / 14.4 and 9 x 64 x 64
// x 104 43.0 / 26.7; y, 11 x 38 x 88 x 48 22.7 / 14.4; x and y, 2 x 16 x 104 x 120 35.6 / 10.3
// and 1 x 87 x 48 x 62 34.5 / 8.2; with the moment 31.2 / 16.4).  The lines lie where
// the two are equal over 700 grids of 1 to 70 columns; a pair's 36 loads per output,
// and its moment as a pass of its own, make up for more idle lanes.
bool xy_cols_pay(const vlp4d_ctx *c, bool x, bool y, bool with_rho) {
  const int nx = c->g.n[0], ny = c->g.n[1];
  const long long nxy = c->g.nxy();
  if (x && y) return with_rho ? nx >= 4 && nxy >= 64 : nx >= 8 && ny >= 4 && nxy >= 64;
  return x ? nx >= (c->dtype == VLP4D_F32 ? 20 : 24) && nxy >= 128 : nx >= 17 && nxy >= 256;
}

int launch_xy_cols(vlp4d_ctx *c, const void *fn, void *fnp1, const StencilTable *tx, const StencilTable *ty, int taps,
                   bool with_rho, cudaStream_t s) {
  if (!c->fused || (!tx && !ty) || (taps == 11 && (!with_rho || c->dtype != VLP4D_F32)) || (with_rho && !(tx && ty)) ||
      !xy_cols_pay(c, tx, ty, with_rho))
    return VLP4D_ERR_UNSUPPORTED;
  XyCols a;
  a.fin = fn;
  a.fout = fnp1;
  a.part = c->rho_part;
  if (tx) a.tx = *tx;
  if (ty) a.ty = *ty;
  xy_cols_tiles(c, a);
  const int rc = c->dtype == VLP4D_F64 ? dispatch_xy_cols<double>(c, a, tx ? taps : 0, ty ? taps : 0, with_rho, s)
                                       : dispatch_xy_cols<float>(c, a, tx ? taps : 0, ty ? taps : 0, with_rho, s);
  if (rc || !with_rho) return rc;
  return launch_rho_finish(c, a.G, s);
}

int launch_v_cols(vlp4d_ctx *c, const void *fn, void *fnp1, const StencilTable *tvx, const StencilTable *tvy,
                  cudaStream_t s) {
  if (!c->fused || (!tvx && !tvy)) return VLP4D_ERR_UNSUPPORTED;
  VCols a;
  a.fin = fn;
  a.fout = fnp1;
  a.nxy = (int)c->g.nxy();
  a.nvx = c->g.n[2];
  a.nvy = c->g.n[3];
  if (tvx) a.tvx = *tvx;
  if (tvy) a.tvy = *tvy;
  if (c->dtype == VLP4D_F64) {
    if (tvx && tvy) return run_v_cols<double, true, true, 4>(c, a, s);
    return tvx ? run_v_cols<double, true, false, 4>(c, a, s) : run_v_cols<double, false, true, 4>(c, a, s);
  }
  if (tvx && tvy) return run_v_cols<float, true, true, 8>(c, a, s);
  return tvx ? run_v_cols<float, true, false, 8>(c, a, s) : run_v_cols<float, false, true, 8>(c, a, s);
}

}  // namespace vlp4d
