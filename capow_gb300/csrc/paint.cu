// Mass assignment (the reference's read_periodic_serial_ascii + add_to_grid + halo fold,
// src/read_data.c:32-179, 514-745) on the GPU.
//
// FP64 path (k_paint64): one thread per particle, the reference's double arithmetic,
// global FP64 atomics into zeroed grids. It is the plain FP64 GPU path.
//
// FP32 path (k_bucket_cta or k_bucket_warp -> k_tile_rec -> k_edge_fixup; deterministic: k_count -> k_scan -> k_scatter ->
// k_tile_rec_det): particles are bucketed into the output tiles their stencils touch (a counting sort; a particle near a tile face is
// listed in each neighbouring tile), then one CTA per tile accumulates every stencil tap of
// its particles in shared memory and writes the tile once with coalesced stores. Every grid
// cell is written exactly once: no memset of the grids, no global atomics on them. Particles
// within a few ulps of a discontinuity of the reference's rules (acceptance bounds, the TSC
// low-tap drop, the LOS==0 x shift, NN cell edges, non-finite input) take the exact FP64 rules
// (k_edge_fixup; in the deterministic variant, inside the tile kernel), so indices and acceptance match
// the reference bit for bit. The deterministic variant accumulates int64 fixed point in shared memory.
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>

#include "launch.cuh"
#include "paint.cuh"
#include "paint_dev.cuh"

#define FULL_MASK 0xffffffffu

// ------------------------------------------------------------------------------------------ util
__device__ __forceinline__ double warp_sum_d(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL_MASK, v, o);
  return v;
}
__device__ __forceinline__ float warp_sum_f(float v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL_MASK, v, o);
  return v;
}

// Reduce `nv` per-thread floats over the block in FP32 within each warp (32 terms) and in FP64
// across warps, and add them to global `dst` (one FP64 atomic per value and block).
template <int NV>
__device__ void block_add_f(const float (&v)[NV], double *const (&dst)[NV]) {
  __shared__ double redf[32][NV];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  float t[NV];
#pragma unroll
  for (int k = 0; k < NV; k++) t[k] = warp_sum_f(v[k]);
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < NV; k++) redf[wid][k] = (double)t[k];
  __syncthreads();
  if (wid == 0 && lane < NV) {
    double a = 0.0;
    for (int w = 0; w < nw; w++) a += redf[w][lane];
    if (a != 0.0) atomicAdd(dst[lane], a);
  }
  __syncthreads();
}

// Reduce `nv` per-thread doubles over the block and add them to global `dst`.
template <int NV>
__device__ void block_add(const double (&v)[NV], double *const (&dst)[NV]) {
  __shared__ double red[32][NV];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  double t[NV];
#pragma unroll
  for (int k = 0; k < NV; k++) t[k] = warp_sum_d(v[k]);
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < NV; k++) red[wid][k] = t[k];
  __syncthreads();
  if (wid == 0) {
#pragma unroll
    for (int k = 0; k < NV; k++) {
      double a = lane < nw ? red[lane][k] : 0.0;
      a = warp_sum_d(a);
      if (lane == 0 && a != 0.0) atomicAdd(dst[k], a);
    }
  }
  __syncthreads();
}

template <typename T>
__device__ __forceinline__ double ld64(const T *p, long long i) {
  return (double)p[i];
}

// ===================================================================================== FP64 path
// One field's deposits of a stencil that reaches a wrap, the halo or a write guard; their sum. Out of line: few particles
// take it, and the instruction cache holds the others' loop.
static __device__ __noinline__ double deposit64(const Geom &g, double *gp, double val, AxisTaps ax, AxisTaps ay, AxisTaps az) {
  double dsum = 0.0;
  for (int c = 0; c < az.n; c++) {
    if (!az.on[c]) continue;
    for (int b = 0; b < ay.n; b++) {
      if (!ay.on[b]) continue;
      for (int a = 0; a < ax.n; a++) {
        if (!ax.on[a]) continue;
        long long L = canon_index(g, ax.idx[a], ay.idx[b], az.idx[c]);
        if (L < 0) continue;
        double d = DMUL(DMUL(DMUL(val, ax.w[a]), ay.w[b]), az.w[c]);
        atomicAdd(gp + L, d);
        dsum += d;
      }
    }
  }
  return dsum;
}

// One particle per thread, K = InterpOrder taps an axis. The stencil of a particle away from the edges shares its
// products (val wx, val wx wy, the reference's order of multiplications) and takes its DC sum from the taps' sums.
// What bounds it: the FP64 pipe (2 lanes per clock and SM; busy 69% of the time). 2.1M particles on 256^3, TSC, two fields,
// two stencils: 2.2 ms; 3.6 with three multiplications and an addition per cell, runtime tap loops and 2432 CTAs.
template <typename T, int K>
__global__ void __launch_bounds__(256) k_paint64(Geom g, FieldSpec fs, PIn<T> in, long long n, GridPtrs grids,
                                                 DevStats *st) {
  double l_grid = 0, l_nsq = 0, l_v[4] = {0, 0, 0, 0}, l_dc[4] = {0, 0, 0, 0};  // l_dc[2 stencil + field]
  unsigned l_read = 0, l_out = 0;
  int fatal = 0, nonfin = 0;
  const int nf = fs.nfields;
  g.order = K;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    double x = ld64(in.x, i), y = ld64(in.y, i), z = ld64(in.z, i);
    double v = fs.need_v ? ld64(in.v, i) : 0.0;
    double w = in.w ? ld64(in.w, i) : 1.0;
    if (!(isfinite(x) && isfinite(y) && isfinite(z) && isfinite(v) && isfinite(w))) {
      nonfin = 1;
      continue;
    }
    if (g.los == 1) x = rsd_shift64(g, x, v);
    else if (g.los == 2) y = rsd_shift64(g, y, v);
    else if (g.los == 3) z = rsd_shift64(g, z, v);
    l_read++;
    if (outside_box(g, x, y, z)) {
      if (g.los == 0) {
        fatal = 1;
        atomicMax(&st->fatal_inv, ~0ULL - (unsigned long long)i);
        continue;
      }
      l_out++;
    }
    const double val[2] = {wpow64(w, v, fs.ea), wpow64(w, v, fs.eb)};
    for (int stn = 0; stn < (g.interlace ? 2 : 1); stn++) {
      AxisTaps ax, ay, az;
      double px = x, py = y, pz = z;
      if (stn) {
        px = DADD(x, g.hx);
        py = DADD(y, g.hy);
        pz = DADD(z, g.hz);
      }
      if (!exact_axes(g, px, py, pz, ax, ay, az)) continue;
      if (stn == 0) l_grid += w;
      bool plain = true;  // every tap on, none at a wrap or in the halo
#pragma unroll
      for (int q = 0; q < K; q++)
        plain = plain && ax.on[q] && ay.on[q] && az.on[q] && (unsigned)ax.idx[q] < (unsigned)g.nx &&
                (unsigned)ay.idx[q] < (unsigned)g.ny && (unsigned)az.idx[q] < (unsigned)g.nz;
      if (plain) {
        double sx = ax.w[0], sy = ay.w[0], sz = az.w[0];
#pragma unroll
        for (int q = 1; q < K; q++) {
          sx += ax.w[q];
          sy += ay.w[q];
          sz += az.w[q];
        }
        const double sum = sx * sy * sz;
        for (int f = 0; f < nf; f++) {
          double *gp = (double *)grids.g[stn * nf + f];
          const double vf = f ? val[1] : val[0];
          l_dc[stn * 2 + f] += vf * sum;
#pragma unroll
          for (int a = 0; a < K; a++) {
            const double va = DMUL(vf, ax.w[a]);
#pragma unroll
            for (int b = 0; b < K; b++) {
              const double vab = DMUL(va, ay.w[b]);
              double *row = gp + ((long long)ax.idx[a] * g.ny + ay.idx[b]) * g.row;
#pragma unroll
              for (int c = 0; c < K; c++) atomicAdd(row + az.idx[c], DMUL(vab, az.w[c]));
            }
          }
        }
        continue;
      }
      for (int f = 0; f < nf; f++)
        l_dc[stn * 2 + f] += deposit64(g, (double *)grids.g[stn * nf + f], f ? val[1] : val[0], ax, ay, az);
    }
    if (fs.moments) {  // src/read_data.c:132-138
      l_nsq += w;
      double wv = DMUL(w, v);
      l_v[0] += wv;
      wv = DMUL(wv, v);
      l_v[1] += wv;
      wv = DMUL(wv, v);
      l_v[2] += wv;
      wv = DMUL(wv, v);
      l_v[3] += wv;
    }
  }
  const double vals[12] = {(double)l_read, (double)l_out, l_grid, l_nsq, l_v[0], l_v[1], l_v[2], l_v[3],
                           l_dc[0], l_dc[1], l_dc[2], l_dc[3]};
  double *const dst[12] = {&st->nread, &st->nout, &st->ngrid, &st->nsq, &st->vr[0], &st->vr[1], &st->vr[2], &st->vr[3],
                           &st->dc[0], &st->dc[nf == 2 ? 1 : 3], &st->dc[nf], &st->dc[3]};
  block_add<12>(vals, dst);
  if (fatal) atomicOr(&st->fatal, 1);
  if (nonfin) atomicOr(&st->nonfinite, 1);
}

static int grid_blocks(long long n, int threads) {
  long long b = (n + threads - 1) / threads;
  if (b > 152LL * 16) b = 152LL * 16;
  if (b < 1) b = 1;
  return (int)b;
}

template <typename T>
static void launch_paint64_t(cudaStream_t s, const Geom &g, const FieldSpec &fs, const PIn<T> &in, long long n,
                             const GridPtrs &grids, DevStats *st) {
  auto *fn = g.order == 1 ? k_paint64<T, 1> : (g.order == 2 ? k_paint64<T, 2> : k_paint64<T, 3>);
  // one resident wave: each CTA ends with a reduction of twelve FP64 sums
  const int nb = std::min(grid_blocks(n, 256), resident_ctas((const void *)fn, 256, 0, 4096));
  fn<<<nb, 256, 0, s>>>(g, fs, in, n, grids, st);
}

void launch_paint64(cudaStream_t s, const Geom &g, const FieldSpec &fs, int dtype, const void *x, const void *y,
                    const void *z, const void *v, const void *w, long long n, const GridPtrs &grids, DevStats *st,
                    long long *launches) {
  if (dtype == CAPOW_F64) {
    PIn<double> in{(const double *)x, (const double *)y, (const double *)z, (const double *)v, (const double *)w};
    launch_paint64_t(s, g, fs, in, n, grids, st);
  } else {
    PIn<float> in{(const float *)x, (const float *)y, (const float *)z, (const float *)v, (const float *)w};
    launch_paint64_t(s, g, fs, in, n, grids, st);
  }
  (*launches)++;
}

// ===================================================================================== FP32 path
// Normal-stencil scales of one particle after the RSD shift, in FP32. Explicit round-to-nearest
// intrinsics keep the result identical in every kernel that recomputes it (the count, scatter
// and tile kernels must agree on each particle's tiles).
// Distinct tile coordinates along one axis, in registers (at most three: a footprint spans at
// most six cells and tiles are at least four cells long, except a short partial last tile).
struct AxisTiles {
  int t0, t1, t2, n;
};

__device__ __forceinline__ void add_tile(AxisTiles &a, int v) {
  const bool dup = ((a.n > 0) & (v == a.t0)) | ((a.n > 1) & (v == a.t1)) | ((a.n > 2) & (v == a.t2));
  const bool put = !dup;
  a.t0 = (put & (a.n == 0)) ? v : a.t0;
  a.t1 = (put & (a.n == 1)) ? v : a.t1;
  a.t2 = (put & (a.n >= 2)) ? v : a.t2;
  a.n = (put & (a.n < 3)) ? a.n + 1 : a.n;
}

__device__ __forceinline__ int tile_at(const AxisTiles &a, int k) { return k == 0 ? a.t0 : (k == 1 ? a.t1 : a.t2); }

__device__ __forceinline__ int tile_id(const TileGeo &tg, int bx, int by, int bz) {
  return (bx * tg.nby + by) * tg.nbz + bz;
}

// Cells any accepted stencil (normal and interlaced) of a particle at scale s can write along one
// axis, widened by the FP32 margin: [floor(s-m)-1, floor(s+m)+2] for TSC, [floor(s-m), floor(s+m)+2]
// for CIC, [floor(s-m), floor(s+m)+1] for NN. Wrapping axes (LOS == 0: periodic y, z and the x halo
// fold) take the cells modulo N; other axes clip to the grid. Returns false when nothing of the
// footprint lies in the grid (the particle is outside the box and rejected).
// [low, lim): where either stencil of a particle at s is accepted along a non-wrapping axis (lim = n,
// or n + 1 for the TSC x axis; low = 0, or -1/2 when the interlaced copy at s + 1/2 is painted too).
// A particle beyond that range by more than the margin is rejected by both and lies outside the box,
// so it is counted out without the exact rules.
__device__ __forceinline__ bool axis_range(float s, int n, bool wrap, int order, float m, float low, float lim,
                                           int &lo, int &hi) {
  if (!(s > -4.0f && s < (float)n + 4.0f)) return false;
  if (!wrap && (s < low - m || s >= lim + m)) return false;
  lo = __float2int_rd(__fsub_rn(s, m)) - (order == 3 ? 1 : 0);
  hi = __float2int_rd(__fadd_rn(s, m)) + (order == 1 ? 1 : 2);
  if (!wrap) {
    lo = lo < 0 ? 0 : lo;
    hi = hi > n - 1 ? n - 1 : hi;
    return lo <= hi;
  }
  const int span = hi - lo;
  // s > -4 and margin < 0.25 give -6 <= lo <= n + 2, and n >= 4: these corrections bring lo into [0, n)
  lo += lo < 0 ? n : 0;
  lo += lo < 0 ? n : 0;
  lo -= lo >= n ? n : 0;
  hi = lo + span;  // cells beyond n - 1 wrap when used
  return true;
}

// The tiles of the cells lo..hi (hi may pass n - 1 on a wrapping axis): the piece inside the grid
// covers tiles lo >> shift .. min(hi, n - 1) >> shift, the wrapped piece 0 .. (hi - n) >> shift.
__device__ __forceinline__ bool axis_footprint(float s, int n, int shift, bool wrap, int order, float m, float low,
                                               float lim, AxisTiles &T) {
  T.n = 0;
  T.t0 = T.t1 = T.t2 = 0;
  int lo, hi;
  if (!axis_range(s, n, wrap, order, m, low, lim, lo, hi)) return false;
  const int top = hi < n - 1 ? hi : n - 1;
  const int a0 = lo >> shift, a1 = top >> shift;  // a1 - a0 <= 2: the footprint spans at most 6 cells
  T.t0 = a0;
  T.t1 = a0 + 1;
  T.t2 = a0 + 2;
  T.n = a1 - a0 + 1;
  if (hi >= n) {  // the wrapped piece (rare: a periodic axis near its last cell)
    const int wtop = hi - n < n - 1 ? hi - n : n - 1;
    for (int t = 0; t <= (wtop >> shift); t++) add_tile(T, t);
  }
  return true;
}

// All tiles of a particle. The first tile of each axis list gives the particle's home tile (the one
// tile that counts it in the statistics).
__device__ __forceinline__ bool footprint(const Geom &g, const TileGeo &tg, float sx, float sy, float sz,
                                          AxisTiles &TX, AxisTiles &TY, AxisTiles &TZ) {
  const bool wrap = g.los == 0;
  const float limx = (float)g.nx + (g.order == 3 ? 1.0f : 0.0f);  // src/read_data.c:618-619
  const float low = g.interlace ? -0.5f : 0.0f;
  if (!axis_footprint(sx, g.nx, tg.lx, wrap, g.order, g.margin, low, limx, TX)) return false;
  if (!axis_footprint(sy, g.ny, tg.ly, wrap, g.order, g.margin, low, (float)g.ny, TY)) return false;
  if (!axis_footprint(sz, g.nz, tg.lz, wrap, g.order, g.margin, low, (float)g.nz, TZ)) return false;
  // CIC rounding edge: a y index equal to NY makes the reference's linear index land in row 0 of
  // the next x slice (src/read_data.c:592-593); that row's tile joins the list.
  if (g.order == 2 && sy > (float)g.ny - 1.5f - g.margin) add_tile(TY, 0);
  return true;
}

// The home tile without building the lists: the tile of the first cell of each axis range
// (the same tile footprint() puts first). Returns -1 when the footprint misses the grid.
__device__ __forceinline__ int home_of(const Geom &g, const TileGeo &tg, float sx, float sy, float sz) {
  const bool wrap = g.los == 0;
  int lx, hx, ly, hy, lz, hz;
  const float limx = (float)g.nx + (g.order == 3 ? 1.0f : 0.0f);
  const float low = g.interlace ? -0.5f : 0.0f;
  if (!axis_range(sx, g.nx, wrap, g.order, g.margin, low, limx, lx, hx)) return -1;
  if (!axis_range(sy, g.ny, wrap, g.order, g.margin, low, (float)g.ny, ly, hy)) return -1;
  if (!axis_range(sz, g.nz, wrap, g.order, g.margin, low, (float)g.nz, lz, hz)) return -1;
  return tile_id(tg, lx >> tg.lx, ly >> tg.ly, lz >> tg.lz);
}

// Exact FP64 view of one particle (RSD shift in the reference's order).
template <typename T>
__device__ __forceinline__ void exact_pos(const Geom &g, const FieldSpec &fs, const PIn<T> &in, long long i, double &x,
                                          double &y, double &z, double &v, double &w) {
  x = (double)in.x[i];
  y = (double)in.y[i];
  z = (double)in.z[i];
  v = fs.need_v ? (double)in.v[i] : 0.0;
  w = in.w ? (double)in.w[i] : 1.0;
  if (g.los == 1) x = rsd_shift64(g, x, v);
  else if (g.los == 2) y = rsd_shift64(g, y, v);
  else if (g.los == 3) z = rsd_shift64(g, z, v);
}

// Decode a canonical padded index into cell coordinates.
__device__ __forceinline__ void decode(const Geom &g, long long L, int &ix, int &iy, int &iz) {
  ix = (int)(L / g.slice);
  long long r = L - (long long)ix * g.slice;
  iy = (int)(r / g.row);
  iz = (int)(r - (long long)iy * g.row);
}

// Warp-aggregated tile counters over runs: consecutive lanes naming the same tile form a run and
// share one atomic, issued by the run's first lane (particles that arrive in spatial order form
// long runs; any order stays correct). Every lane of the warp must call this; lanes with key < 0
// take no slot. Returns the lane's slot: the counter's old value plus its offset in the run.
__device__ __forceinline__ unsigned warp_run_add(unsigned *counter, int key, bool want_slot) {
  const int lane = threadIdx.x & 31;
  const int prev = __shfl_up_sync(FULL_MASK, key, 1);
  const unsigned heads = __ballot_sync(FULL_MASK, lane == 0 || key != prev);
  const unsigned after = heads & ~((2u << lane) - 1u);  // run heads above this lane (0 for lane 31)
  const int head = 31 - __clz(heads & ((2u << lane) - 1u));
  unsigned base = 0;
  if (head == lane && key >= 0) base = atomicAdd(counter + key, (unsigned)((after ? __ffs(after) - 1 : 32) - lane));
  if (!want_slot) return 0;
  base = __shfl_sync(FULL_MASK, base, head);
  return base + (unsigned)(lane - head);
}

// Tile id of the lane's (a, b, c)-th footprint tile, or -1 when the lane has none there.
__device__ __forceinline__ int tile_key(const TileGeo &tg, bool has, const AxisTiles &TX, const AxisTiles &TY,
                                        const AxisTiles &TZ, int a, int b, int c) {
  const int id = tile_id(tg, tile_at(TX, a), tile_at(TY, b), tile_at(TZ, c));
  return (has & (a < TX.n) & (b < TY.n) & (c < TZ.n)) ? id : -1;
}

// Pass 1: tile counts; statistics that need no exact decision (reads, velocity moments, the
// fixed-point bound); particles whose footprint misses the grid (outside the box, rejected).
// The particle loop is warp-uniform (lanes past n take part without a particle) so the tile counters
// can be aggregated over runs of lanes: particles that arrive in spatial order share their tiles.
template <typename T>
__global__ void __launch_bounds__(256) k_count(Geom g, FieldSpec fs, TileGeo tg, PIn<T> in, long long n,
                                               unsigned *counts, DevStats *st, int split_edge) {
  float f_read = 0, f_out = 0, f_nsq = 0, f_v[4] = {0, 0, 0, 0}, f_abs[2] = {0, 0}, f_grid = 0;
  int fatal = 0, nonfin = 0;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i0 = blockIdx.x * (long long)blockDim.x + (threadIdx.x & ~31); i0 < n; i0 += stride) {
    const long long i = i0 + (threadIdx.x & 31);
    bool has = false;
    AxisTiles TX, TY, TZ;
    TX.n = TY.n = TZ.n = 0;
    if (i < n) {
      const Prep p = prep32(g, fs, in, i);
      if (!p.fin) {
        nonfin = 1;
      } else {
        f_read += 1.0f;
        if (fs.moments) {  // src/read_data.c:132-138, every particle read
          f_nsq += p.w;
          float wv = p.w * p.v;
          f_v[0] += wv; wv *= p.v;
          f_v[1] += wv; wv *= p.v;
          f_v[2] += wv; wv *= p.v;
          f_v[3] += wv;
        }
        float pa = p.w, pb = p.w;
        for (int e = 0; e < fs.ea; e++) pa *= p.v;
        for (int e = 0; e < fs.eb; e++) pb *= p.v;
        f_abs[0] += fabsf(pa);
        f_abs[1] += fabsf(pb);
        if (!footprint(g, tg, p.sx, p.sy, p.sz, TX, TY, TZ)) {
          f_out += 1.0f;  // clearly outside the box (src/read_data.c:81-88)
          if (g.los == 0) {
            fatal = 1;
            atomicMax(&st->fatal_inv, ~0ULL - (unsigned long long)i);
          }
        } else if (split_edge && is_edge(g, p.sx, p.sy, p.sz)) {
          // painted and counted by k_edge_fixup
        } else {
          has = true;
          // NGRID (src/read_data.c:92-126) and NOUT: exact for particles away from every edge
          if (split_edge && accept32(g, p.sx, p.sy, p.sz)) f_grid += p.w;
          if (split_edge && outside32(g, p.sx, p.sy, p.sz)) f_out += 1.0f;
        }
      }
    }
    const int na = __reduce_max_sync(FULL_MASK, has ? TX.n : 0), nb = __reduce_max_sync(FULL_MASK, has ? TY.n : 0),
              nc = __reduce_max_sync(FULL_MASK, has ? TZ.n : 0);
    // runtime loops over the warp's footprint tiles (warp-uniform bounds): one copy of the body
#pragma unroll 1
    for (int a = 0; a < na; a++)
#pragma unroll 1
      for (int b = 0; b < nb; b++)
#pragma unroll 1
        for (int c = 0; c < nc; c++) warp_run_add(counts, tile_key(tg, has, TX, TY, TZ, a, b, c), false);
  }
  // FP32 per-thread partials and warp sums, FP64 across warps
  const float vals[10] = {f_read, f_out, f_nsq, f_v[0], f_v[1], f_v[2], f_v[3], f_abs[0], f_abs[1], f_grid};
  double *const dst[10] = {&st->nread, &st->nout, &st->nsq, &st->vr[0], &st->vr[1], &st->vr[2], &st->vr[3],
                           &st->absw[0], &st->absw[1], &st->ngrid};
  block_add_f<10>(vals, dst);
  if (fatal) atomicOr(&st->fatal, 1);
  if (nonfin) atomicOr(&st->nonfinite, 1);
}

// Pass 2: exclusive scan of the tile counts (one CTA), cursor copy, record total, fixed-point scales.
__global__ void __launch_bounds__(1024) k_scan(const unsigned *counts, int ntiles, unsigned *offsets, unsigned *cursor,
                                               DevStats *st, unsigned long long capacity, double *fixed_scale) {
  __shared__ unsigned long long part[1024];
  const int tid = threadIdx.x, nt = blockDim.x;
  const int per = (ntiles + nt - 1) / nt;
  const int b = tid * per, e = min(ntiles, b + per);
  unsigned long long s = 0;
  for (int i = b; i < e; i++) s += counts[i];
  part[tid] = s;
  __syncthreads();
  for (int o = 1; o < nt; o <<= 1) {  // Hillis-Steele inclusive scan of the per-thread sums
    unsigned long long a = tid >= o ? part[tid - o] : 0;
    __syncthreads();
    part[tid] += a;
    __syncthreads();
  }
  unsigned long long run = part[tid] - s;
  for (int i = b; i < e; i++) {
    offsets[i] = (unsigned)run;
    cursor[i] = (unsigned)run;
    run += counts[i];
  }
  if (tid == nt - 1) {
    offsets[ntiles] = (unsigned)part[nt - 1];
    st->nrecords = (unsigned)part[nt - 1];
    if (part[nt - 1] > capacity) st->overflow = 1;
    // fixed-point scale per field: 2^S with sum|contrib| * 2^S < 2^62
    for (int f = 0; f < 2; f++) {
      double bound = st->absw[f] * 1.0001 + 1.0;
      int S = 62 - (int)ceil(log2(bound));
      if (S > 60) S = 60;
      fixed_scale[f] = ldexp(1.0, S);
    }
  }
}

#define SPECIAL_MARK (-3.0e38f)

// Pass 3: scatter particles into their tiles' lists. A record holds the normal-stencil scales and
// the velocity, or, for a particle taking the exact rules, a mark and the particle index. Same
// warp-uniform loop and run aggregation of the tile cursors as k_count.
template <typename T>
__global__ void __launch_bounds__(256) k_scatter(Geom g, FieldSpec fs, TileGeo tg, PIn<T> in, long long n,
                                                 unsigned *cursor, float4 *recs, float *recw,
                                                 unsigned long long capacity, unsigned *edge_list,
                                                 unsigned *edge_count) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i0 = blockIdx.x * (long long)blockDim.x + (threadIdx.x & ~31); i0 < n; i0 += stride) {
    const long long i = i0 + (threadIdx.x & 31);
    bool has = false;
    AxisTiles TX, TY, TZ;
    TX.n = TY.n = TZ.n = 0;
    float4 rec = make_float4(0.f, 0.f, 0.f, 0.f);
    float w = 1.0f;
    if (i < n) {
      const Prep p = prep32(g, fs, in, i);
      if (p.fin && footprint(g, tg, p.sx, p.sy, p.sz, TX, TY, TZ)) {
        const bool edge = is_edge(g, p.sx, p.sy, p.sz);
        if (edge && edge_list) {  // painted by k_edge_fixup after the tiles
          edge_list[atomicAdd(edge_count, 1u)] = (unsigned)i;
        } else {
          has = true;
          w = p.w;
          rec = edge ? make_float4(SPECIAL_MARK, __uint_as_float((unsigned)i), 0.0f, 0.0f)
                     : make_float4(p.sx, p.sy, p.sz, p.v);
        }
      }
    }
    const int na = __reduce_max_sync(FULL_MASK, has ? TX.n : 0), nb = __reduce_max_sync(FULL_MASK, has ? TY.n : 0),
              nc = __reduce_max_sync(FULL_MASK, has ? TZ.n : 0);
    // runtime loops over the warp's footprint tiles (warp-uniform bounds): one copy of the body
#pragma unroll 1
    for (int a = 0; a < na; a++)
#pragma unroll 1
      for (int b = 0; b < nb; b++)
#pragma unroll 1
        for (int c = 0; c < nc; c++) {
          const int key = tile_key(tg, has, TX, TY, TZ, a, b, c);
          const unsigned slot = warp_run_add(cursor, key, true);
          if (key >= 0 && slot < capacity) {
            recs[slot] = rec;
            if (recw) recw[slot] = w;
          }
        }
  }
}

// The tiles of one particle as a first tile and per-axis extents: tile (a, b, c), a < nx, b < ny, c < nz, is
// id + a SX + b SY + c SZ less a whole axis of tiles where a (b, c) has passed the axis's wrap (kx, ky, kz:
// the first wrapped step). footprint()'s lists are consecutive tiles modulo the axis, so this holds them all.
struct Foot {
  unsigned id, ext;  // ext: nx, ny, nz, kx, ky, kz in 2 bits each
};

__device__ __forceinline__ Foot pack_foot(const TileGeo &tg, const AxisTiles &TX, const AxisTiles &TY,
                                          const AxisTiles &TZ) {
  Foot f;
  f.id = (unsigned)tile_id(tg, TX.t0, TY.t0, TZ.t0);
  const int kx = min(tg.nbx - TX.t0, 3), ky = min(tg.nby - TY.t0, 3), kz = min(tg.nbz - TZ.t0, 3);
  f.ext = (unsigned)(TX.n | TY.n << 2 | TZ.n << 4 | kx << 6 | ky << 8 | kz << 10);
  return f;
}

// Tile k < nx ny nz of a footprint (z fastest).
__device__ __forceinline__ int foot_tile(const TileGeo &tg, const Foot &f, int k) {
  const int nz = (f.ext >> 4) & 3, ny = (f.ext >> 2) & 3;
  const int q = nz == 1 ? k : (nz == 2 ? k >> 1 : (k * 86) >> 8);  // k / nz for k < 27
  const int c = k - q * nz;
  const int a = ny == 1 ? q : (ny == 2 ? q >> 1 : (q * 86) >> 8);
  const int b = q - a * ny;
  int id = (int)f.id + (a * tg.nby + b) * tg.nbz + c;
  if (a >= (int)((f.ext >> 6) & 3)) id -= tg.ntiles;
  if (b >= (int)((f.ext >> 8) & 3)) id -= tg.nby * tg.nbz;
  if (c >= (int)((f.ext >> 10) & 3)) id -= tg.nbz;
  return id;
}

// A particle whose stencils lie inside the grid by whole cells along every axis: no edge of the reference's
// rules within reach, accepted, inside the box, and its footprint neither wraps nor is clipped. (NN has an
// edge at every cell, so it never qualifies.) s and s + 1/2 in [1 + m, n - 2 - m], m the margin.
__device__ __forceinline__ bool interior32(const Geom &g, float sx, float sy, float sz) {
  const float lo = 1.0f + 2.0f * g.margin, off = 2.5f + 2.0f * g.margin;
  return (g.order > 1) & (sx >= lo) & (sx <= (float)g.nx - off) & (sy >= lo) & (sy <= (float)g.ny - off) & (sz >= lo) &
         (sz <= (float)g.nz - off);
}

// axis_footprint of an interior particle: first tile and tile count (at most 3: six cells, tiles of four or more).
__device__ __forceinline__ void axis_interior(float s, float m, int order, int shift, int &t0, int &n) {
  const int lo = __float2int_rd(__fsub_rn(s, m)) - (order == 3 ? 1 : 0), hi = __float2int_rd(__fadd_rn(s, m)) + 2;
  t0 = lo >> shift;
  n = (hi >> shift) - t0 + 1;
}

// Compensated FP32 sum (the rounding error of each addition is carried to the next one): a thread of the
// bucketing sums a hundred particles, and the mean velocity that the shot noise of a cross spectrum takes
// from these sums is a small difference of large ones.
struct CSum {
  float s, c;
  __device__ __forceinline__ CSum() : s(0.0f), c(0.0f) {}
  __device__ __forceinline__ void add(float v) {
    const float y = __fsub_rn(v, c), u = __fadd_rn(s, y);
    c = __fsub_rn(__fsub_rn(u, s), y);
    s = u;
  }
};

// Block sum of NV compensated sums, each warp's in pairs of floats (the pair's high part s and what its
// additions rounded away), FP64 across warps, added to global dst.
template <int NV>
__device__ void block_add_cs(const CSum (&v)[NV], double *const (&dst)[NV]) {
  __shared__ double redc[32][NV];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int k = 0; k < NV; k++) {
    float hi = v[k].s, lo = -v[k].c;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float h2 = __shfl_xor_sync(FULL_MASK, hi, o), l2 = __shfl_xor_sync(FULL_MASK, lo, o);
      const float u = __fadd_rn(hi, h2), b = __fsub_rn(u, hi);
      lo = __fadd_rn(__fadd_rn(lo, l2), __fadd_rn(__fsub_rn(hi, __fsub_rn(u, b)), __fsub_rn(h2, b)));
      hi = u;
    }
    if (lane == 0) redc[wid][k] = (double)hi + (double)lo;
  }
  __syncthreads();
  if (wid == 0 && lane < NV) {
    double a = 0.0;
    for (int w = 0; w < nw; w++) a += redc[w][lane];
    if (a != 0.0) atomicAdd(dst[lane], a);
  }
  __syncthreads();
}

// One particle's sums (src/read_data.c:132-138 and the fixed-point bound), over a thread's particles.
struct BucketSums {
  float read, out, abs_a, abs_b;
  CSum nsq, v[4], grid;
  int fatal, nonfin;
  __device__ __forceinline__ BucketSums() : read(0.0f), out(0.0f), abs_a(0.0f), abs_b(0.0f), fatal(0), nonfin(0) {}
  __device__ __forceinline__ void add_read(const FieldSpec &fs, const Prep &q) {
    read += 1.0f;
    if (fs.moments) {  // every particle read
      nsq.add(q.w);
      float wv = q.w * q.v;
      v[0].add(wv); wv *= q.v;
      v[1].add(wv); wv *= q.v;
      v[2].add(wv); wv *= q.v;
      v[3].add(wv);
    }
    float pa = q.w, pb = q.w;
    for (int e = 0; e < fs.ea; e++) pa *= q.v;
    for (int e = 0; e < fs.eb; e++) pb *= q.v;
    abs_a += fabsf(pa);
    abs_b += fabsf(pb);
  }
  __device__ __forceinline__ void finish(DevStats *st, int ovf_full) {
    const float vals[4] = {read, out, abs_a, abs_b};
    double *const dst[4] = {&st->nread, &st->nout, &st->absw[0], &st->absw[1]};
    block_add_f<4>(vals, dst);
    const CSum cs[6] = {grid, nsq, v[0], v[1], v[2], v[3]};
    double *const dc[6] = {&st->ngrid, &st->nsq, &st->vr[0], &st->vr[1], &st->vr[2], &st->vr[3]};
    block_add_cs<6>(cs, dc);
    if (fatal) atomicOr(&st->fatal, 1);
    if (nonfin) atomicOr(&st->nonfinite, 1);
    if (ovf_full) atomicOr(&st->overflow, 1);
  }
};

constexpr unsigned FOOT_NONE = 0xffffffffu;  // a particle with no tiles: one empty entry

// Footprint of an interior particle.
__device__ __forceinline__ Foot interior_foot(const Geom &g, const TileGeo &tg, float sx, float sy, float sz) {
  int tx, ty, tz, nx, ny, nz;
  axis_interior(sx, g.margin, g.order, tg.lx, tx, nx);
  axis_interior(sy, g.margin, g.order, tg.ly, ty, ny);
  axis_interior(sz, g.margin, g.order, tg.lz, tz, nz);
  Foot f;
  f.id = (unsigned)tile_id(tg, tx, ty, tz);
  f.ext = (unsigned)(nx | ny << 2 | nz << 4 | 0xfc0);
  return f;
}

// Footprint of any other particle by the full rules (idx its catalogue index): none when it is outside or
// goes to the exact rules.
__device__ __forceinline__ Foot near_foot(const Geom &g, const TileGeo &tg, float sx, float sy, float sz, float w,
                                          long long idx, unsigned *edge_list, unsigned *edge_count, DevStats *st,
                                          BucketSums &sum) {
  Foot f;
  f.id = FOOT_NONE;
  f.ext = 0x15;
  AxisTiles TX, TY, TZ;
  TX.n = TY.n = TZ.n = 0;
  if (!footprint(g, tg, sx, sy, sz, TX, TY, TZ)) {
    sum.out += 1.0f;  // clearly outside the box (src/read_data.c:81-88)
    if (g.los == 0) {
      sum.fatal = 1;
      atomicMax(&st->fatal_inv, ~0ULL - (unsigned long long)idx);
    }
  } else if (is_edge(g, sx, sy, sz)) {
    edge_list[atomicAdd(edge_count, 1u)] = (unsigned)idx;  // painted and counted by k_edge_fixup
  } else {
    f = pack_foot(tg, TX, TY, TZ);
    if (accept32(g, sx, sy, sz)) sum.grid.add(w);        // NGRID (src/read_data.c:92-126)
    if (outside32(g, sx, sy, sz)) sum.out += 1.0f;
  }
  return f;
}

// A warp's particles spread over its lanes: with cnt (at least 1) tiles of this lane's particle, entry e of the
// warp belongs to the particle whose first entry is the last one at or before e. next() gives the owner of
// entry t + lane for t = 0, 32, ...
struct WarpSpread {
  int off, total, before;
  __device__ __forceinline__ WarpSpread(int cnt, int lane) {
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(FULL_MASK, incl, o);
      if (lane >= o) incl += u;
    }
    off = incl - cnt;
    total = __shfl_sync(FULL_MASK, incl, 31);
    before = 0;
  }
  __device__ __forceinline__ int next(int t, int lane) {
    const unsigned firsts = __reduce_or_sync(FULL_MASK, (unsigned)(off - t) < 32u ? 1u << (off - t) : 0u);
    const int own = before + __popc(firsts & (0xffffffffu >> (31 - lane))) - 1;
    before += __popc(firsts);
    return own;
  }
};

// Where records go: their tile's bucket, or when it is full the overflow list.
struct BucketOut {
  float4 *recs;
  float *recw;
  unsigned cap;
  float4 *ovf_recs;
  float *ovf_w;
  unsigned *ovf_tile, *ovf_count;
  unsigned long long ovf_cap;
  __device__ __forceinline__ int put(int key, unsigned slot, const float4 &rec, float w) const {
    if (slot < cap) {
      const unsigned long long r = (unsigned long long)key * cap + slot;
      recs[r] = rec;
      if (recw) recw[r] = w;
      return 0;
    }
    const unsigned o = atomicAdd(ovf_count, 1u);
    if (o >= ovf_cap) return 1;
    ovf_recs[o] = rec;
    if (ovf_w) ovf_w[o] = w;
    ovf_tile[o] = (unsigned)key;
    return 0;
  }
};

// One-pass bucketing, passes 1-3 in one: the statistics of k_count and the records of k_scatter, each written
// into its tile's fixed-capacity bucket; a record that finds its bucket full goes to the overflow list with its
// tile. A particle has 1.1 to 2.9 entries (tiles); a warp spreads its particles' entries over its lanes, so that
// they cost no idle lanes, and lanes with equal tiles share one reservation of bucket slots. What bounds both
// variants below is instruction issue. They differ in how slots are reserved.
//
// k_bucket_cta, for up to BK_DIRECT_TILES tiles of 64 particles and more: a CTA ranks the entries of a chunk of BK_THREADS * ppt
// particles by shared counters of every tile, reserves each touched tile's slots with one global atomic, then
// writes the records. With few tiles and particles in random order the global atomics of the warps would meet
// on the same addresses: 2,097,152 such particles took 337 us into the 256 tiles of a 128^3 grid when each run
// of lanes made its own.
constexpr int BK_THREADS = 512;
constexpr int BK_PPT = 4;              // particles per thread and chunk, at most
constexpr int BK_P = BK_THREADS * BK_PPT;
constexpr int BK_E = 4096;             // entries held; any beyond go out one by one

static size_t bucket_smem(int ntiles) {
  return sizeof(float4) * BK_P + 4 * BK_P + 4 * BK_E + 2 * BK_E + 2 * BK_P + 4 * (size_t)ntiles;
}

template <typename T>
__global__ void __launch_bounds__(BK_THREADS, 2)
    k_bucket_cta(Geom g, FieldSpec fs, TileGeo tg, PIn<T> in, long long n, long long ibase, int ppt, unsigned *counts,
                 BucketOut out, unsigned *edge_list, unsigned *edge_count, DevStats *st) {
  extern __shared__ __align__(16) unsigned char smb[];
  float4 *srec = (float4 *)smb;
  float *sw = (float *)(srec + BK_P);
  unsigned *shr = (unsigned *)(sw + BK_P);            // entry: tile | rank << 16
  unsigned short *sown = (unsigned short *)(shr + BK_E);
  unsigned short *slist = sown + BK_E;                // the chunk's particles near the grid's faces
  unsigned *sc = (unsigned *)(slist + BK_P);          // counters, then the reserved first slots
  __shared__ unsigned s_ent, s_near;
  const int lane = threadIdx.x & 31;
  for (int h = threadIdx.x; h < tg.ntiles; h += BK_THREADS) sc[h] = 0;
  if (threadIdx.x == 0) s_ent = s_near = 0;
  __syncthreads();
  BucketSums sum;
  int ovf_full = 0;
  auto add_entries = [&](const Foot &ft, int li) {
    WarpSpread ws((int)((ft.ext & 3) * ((ft.ext >> 2) & 3) * ((ft.ext >> 4) & 3)), lane);
    unsigned base = 0;
    if (lane == 0) base = atomicAdd(&s_ent, (unsigned)ws.total);
    base = __shfl_sync(FULL_MASK, base, 0);
    for (int t = 0; t < ws.total; t += 32) {
      const int own = ws.next(t, lane), e = t + lane;
      Foot f;
      f.id = __shfl_sync(FULL_MASK, ft.id, own);
      f.ext = __shfl_sync(FULL_MASK, ft.ext, own);
      const int k = e - __shfl_sync(FULL_MASK, ws.off, own), oli = __shfl_sync(FULL_MASK, li, own);
      const unsigned pos = base + (unsigned)e;
      const bool held = e < ws.total && pos < (unsigned)BK_E, real = e < ws.total && f.id != FOOT_NONE;
      const int key = real ? foot_tile(tg, f, k) : -1;
      // lanes of one tile take consecutive ranks from one counter access
      const unsigned peers = __match_any_sync(FULL_MASK, held ? key : -1);
      const int head = __ffs(peers) - 1;
      unsigned rank = 0;
      if (held && real && head == lane) rank = atomicAdd(&sc[key], (unsigned)__popc(peers));
      rank = __shfl_sync(FULL_MASK, rank, head) + (unsigned)__popc(peers & ((1u << lane) - 1u));
      if (held) {
        shr[pos] = real ? (unsigned)key | rank << 16 : FOOT_NONE;
        sown[pos] = (unsigned short)oli;
      } else if (real) {  // more entries than the list holds (tiles that are small for the footprint)
        ovf_full |= out.put(key, atomicAdd(counts + key, 1u), srec[oli], sw[oli]);
      }
    }
  };
  const int chunk = BK_THREADS * ppt;
  for (long long c0 = (long long)blockIdx.x * chunk; c0 < n; c0 += (long long)gridDim.x * chunk) {
#pragma unroll 1
    for (int p = 0; p < ppt; p++) {
      const int li = p * BK_THREADS + threadIdx.x;
      const long long i = c0 + li;
      if (i - lane >= n) break;  // the whole warp is past the end
      Foot ft;
      ft.id = FOOT_NONE;
      ft.ext = 0x15;
      if (i < n) {
        const Prep q = prep32(g, fs, in, i);
        if (!q.fin) {
          sum.nonfin = 1;
        } else {
          sum.add_read(fs, q);
          srec[li] = make_float4(q.sx, q.sy, q.sz, q.v);
          sw[li] = q.w;
          if (interior32(g, q.sx, q.sy, q.sz)) {
            ft = interior_foot(g, tg, q.sx, q.sy, q.sz);
            sum.grid.add(q.w);  // NGRID (src/read_data.c:92-126)
          } else {
            slist[atomicAdd(&s_near, 1u)] = (unsigned short)li;
          }
        }
      }
      __syncwarp();  // srec and sw of the warp's particles are written
      if (g.order > 1) add_entries(ft, li);  // (NN: all of them below, and an entry of none for each would fill the list)
    }
    __syncthreads();
    // the few particles near a face of the grid (for NN: all), by the full rules, in dense warps
    const int nnear = (int)s_near;
    for (int q0 = threadIdx.x - lane; q0 < nnear; q0 += BK_THREADS) {
      const int q = q0 + lane, li = q < nnear ? slist[q] : 0;
      Foot ft;
      ft.id = FOOT_NONE;
      ft.ext = 0x15;
      if (q < nnear) {
        const float4 r = srec[li];
        ft = near_foot(g, tg, r.x, r.y, r.z, sw[li], ibase + c0 + li, edge_list, edge_count, st, sum);
      }
      add_entries(ft, li);
    }
    __syncthreads();
    const int ne = (int)min(s_ent, (unsigned)BK_E);
    for (int h = threadIdx.x; h < tg.ntiles; h += BK_THREADS) {
      const unsigned c = sc[h];
      if (c) sc[h] = atomicAdd(counts + h, c);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < ne; e += BK_THREADS) {
      const unsigned hr = shr[e];
      if (hr == FOOT_NONE) continue;
      const int own = sown[e], key = (int)(hr & 0xffffu);
      ovf_full |= out.put(key, sc[key] + (hr >> 16), srec[own], sw[own]);
    }
    __syncthreads();
    for (int h = threadIdx.x; h < tg.ntiles; h += BK_THREADS) sc[h] = 0;
    if (threadIdx.x == 0) s_ent = s_near = 0;
    __syncthreads();
  }
  sum.finish(st, ovf_full);
}

// k_bucket_warp, for more tiles or fewer particles: the lanes of a warp with equal tiles share one global atomic, two groups of 32
// entries at a time so that their atomics are in flight together, and the next particles' loads run behind
// them. (A CTA-wide ranking through a hash table of the touched tiles was slower: 550 against 500 us for 16.7M
// particles in lattice order at 512^3.)
template <typename T>
__global__ void __launch_bounds__(256, 4)
    k_bucket_warp(Geom g, FieldSpec fs, TileGeo tg, PIn<T> in, long long n, long long ibase, unsigned *counts,
                  BucketOut out, unsigned *edge_list, unsigned *edge_count, DevStats *st) {
  __shared__ float4 s_rec[256];
  __shared__ float s_w[256];
  const int lane = threadIdx.x & 31;
  float4 *wrec = s_rec + (threadIdx.x - lane);
  float *ww = s_w + (threadIdx.x - lane);
  BucketSums sum;
  int ovf_full = 0;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i0 = blockIdx.x * (long long)blockDim.x + threadIdx.x - lane; i0 < n; i0 += stride) {
    const long long i = i0 + lane;
    Foot ft;
    ft.id = FOOT_NONE;
    ft.ext = 0x15;
    if (i < n) {
      const Prep q = prep32(g, fs, in, i);
      if (!q.fin) {
        sum.nonfin = 1;
      } else {
        sum.add_read(fs, q);
        wrec[lane] = make_float4(q.sx, q.sy, q.sz, q.v);
        ww[lane] = q.w;
        if (interior32(g, q.sx, q.sy, q.sz)) {
          ft = interior_foot(g, tg, q.sx, q.sy, q.sz);
          sum.grid.add(q.w);  // NGRID (src/read_data.c:92-126)
        } else {
          ft = near_foot(g, tg, q.sx, q.sy, q.sz, q.w, ibase + i, edge_list, edge_count, st, sum);
        }
      }
    }
    __syncwarp();
    WarpSpread ws((int)((ft.ext & 3) * ((ft.ext >> 2) & 3) * ((ft.ext >> 4) & 3)), lane);
    for (int t = 0; t < ws.total; t += 64) {
      int key[2], own[2], head[2];
      unsigned base[2], rank[2];
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const int e = t + 32 * u + lane;
        own[u] = ws.next(t + 32 * u, lane) & 31;
        Foot f;
        f.id = __shfl_sync(FULL_MASK, ft.id, own[u]);
        f.ext = __shfl_sync(FULL_MASK, ft.ext, own[u]);
        const int k = e - __shfl_sync(FULL_MASK, ws.off, own[u]);
        key[u] = e < ws.total && f.id != FOOT_NONE ? foot_tile(tg, f, k) : -1;
        const unsigned peers = __match_any_sync(FULL_MASK, key[u]);
        head[u] = __ffs(peers) - 1;
        rank[u] = (unsigned)__popc(peers & ((1u << lane) - 1u));
        base[u] = 0;
        if (head[u] == lane && key[u] >= 0) base[u] = atomicAdd(counts + key[u], (unsigned)__popc(peers));
      }
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const unsigned slot = __shfl_sync(FULL_MASK, base[u], head[u]) + rank[u];
        if (key[u] >= 0) ovf_full |= out.put(key[u], slot, wrec[own[u]], ww[own[u]]);
      }
    }
    __syncwarp();  // the next particles overwrite wrec
  }
  sum.finish(st, ovf_full);
}

template <typename T>
static void launch_bucket(cudaStream_t s, const Geom &g, const FieldSpec &fs, const TileGeo &tg, const PIn<T> &in,
                          long long n, long long ibase, const PaintBufs &b, DevStats *st) {
  const BucketOut out{b.recs,     in.w ? b.recw : nullptr, b.bucket_cap, b.ovf_recs, in.w ? b.ovf_w : nullptr,
                      b.ovf_tile, b.ovf_count,             b.ovf_cap};
  // (Below 64 particles a tile the CTA's passes over its counters cost more than the warps' atomics: 20,000 and 100,000
  // particles on 256^3 and 300x200x250, before the tiles: 36 -> 31 and 48 -> 41 us; above 250 in random order the CTAs win,
  // 1M on 128^3: 64 against 165 us.)
  if (tg.ntiles <= BK_DIRECT_TILES && n >= 64LL * tg.ntiles) {
    const size_t smem = bucket_smem(tg.ntiles);
    allow_smem(k_bucket_cta<T>, 8192);
    // one resident wave (two CTAs per SM); a small catalogue takes fewer particles per chunk, to fill it, but as many as leave
    // no second chunk to some of the CTAs. No more than the list has room for, though: the entries beyond it make a global
    // atomic each (small tiles, a particle near a face one entry more). 21 x 21 x 33, CIC, 535,000 particles by chunks of 4 a
    // thread 182 us a call, of 3 162; TSC, 2M: 692 by 4, 466 by 3. The line at 0.65 of another particle: 4 against 3 at 3.56
    // is 271 to 256 us, at 3.71 (48^3) 244 to 242 for 2M and 144 to 150 for 535,000.
    const long long wave = 152LL * 2 * BK_THREADS;
    const double entries = tile_dup_estimate(g, tg) +
                           (g.order > 1 ? 1.0 - (1.0 - 3.5 / g.nx) * (1.0 - 3.5 / g.ny) * (1.0 - 3.5 / g.nz) : 0.0);
    const int fits = std::max(1, (int)((double)BK_E / (BK_THREADS * entries) + 0.35));
    const int ppt = (int)std::min<long long>(std::min(BK_PPT, fits), std::max<long long>(1, (n + wave - 1) / wave));
    const long long chunks = (n + BK_THREADS * ppt - 1) / (BK_THREADS * ppt);
    const int nb = (int)(chunks < 1 ? 1 : (chunks > 152 * 2 ? 152 * 2 : chunks));
    k_bucket_cta<T><<<nb, BK_THREADS, smem, s>>>(g, fs, tg, in, n, ibase, ppt, b.counts, out, b.edge_list, b.edge_count,
                                                 st);
  } else {
    const long long nb = (n + 255) / 256;
    k_bucket_warp<T><<<(int)(nb < 1 ? 1 : (nb > 152 * 8 ? 152 * 8 : nb)), 256, 0, s>>>(
        g, fs, tg, in, n, ibase, b.counts, out, b.edge_list, b.edge_count, st);
  }
}

// Deterministic accumulation: round(value * 2^S) added as an integer (S from k_scan, per field).
__device__ __forceinline__ void acc_add64(unsigned long long *p, double v, double scale) {
  atomicAdd(p, (unsigned long long)__double2ll_rn(v * scale));
}

// One axis of a record's stencil: the taps' offsets in the shared tile
// (index within the tile times the axis pitch) and weights; a tap that the reference drops or that
// lies outside this tile gets weight 0.
__device__ __forceinline__ void stage_axis32(const AxisTapsF &t, int origin, int extent, int pitch, float *W,
                                             int *O) {
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const int l = t.idx[k] - origin;
    const bool ok = t.idx[k] >= 0 && l >= 0 && l < extent;
    W[k] = ok ? t.w[k] : 0.0f;
    O[k] = ok ? l * pitch : 0;
  }
}

// Same for exact taps in the reference's index space. x: halo slices fold onto 0.. (LOS == 0) or are
// dropped; z: the padding column (a CIC rounding edge) is dropped; y == NY (a CIC rounding edge) is
// the aliased write handled by the caller.
__device__ __forceinline__ void stage_axis64(const Geom &g, const AxisTaps &t, int axis, int origin, int extent,
                                             int pitch, float *W, int *O) {
#pragma unroll
  for (int k = 0; k < 3; k++) {
    int idx = t.idx[k];
    bool ok = k < t.n && t.on[k];
    const int n = axis == 0 ? g.nx : (axis == 1 ? g.ny : g.nz);
    if (axis == 0 && idx >= n) {
      if (g.los == 0 && idx < n + g.order) idx -= n;
      else ok = false;
    }
    if (idx < 0 || idx >= n) ok = false;
    const int l = idx - origin;
    ok = ok && l >= 0 && l < extent;
    W[k] = ok ? (float)t.w[k] : 0.0f;
    O[k] = ok ? l * pitch : 0;
  }
}

// Compile-time-order FP32 taps of one axis (kind 0: x, 1: y or z).
// Power-of-two scale 2^S for a tile's int32 fixed-point cells. A record's taps add at most |w v^e|
// to one slot, so no cell of the slot exceeds the tile's sum of |w v^e| over its records; that sum
// (FP32, raised by 0.1 % for its own rounding) times 2^S < 2^31 keeps every partial sum inside int32: the 0.1 % are two
// million units, the half-unit roundings of a tile's deposits (one per record and cell, at most TILE_DENSE_RECORDS) 8192.
__device__ __forceinline__ int tile_scale_exp(float sum_abs) {
  const float bound = sum_abs * 1.001f;
  if (!(bound > 0.0f) || !isfinite(bound)) return 0;
  const int e = ilogbf(bound);  // bound < 2^(e+1)
  const int S = 30 - e;
  return S > 100 ? 100 : (S < -100 ? -100 : S);
}

// Largest scale exponent that keeps every single deposit of a tile below 2^22 in magnitude
// (|w v^e| 2^S < 2^22, tap weights <= 1), where rint_small rounds exactly.
__device__ __forceinline__ int tile_scale_max(float max_abs) {
  const float mb = max_abs * 1.001f;
  return (mb > 0.0f && isfinite(mb)) ? 21 - ilogbf(mb) : 100;
}

// Round-to-nearest-even of a * b as an int32, for |a * b| < 2^22: the fused multiply-add rounds the
// exact product plus 1.5 * 2^23 to an integer, whose FP32 bit pattern is 0x4B400000 + that integer.
// (Two FP32/integer-pipe instructions instead of a conversion.)
__device__ __forceinline__ int rint_small(float a, float b) {
  return __float_as_int(__fmaf_rn(a, b, 12582912.0f)) - 0x4B400000;
}

// The int32 quantum of a tile is about 2^-30 of the tile's total |w v^e|, and a cell sums up to one
// rounded deposit per record: the cells' relative error grows with the record count. A tile with
// more records than this (a dense clump or a coarse grid; ordinary catalogues put about a thousand records
// in a tile) is accumulated in two int32 limbs per cell instead (tile_paint_dense). For a tile smaller than
// the default one the limit goes down with its cells, so that it stands for the same density.
#define TILE_DENSE_RECORDS 16384u

// Scaled values w v^e of a record's two fields.
__device__ __forceinline__ void record_values(const FieldSpec &fs, const float4 &rec, float w, float &va, float &vb) {
  va = w;
  vb = w;
  for (int e = 0; e < fs.ea; e++) va *= rec.w;
  for (int e = 0; e < fs.eb; e++) vb *= rec.w;
}

// One axis of an inner tile's record (axis32k and stage_axis32 where no tap reaches a face of the grid): weights, 0 for
// a tap outside the tile, and offsets (ZERO: 0 for a tap outside; the others' are not used then).
template <int K, bool ZERO>
__device__ __forceinline__ void inner_axis32(float s, int origin, int extent, int pitch, float *W, int *O) {
  const int i = (int)(K == 3 ? s + 0.5f : s), l = i - origin;
  const float d = s - (float)i;
  const int o = l * pitch;
  if (K == 3) {
    W[0] = 0.75f - d * d;
    W[1] = 0.5f * (0.5f - d) * (0.5f - d);
    W[2] = 0.5f * (0.5f + d) * (0.5f + d);
    O[1] = o - pitch;
  } else {
    W[0] = K == 2 ? 1.0f - d : 1.0f;
    W[1] = d;
    O[1] = o + pitch;
  }
  O[0] = o;
  O[2] = o + pitch;
#pragma unroll
  for (int k = 0; k < K; k++) {
    const int t = k == 0 ? l : (K == 3 && k == 1 ? l - 1 : l + 1);
    if ((unsigned)t >= (unsigned)extent) {
      W[k] = 0.0f;
      if (ZERO) O[k] = 0;
    }
  }
}

// The deposits of the records [rb, re) into the int32 shared tile (lane = record; both stencils).
// FASTR: rounded by rint_small (every deposit below 2^22); otherwise by conversion. INNER: the tile lies 4 cells and more
// inside the grid, where no tap of its records wraps, drops or is refused (16.7M particles on 512^3, four slots: the rules of
// the faces were 100M of 1193M warp instructions for TSC, 1.41 -> 1.35 ms, 75M of 660M for CIC).
template <int K, int NF, bool IL, bool FASTR, bool INNER>
__device__ __forceinline__ void tile_rec_deposit(const Geom &g, const FieldSpec &fs, const TileGeo &tg,
                                                 const float4 *recs, const float *recw, unsigned long long rb,
                                                 unsigned long long re, float scA, float scB, int x0, int y0,
                                                 int z0, int ex, int ey, int ez, int *smi) {
  constexpr int NS = IL ? 2 : 1;
  const int slotw = tg.slot;
  for (unsigned long long r = rb + threadIdx.x; r < re; r += blockDim.x) {
    const float4 rec = recs[r];
    float va, vb;
    record_values(fs, rec, recw ? recw[r] : 1.0f, va, vb);
    va *= scA;
    vb *= scB;
#pragma unroll
    for (int s = 0; s < NS; s++) {
      const float sx = s ? __fadd_rn(rec.x, 0.5f) : rec.x, sy = s ? __fadd_rn(rec.y, 0.5f) : rec.y,
                  sz = s ? __fadd_rn(rec.z, 0.5f) : rec.z;
      float wx[3], wy[3], wz[3];
      int ox[3], oy[3], oz[3];
      if (INNER) {
        inner_axis32<K, false>(sx, x0, ex, tg.px, wx, ox);
        inner_axis32<K, false>(sy, y0, ey, tg.py, wy, oy);
        inner_axis32<K, true>(sz, z0, ez, 1, wz, oz);
      } else {
        if (!accept32(g, sx, sy, sz)) continue;
        AxisTapsF ax, ay, az;
        axis32k<K>(sx, 0, g.nx, g.los, ax);
        axis32k<K>(sy, 1, g.ny, g.los, ay);
        axis32k<K>(sz, 1, g.nz, g.los, az);
        stage_axis32(ax, x0, ex, tg.px, wx, ox);
        stage_axis32(ay, y0, ey, tg.py, wy, oy);
        stage_axis32(az, z0, ez, 1, wz, oz);
      }
      int *sA = smi + (s * NF) * slotw;
#pragma unroll
      for (int a = 0; a < K; a++)
#pragma unroll
        for (int b2 = 0; b2 < K; b2++) {
          const float wxy = wx[a] * wy[b2];
          const float pa = va * wxy, pb = vb * wxy;
          const int oxy = ox[a] + oy[b2];
          // one test per (x, y) tap pair: an x or y tap outside the tile has weight 0. A z tap outside
          // it (the z edge of a tile is 32 cells: rare) has weight 0 and offset 0 and adds 0 there.
          if (wxy != 0.0f) {
#pragma unroll
            for (int c = 0; c < K; c++) {
              atomicAdd(sA + oxy + oz[c], FASTR ? rint_small(pa, wz[c]) : __float2int_rn(pa * wz[c]));
              if (NF == 2)
                atomicAdd(sA + slotw + oxy + oz[c], FASTR ? rint_small(pb, wz[c]) : __float2int_rn(pb * wz[c]));
            }
          }
        }
    }
  }
}

// A deposit p (an FP32 value already in the tile's fixed point) split as p = h 2^k + l with
// h = floor(p 2^-k) and l = p - h 2^k in [0, 2^k] (k <= 22, |h| < 2^22), both made integers by the FMA rounding
// of rint_small and added with two native int32 shared atomics; the cell's value is hi 2^k + lo. The FMA
// that forms l is exact except for a negative p of magnitude below 2^k, where the deposit may come out
// one unit of the fixed point away from round(p): still a fixed function of p, whatever the order.
__device__ __forceinline__ void limb_add(int *lo, int *hi, float p, float two_mk, float two_k) {
  const float h = floorf(p * two_mk);
  const float l = __fmaf_rn(-h, two_k, p);
  atomicAdd(lo, rint_small(l, 1.0f));
  atomicAdd(hi, rint_small(h, 1.0f));
}

__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The shared::cluster address of this CTA's shared address in CTA `rank` of the cluster, and loads from it.
__device__ __forceinline__ unsigned map_cluster(unsigned smem, int rank) {
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem), "r"(rank));
  return r;
}
__device__ __forceinline__ int ld_cluster_s32(unsigned a) {
  int v;
  asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float ld_cluster_f32(unsigned a) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}

// Place of a tile and of a CTA in the tile's cluster (of S CTAs, this one's rank).
struct TileAt {
  int x0, y0, z0, ex, ey, ez, S, rank;
};

// A tile's write-out: pairs of cells along z as float2 (8-byte aligned global rows). A thread keeps one (y, z)
// pair of the tile's x-planes and walks x: the pair's address in shared memory and in the grid only advance by
// px and the grid slice. cell(word) gives the pair at a shared word of a plane's slot; store(x, a0, a1) gets it.
// In a cluster each CTA writes its share of the pairs and planes.
template <bool CL, typename F>
__device__ __forceinline__ void tile_walk(const Geom &g, const TileGeo &tg, const TileAt &at, F &&store) {
  const int ppl = (tg.ty * tg.tz) >> 1;  // pairs per x-plane
  const int nthr = (int)blockDim.x * at.S;
  // a cluster has more threads than a plane has pairs: they share the x-planes
  const int xs = CL ? max(1, min(at.ex, nthr / ppl)) : 1;
  for (int q = at.rank * (int)blockDim.x + threadIdx.x; q < ppl * xs; q += nthr) {
    const int w = CL ? q % ppl : q, lx0 = CL ? q / ppl : 0;
    const int c = w << 1;
    const int rz = c & (tg.tz - 1), ly = c >> tg.lz;
    if (ly >= at.ey || rz >= at.ez) continue;
    const bool two = rz + 1 < at.ez;
    const int cb = ly * tg.py + rz;
    const long long gb = (long long)at.x0 * g.slice + (long long)(at.y0 + ly) * g.row + at.z0 + rz;
    for (int lx = lx0; lx < at.ex; lx += xs) store(cb + lx * tg.px, gb + (long long)lx * g.slice, two);
  }
}

__device__ __forceinline__ float store_pair(float *dst, float a0, float a1, bool two) {
  if (two) {
    *reinterpret_cast<float2 *>(dst) = make_float2(a0, a1);
    return a0 + a1;
  }
  dst[0] = a0;
  return a0;
}

// A dense tile, one slot at a time: the records [r0, r1) of this CTA into cells of two int32 limbs, hi 2^K + lo, lo
// unsigned: two native atomics a deposit. (int64 cells need 64-bit shared atomics, compare-and-swap loops: 5.4M weighted
// particles, TSC, interlaced, into 32^3: 53 ms, by limbs 1.25 ms; 8M, CIC, interlaced, into 128^3: 0.57 and 0.43 ms. The
// grids' errors against 64 bits are the same.) The scale is the finest that holds
//  * every cell: the sum of |w v^e| 2^S below 2^49, so that a cell's high limb stays inside int32, and
//  * every deposit: the largest |w v^e| 2^S below 2^41, so that its high limb stays inside rint_small's 2^22 (a share of a
//    few hundred records lets one of them reach far into the sum's range).
// Every 7936 records the low limbs' carries go to the high ones: 2^K plus 7936 deposits of up to 2^K fit 32 bits.
// Where one record holds more than a quarter of the sum or 256 times the mean, the cells are int64 at 2^60 of the sum
// instead, as slow as before. Elsewhere the quantum is below 2^-32 of the mean record (or 2^-48 of the sum), and the rounding
// of the deposits stays below the rounding of the FP32 cell that they end in.
constexpr int DENSE_K = 19;
constexpr unsigned DENSE_ROUND = 7936;  // a multiple of the CTA's threads

// Scale exponent of one field's cells: sum and max of |w v^e| over cnt records.
__device__ __forceinline__ int dense_scale(float sum, float max, float cnt, bool &wide) {
  const float sb = sum * 1.001f, mb = max * 1.001f;
  wide = false;
  if (!(sb > 0.0f) || !isfinite(sb)) return 0;
  wide = max > 0.25f * sum || max * (cnt * 0x1p-8f) > sum;
  const int es = ilogbf(sb), em = ilogbf(mb);  // sum < 2^(es + 1), max < 2^(em + 1)
  const int S = wide ? 60 - es : min(48 - es, 40 - em);
  return S > 100 ? 100 : (S < -100 ? -100 : S);
}

// Deposits of the records [r0, r1) into one slot's cells: WIDE: int64 cells at smi; otherwise the limbs lo, hi.
template <int K, bool WIDE>
__device__ __forceinline__ void dense_deposit(const Geom &g, const FieldSpec &fs, const TileGeo &tg, const float4 *recs,
                                              const float *recw, unsigned long long r0, unsigned long long r1, int sten,
                                              int fld, float sc, const TileAt &at, int *smi) {
  int *lo = smi, *hi = smi + tg.slot;
  const float two_k = (float)(1 << DENSE_K), two_mk = 1.0f / two_k;
  for (unsigned long long r = r0 + threadIdx.x; r < r1; r += blockDim.x) {
    const float4 rec = recs[r];
    float va, vb;
    record_values(fs, rec, recw ? recw[r] : 1.0f, va, vb);
    const float v = (fld ? vb : va) * sc;
    const float sx = sten ? __fadd_rn(rec.x, 0.5f) : rec.x, sy = sten ? __fadd_rn(rec.y, 0.5f) : rec.y,
                sz = sten ? __fadd_rn(rec.z, 0.5f) : rec.z;
    if (!accept32(g, sx, sy, sz)) continue;
    AxisTapsF ax, ay, az;
    axis32k<K>(sx, 0, g.nx, g.los, ax);
    axis32k<K>(sy, 1, g.ny, g.los, ay);
    axis32k<K>(sz, 1, g.nz, g.los, az);
    float wx[3], wy[3], wz[3];
    int ox[3], oy[3], oz[3];
    stage_axis32(ax, at.x0, at.ex, tg.px, wx, ox);
    stage_axis32(ay, at.y0, at.ey, tg.py, wy, oy);
    stage_axis32(az, at.z0, at.ez, 1, wz, oz);
#pragma unroll
    for (int a = 0; a < K; a++)
#pragma unroll
      for (int b2 = 0; b2 < K; b2++) {
        const float wxy = wx[a] * wy[b2];
        if (wxy == 0.0f) continue;
        const float pv = v * wxy;
        const int oxy = ox[a] + oy[b2];
#pragma unroll
        for (int c = 0; c < K; c++) {
          if (wz[c] == 0.0f) continue;
          if (WIDE)
            atomicAdd((unsigned long long *)smi + oxy + oz[c], (unsigned long long)__float2ll_rn(pv * wz[c]));
          else
            limb_add(lo + oxy + oz[c], hi + oxy + oz[c], pv * wz[c], two_mk, two_k);
        }
      }
  }
}

// (r0, r1: this CTA's records of the tile's cnt; st4: sum |w v^ea|, sum |w v^eb|, and the two largest, over r0 to r1.) The
// CTAs of a cluster take one scale, from the tile's sums, so that their cells add up as integers and a cell is rounded once.
template <int K, int NF, bool IL, bool CL>
__device__ void tile_paint_dense(const Geom &g, const FieldSpec &fs, const TileGeo &tg, const float4 *recs,
                                 const float *recw, unsigned long long r0, unsigned long long r1, unsigned cnt, float4 st4,
                                 const TileAt &at, int *smi, float4 *s_stat, GridPtrs grids, DevStats *st) {
  constexpr int NS = IL ? 2 : 1;
  const int slotw = tg.slot;
  int *lo = smi, *hi = smi + slotw;
  if (CL) {
    if (threadIdx.x == 0) *s_stat = st4;
    cluster_sync_all();
    const unsigned q = (unsigned)__cvta_generic_to_shared(s_stat);
    st4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int k = 0; k < at.S; k++) {
      const unsigned p = map_cluster(q, k);
      st4.x += ld_cluster_f32(p);
      st4.y += ld_cluster_f32(p + 4);
      st4.z = fmaxf(st4.z, ld_cluster_f32(p + 8));
      st4.w = fmaxf(st4.w, ld_cluster_f32(p + 12));
    }
  }
  bool wide[2];
  const int Sx[2] = {dense_scale(st4.x, st4.z, (float)cnt, wide[0]), dense_scale(st4.y, st4.w, (float)cnt, wide[1])};
#pragma unroll 1
  for (int slot = 0; slot < NS * NF; slot++) {
    const int sten = slot / NF, fld = slot % NF;
    const int S = fld ? Sx[1] : Sx[0];
    const bool wd = fld ? wide[1] : wide[0];
    const float sc = ldexpf(1.0f, S), inv = ldexpf(1.0f, -S);
    for (int c = threadIdx.x; c < 2 * slotw; c += blockDim.x) smi[c] = 0;
    __syncthreads();
    if (wd) {
      dense_deposit<K, true>(g, fs, tg, recs, recw, r0, r1, sten, fld, sc, at, smi);
    } else {
      for (unsigned long long rr = r0; rr < r1; rr += DENSE_ROUND) {
        if (rr > r0) {  // carries of the records so far
          __syncthreads();
          for (int c = threadIdx.x; c < slotw; c += blockDim.x) {
            const unsigned v = (unsigned)lo[c];
            hi[c] += (int)(v >> DENSE_K);
            lo[c] = (int)(v & ((1u << DENSE_K) - 1));
          }
          __syncthreads();
        }
        dense_deposit<K, false>(g, fs, tg, recs, recw, rr, min(r1, rr + DENSE_ROUND), sten, fld, sc, at, smi);
      }
    }
    if (CL) cluster_sync_all();
    else __syncthreads();
    float *gp = (float *)grids.g[slot];
    float dsum = 0.0f;
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smi);
    // a cell's two words (low, high) lie dh apart, the next cell's dc further on
    const int sh = wd ? 32 : DENSE_K, dh = wd ? 1 : slotw, dc = wd ? 2 : 1;
    auto value = [sh](int l, int h) { return ((long long)h << sh) + (long long)(unsigned)l; };
    tile_walk<CL>(g, tg, at, [&](int cp, long long go, bool two) {
      long long v0 = 0, v1 = 0;
      if (CL) {
        for (int k = 0; k < at.S; k++) {
          const unsigned q = map_cluster(sa, k) + 4 * dc * cp;
          v0 += value(ld_cluster_s32(q), ld_cluster_s32(q + 4 * dh));
          v1 += value(ld_cluster_s32(q + 4 * dc), ld_cluster_s32(q + 4 * (dc + dh)));
        }
      } else {
        const int *q = smi + dc * cp;
        v0 = value(q[0], q[dh]);
        v1 = value(q[dc], q[dc + dh]);
      }
      dsum += store_pair(gp + go, (float)v0 * inv, (float)v1 * inv, two);
    });
    const float vals[1] = {dsum};
    double *const dst1[1] = {&st->dc[slot]};
    block_add_f<1>(vals, dst1);
    if (CL) cluster_sync_all();  // every CTA has read this one's cells
  }
}

// FP32 tile kernel for particles away from every edge of the reference's rules (those are painted
// by k_edge_fixup). One CTA per tile, or (CL) a cluster of `split` CTAs that share a tile's records; shared
// memory holds the tile of every grid slot, both stencils, [tx][ty][tz] with the padded pitches py = 3, px = 9
// (mod 32) so that deposits at equal z spread over the banks, as int32 fixed point with a per-CTA
// power-of-two scale, so every deposit is one native integer shared-memory atomic (an ordinary tile's scale
// also keeps each deposit below 2^22, where rint_small rounds it). Lane = record: each thread reads one
// record, derives its taps once per stencil and adds the K^3 products, so a record is read once and nothing
// is staged. The cells are converted back to FP32 when the tile is written; in a cluster each CTA writes its
// share of the tile as the sum of every CTA's cells (through distributed shared memory). (NGRID of these
// particles is counted by the bucketing or k_count.)
// (Four CTAs per SM for one slot, whose cells are 40 KB: 62 registers instead of 79.)
template <int K, int NF, bool IL, bool CL>
__global__ void __launch_bounds__(256, NF * (IL ? 2 : 1) == 1 && !CL ? 4 : 3)
    k_tile_rec(Geom g, FieldSpec fs, TileGeo tg, const unsigned *offsets, const unsigned *counts, unsigned cap,
               const float4 *recs, const float *recw, unsigned long long capacity, int split, unsigned dense, GridPtrs grids,
               DevStats *st) {
  extern __shared__ __align__(16) int smi[];
  constexpr int NS = IL ? 2 : 1, SL = NS * NF;
  TileAt at;
  at.S = CL ? split : 1;
  const int tile = CL ? blockIdx.x / at.S : blockIdx.x;
  at.rank = CL ? blockIdx.x - tile * at.S : 0;
  const int bz = tile % tg.nbz, by = (tile / tg.nbz) % tg.nby, bx = tile / (tg.nbz * tg.nby);
  at.x0 = bx * tg.tx;
  at.y0 = by * tg.ty;
  at.z0 = bz * tg.tz;
  at.ex = min(tg.tx, g.nx - at.x0);
  at.ey = min(tg.ty, g.ny - at.y0);
  at.ez = min(tg.tz, g.nz - at.z0);
  unsigned long long rb, re;
  if (cap) {  // bucket mode: the tile's own bucket
    rb = (unsigned long long)tile * cap;
    re = rb + min(counts[tile], cap);
  } else {
    rb = offsets[tile];
    re = offsets[tile + 1];
  }
  if (re > capacity) re = capacity;
  if (rb > re) rb = re;
  const unsigned cnt = (unsigned)(re - rb);
  if (CL) {  // this CTA's share
    const unsigned per = (cnt + (unsigned)at.S - 1) / (unsigned)at.S;
    rb = min(re, rb + (unsigned long long)at.rank * per);
    re = min(re, rb + per);
  }
  // The first two records of each thread are loaded before the cells are cleared: a tile has a few records per thread, and
  // the wait for them stood between the clearing and the deposits (CIC, 1024^3, 134M particles, with the shorter deposits: 7.77 -> 7.22 ms).
  constexpr int PRE = 2;
  float4 prec[PRE];
  float pw[PRE];
#pragma unroll
  for (int u = 0; u < PRE; u++) {
    const unsigned long long r = rb + threadIdx.x + u * blockDim.x;
    if (r < re) {
      prec[u] = recs[r];
      pw[u] = recw ? recw[r] : 1.0f;
    }
  }
  int4 *sm4 = reinterpret_cast<int4 *>(smi);
  const int slotw = tg.slot;  // words per padded slot
  for (int c = threadIdx.x; c < (SL * slotw) >> 2; c += blockDim.x) sm4[c] = make_int4(0, 0, 0, 0);
  for (int c = ((SL * slotw) & ~3) + threadIdx.x; c < SL * slotw; c += blockDim.x) smi[c] = 0;
  // pre-pass over the records: sum and largest |w v^e| per field (the records stay in L1 for the deposits)
  __shared__ float red_abs[4][8];
  __shared__ float s_inv[2];  // 1 / scale of the CTA's cells per field
  __shared__ float4 s_stat;   // (dense tiles) the sums and largest values below
  {
    float la = 0.0f, lb = 0.0f, ma = 0.0f, mb = 0.0f;
    auto add = [&](const float4 &rec, float w) {
      float va, vb;
      record_values(fs, rec, w, va, vb);
      la += fabsf(va);
      lb += fabsf(vb);
      ma = fmaxf(ma, fabsf(va));
      mb = fmaxf(mb, fabsf(vb));
    };
#pragma unroll
    for (int u = 0; u < PRE; u++)
      if (rb + threadIdx.x + u * blockDim.x < re) add(prec[u], pw[u]);
    for (unsigned long long r = rb + threadIdx.x + PRE * blockDim.x; r < re; r += blockDim.x)
      add(recs[r], recw ? recw[r] : 1.0f);
    la = warp_sum_f(la);
    lb = warp_sum_f(lb);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      ma = fmaxf(ma, __shfl_xor_sync(0xffffffffu, ma, o));
      mb = fmaxf(mb, __shfl_xor_sync(0xffffffffu, mb, o));
    }
    if ((threadIdx.x & 31) == 0) {
      red_abs[0][threadIdx.x >> 5] = la;
      red_abs[1][threadIdx.x >> 5] = lb;
      red_abs[2][threadIdx.x >> 5] = ma;
      red_abs[3][threadIdx.x >> 5] = mb;
    }
    __syncthreads();
  }
  float ta = 0.0f, tb = 0.0f, xa = 0.0f, xb = 0.0f;
  for (int k = 0; k < (int)(blockDim.x >> 5); k++) {
    ta += red_abs[0][k];
    tb += red_abs[1][k];
    xa = fmaxf(xa, red_abs[2][k]);
    xb = fmaxf(xb, red_abs[3][k]);
  }
  if (cnt > dense) {  // uniform over the tile's CTAs
    tile_paint_dense<K, NF, IL, CL>(g, fs, tg, recs, recw, rb, re, cnt, make_float4(ta, tb, xa, xb), at, smi, &s_stat, grids,
                                    st);
    return;
  }
  // The scale is set by the sum (tile_scale_exp). When keeping every deposit below 2^22 costs
  // it at most 3 bits (an ordinary tile: hundreds of comparable records), the tile takes that scale
  // and the fast rounding; otherwise (few records, or one dominant record) it keeps the sum's scale
  // and rounds by conversion.
  const int SAs = tile_scale_exp(ta), SBs = tile_scale_exp(tb);
  const int SAf = min(SAs, tile_scale_max(xa)), SBf = min(SBs, tile_scale_max(xb));
  const bool fast = (SAs - SAf <= 3) && (NF == 1 || SBs - SBf <= 3);
  const int SA = fast ? SAf : SAs, SB = fast ? SBf : SBs;
  const float scA = ldexpf(1.0f, SA), scB = ldexpf(1.0f, SB);
  if (CL && threadIdx.x == 0) {
    s_inv[0] = ldexpf(1.0f, -SA);
    s_inv[1] = ldexpf(1.0f, -SB);
  }
  const bool inner = at.x0 >= 4 && at.x0 + at.ex <= g.nx - 5 && at.y0 >= 4 && at.y0 + at.ey <= g.ny - 5 && at.z0 >= 4 &&
                     at.z0 + at.ez <= g.nz - 5;
  if (fast && inner)
    tile_rec_deposit<K, NF, IL, true, true>(g, fs, tg, recs, recw, rb, re, scA, scB, at.x0, at.y0, at.z0, at.ex, at.ey, at.ez,
                                            smi);
  else if (fast)
    tile_rec_deposit<K, NF, IL, true, false>(g, fs, tg, recs, recw, rb, re, scA, scB, at.x0, at.y0, at.z0, at.ex, at.ey, at.ez,
                                             smi);
  else
    tile_rec_deposit<K, NF, IL, false, false>(g, fs, tg, recs, recw, rb, re, scA, scB, at.x0, at.y0, at.z0, at.ex, at.ey, at.ez,
                                              smi);
  if (CL) cluster_sync_all();
  else __syncthreads();
  // write every slot. The slots' DC sums go to one block reduction at the end (FP32 per thread and warp,
  // FP64 across warps).
  float dsums[SL], invs[SL];
#pragma unroll
  for (int slot = 0; slot < SL; slot++) {
    dsums[slot] = 0.0f;
    invs[slot] = ldexpf(1.0f, -((slot % NF) == 0 ? SA : SB));
  }
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smi), ia = (unsigned)__cvta_generic_to_shared(s_inv);
  tile_walk<CL>(g, tg, at, [&](int cp, long long go, bool two) {
#pragma unroll
    for (int slot = 0; slot < SL; slot++) {
      float a0, a1;
      if (CL) {
        a0 = a1 = 0.0f;
        for (int k = 0; k < at.S; k++) {
          const unsigned q = map_cluster(sa, k) + 4 * (slot * slotw + cp);
          const float inv = ld_cluster_f32(map_cluster(ia, k) + 4 * (slot % NF));
          a0 += (float)ld_cluster_s32(q) * inv;
          a1 += (float)ld_cluster_s32(q + 4) * inv;
        }
      } else {
        const int *sl = smi + slot * slotw + cp;
        a0 = (float)sl[0] * invs[slot];
        a1 = (float)sl[1] * invs[slot];
      }
      dsums[slot] += store_pair((float *)grids.g[slot] + go, a0, a1, two);
    }
  });
  double *dsts[SL];
#pragma unroll
  for (int slot = 0; slot < SL; slot++) dsts[slot] = &st->dc[slot];
  block_add_f<SL>(dsums, dsts);
  if (CL) cluster_sync_all();  // every CTA has read this one's cells
}

// --------------------------------------------------------------------- deterministic tile paint
// Tiles with at most this many records accumulate in two-limb cells at a tile scale; denser ones in
// uint64 cells at the run's global scale (64-bit shared atomics: slower, and rare).
#define DET_FAST_RECORDS 8192u

// Scale exponent of a tile: (record count) * (largest |w v^e| of its records) * 2^S < 2^40, so that no
// cell of one pass (each record adds at most |w v^e| 2^S to a cell) leaves the limbs' range. Both inputs
// are independent of the order of the records.
__device__ __forceinline__ int det_scale_exp(unsigned cnt, float max_abs) {
  const float bound = (float)cnt * max_abs * 1.001f;
  if (!(bound > 0.0f) || !isfinite(bound)) return 0;
  const int S = 39 - ilogbf(bound);
  return S > 100 ? 100 : (S < -100 ? -100 : S);
}

struct DetPass {
  int *lo, *hi;                  // two-limb cells of field 0 (field 1: + 2 slot); null in the uint64 mode
  unsigned long long *u;         // uint64 cells of field 0 (field 1: + slot)
  int slotw;
  float scA, scB, two_mk, two_k;  // fixed-point scales of the fields; 2^-k, 2^k
  double sc0, sc1;                // the same scales in FP64 (the CIC rounding-edge products)
};

template <int NF>
__device__ __forceinline__ void det_add(const DetPass &d, int off, float pa, float pb) {
  if (d.lo) {
    limb_add(d.lo + off, d.hi + off, pa, d.two_mk, d.two_k);
    if (NF == 2) limb_add(d.lo + 2 * d.slotw + off, d.hi + 2 * d.slotw + off, pb, d.two_mk, d.two_k);
  } else {
    atomicAdd(d.u + off, (unsigned long long)__float2ll_rn(pa));
    if (NF == 2) atomicAdd(d.u + d.slotw + off, (unsigned long long)__float2ll_rn(pb));
  }
}

// |w v^e| of one record for the tile's scale: the FP32 value, or for a special record its exact one.
template <typename T>
__device__ __forceinline__ void det_record_value(const Geom &g, const FieldSpec &fs, const PIn<T> &in, long long n,
                                                 const float4 &rec, float w, float &va, float &vb) {
  if (rec.x == SPECIAL_MARK) {
    const unsigned idx = __float_as_uint(rec.y);
    va = vb = 0.0f;
    if ((long long)idx >= n) return;
    double x, y, z, v, wd;
    exact_pos(g, fs, in, idx, x, y, z, v, wd);
    va = (float)wpow64(wd, v, fs.ea);
    vb = (float)wpow64(wd, v, fs.eb);
    return;
  }
  va = w;
  vb = w;
  for (int e = 0; e < fs.ea; e++) va *= rec.w;
  for (int e = 0; e < fs.eb; e++) vb *= rec.w;
}

// The exact FP64 rules of one special record (a particle within a few ulps of a discontinuity of the
// reference's rules, listed by its index) for stencil stn: its taps inside this tile. With stats its
// home tile also counts it in NGRID, in the out-of-box count and for the LOS == 0 error.
template <typename T, int NF>
__device__ void det_special(const Geom &g, const FieldSpec &fs, const TileGeo &tg, const PIn<T> &in, long long n,
                            unsigned idx, int tile, int x0, int y0, int z0, int ex, int ey, int ez, int stn,
                            bool stats, const DetPass &d, double &d_grid, double &d_out, int &fatal, DevStats *st) {
  if ((long long)idx >= n) return;
  double x, y, z, v, wd;
  exact_pos(g, fs, in, idx, x, y, z, v, wd);
  if (stats) {
    const Prep p = prep32(g, fs, in, idx);
    if (home_of(g, tg, p.sx, p.sy, p.sz) == tile) {
      if (outside_box(g, x, y, z)) {  // src/read_data.c:81-88
        d_out += 1.0;
        if (g.los == 0) {
          fatal = 1;
          atomicMax(&st->fatal_inv, ~0ULL - (unsigned long long)idx);
        }
      }
      AxisTaps ax, ay, az;
      if (exact_axes(g, x, y, z, ax, ay, az)) d_grid += wd;
    }
  }
  const double va64 = wpow64(wd, v, fs.ea), vb64 = wpow64(wd, v, fs.eb);
  const float va = (float)va64 * d.scA, vb = (float)vb64 * d.scB;
  AxisTaps ax, ay, az;
  const double px = stn ? DADD(x, g.hx) : x, py = stn ? DADD(y, g.hy) : y, pz = stn ? DADD(z, g.hz) : z;
  if (!exact_axes(g, px, py, pz, ax, ay, az)) return;
  float W[9];
  int O[9];
  stage_axis64(g, ax, 0, x0, ex, tg.px, W, O);
  stage_axis64(g, ay, 1, y0, ey, tg.py, W + 3, O + 3);
  stage_axis64(g, az, 2, z0, ez, 1, W + 6, O + 6);
  // CIC rounding edge: y index NY lands in row 0 of the next x slice (src/read_data.c:592-593)
  if (g.order == 2 && ay.n > 0 && ay.idx[0] == g.ny && ay.on[0]) {
    for (int a = 0; a < ax.n; a++)
      for (int c = 0; c < az.n; c++) {
        if (!(ax.on[a] && az.on[c])) continue;
        const long long L = canon_index(g, ax.idx[a], ay.idx[0], az.idx[c]);
        if (L < 0) continue;
        int ix, iy, iz;
        decode(g, L, ix, iy, iz);
        ix -= x0;
        iy -= y0;
        iz -= z0;
        if (ix < 0 || ix >= ex || iy < 0 || iy >= ey || iz < 0 || iz >= ez) continue;
        const double tw = DMUL(DMUL(ax.w[a], ay.w[0]), az.w[c]);
        det_add<NF>(d, ix * tg.px + iy * tg.py + iz, (float)(DMUL(va64, tw) * d.sc0), (float)(DMUL(vb64, tw) * d.sc1));
      }
  }
  for (int a = 0; a < 3; a++)
    for (int b2 = 0; b2 < 3; b2++)
      for (int c = 0; c < 3; c++) {
        const float wt = W[a] * W[3 + b2] * W[6 + c];
        if (wt != 0.0f) det_add<NF>(d, O[a] + O[3 + b2] + O[6 + c], va * wt, vb * wt);
      }
}

// Deterministic tile kernel (k_count -> k_scan -> k_scatter -> here): one CTA per tile and, as in k_tile_rec,
// lane = record; the two stencils one after the other (one pass each over the tile's records), each pass
// holding both fields of its stencil in shared memory as int64 fixed point. The cells of a tile with at most
// DET_FAST_RECORDS records are two int32 limbs at the tile's own scale (det_scale_exp: from the record count
// and the largest |w v^e|, both independent of the order of the records); denser tiles use uint64 cells at
// the run's global scale (k_scan: the catalogue's sum of |w v^e| times 2^S below 2^62). A deposit is the FP32
// product at that scale rounded once to an integer, and integer addition makes every cell, and so the grids,
// independent of the order of the deposits: bit-reproducible. Special records take the exact FP64 rules
// here (det_special). The home tile of each record counts it in NGRID and the out-of-box count (k_count only
// counted the tiles); the slots' DC sums go to the exact global integer sums at the global scale.
template <typename T, int K, int NF, bool IL>
__global__ void __launch_bounds__(256, 3) k_tile_rec_det(Geom g, FieldSpec fs, TileGeo tg, PIn<T> in, long long n,
                                                         const unsigned *offsets, const float4 *recs,
                                                         const float *recw, unsigned long long capacity,
                                                         GridPtrs grids, const double *fixed_scale, DevStats *st) {
  extern __shared__ __align__(16) int smd[];
  constexpr int NS = IL ? 2 : 1;
  const int tile = blockIdx.x;
  const int bz = tile % tg.nbz, by = (tile / tg.nbz) % tg.nby, bx = tile / (tg.nbz * tg.nby);
  const int x0 = bx * tg.tx, y0 = by * tg.ty, z0 = bz * tg.tz;
  const int ex = min(tg.tx, g.nx - x0), ey = min(tg.ty, g.ny - y0), ez = min(tg.tz, g.nz - z0);
  const int slotw = tg.slot;
  unsigned long long rb = offsets[tile], re = offsets[tile + 1];
  if (re > capacity) re = capacity;
  if (rb > re) rb = re;
  const unsigned cnt = (unsigned)(re - rb);
  const bool fast = cnt <= DET_FAST_RECORDS;
  __shared__ float red_max[2][32];
  float ma = 0.0f, mb = 0.0f;
  if (fast) {  // the tile's largest |w v^e| per field
    for (unsigned long long r = rb + threadIdx.x; r < re; r += blockDim.x) {
      float va, vb;
      det_record_value(g, fs, in, n, recs[r], recw ? recw[r] : 1.0f, va, vb);
      ma = fmaxf(ma, fabsf(va));
      mb = fmaxf(mb, fabsf(vb));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      ma = fmaxf(ma, __shfl_xor_sync(FULL_MASK, ma, o));
      mb = fmaxf(mb, __shfl_xor_sync(FULL_MASK, mb, o));
    }
    if ((threadIdx.x & 31) == 0) {
      red_max[0][threadIdx.x >> 5] = ma;
      red_max[1][threadIdx.x >> 5] = mb;
    }
    __syncthreads();
    for (int k = 0; k < (int)(blockDim.x >> 5); k++) {
      ma = fmaxf(ma, red_max[0][k]);
      mb = fmaxf(mb, red_max[1][k]);
    }
  }
  const double G0 = fixed_scale[0], G1 = fixed_scale[1];
  const int SA = det_scale_exp(cnt, ma), SB = det_scale_exp(cnt, mb);
  const int kb = 31 - (32 - __clz(cnt));  // k with cnt 2^k < 2^31
  const int k = kb > 22 ? 22 : kb;
  DetPass d;
  d.slotw = slotw;
  if (fast) {
    d.lo = smd;
    d.hi = smd + slotw;
    d.u = nullptr;
    d.scA = ldexpf(1.0f, SA);
    d.scB = ldexpf(1.0f, SB);
    d.two_mk = ldexpf(1.0f, -k);
    d.two_k = ldexpf(1.0f, k);
  } else {
    d.lo = d.hi = nullptr;
    d.u = reinterpret_cast<unsigned long long *>(smd);
    d.scA = (float)G0;
    d.scB = (float)G1;
    d.two_mk = d.two_k = 1.0f;
  }
  d.sc0 = (double)d.scA;
  d.sc1 = (double)d.scB;
  float f_grid = 0.0f, f_out = 0.0f;
  double d_grid = 0.0, d_out = 0.0;
  int fatal = 0;
#pragma unroll 1
  for (int stn = 0; stn < NS; stn++) {
    for (int c = threadIdx.x; c < NF * 2 * slotw; c += blockDim.x) smd[c] = 0;
    __syncthreads();
    for (unsigned long long r = rb + threadIdx.x; r < re; r += blockDim.x) {
      const float4 rec = recs[r];
      if (rec.x == SPECIAL_MARK) {
        det_special<T, NF>(g, fs, tg, in, n, __float_as_uint(rec.y), tile, x0, y0, z0, ex, ey, ez, stn, stn == 0, d,
                           d_grid, d_out, fatal, st);
        continue;
      }
      const float w = recw ? recw[r] : 1.0f;
      if (stn == 0 && home_of(g, tg, rec.x, rec.y, rec.z) == tile) {
        if (accept32(g, rec.x, rec.y, rec.z)) f_grid += w;
        if (outside32(g, rec.x, rec.y, rec.z)) f_out += 1.0f;  // src/read_data.c:81-88
      }
      float va = w, vb = w;
      for (int e = 0; e < fs.ea; e++) va *= rec.w;
      for (int e = 0; e < fs.eb; e++) vb *= rec.w;
      va *= d.scA;
      vb *= d.scB;
      const float sx = stn ? __fadd_rn(rec.x, 0.5f) : rec.x, sy = stn ? __fadd_rn(rec.y, 0.5f) : rec.y,
                  sz = stn ? __fadd_rn(rec.z, 0.5f) : rec.z;
      if (!accept32(g, sx, sy, sz)) continue;
      AxisTapsF ax, ay, az;
      axis32k<K>(sx, 0, g.nx, g.los, ax);
      axis32k<K>(sy, 1, g.ny, g.los, ay);
      axis32k<K>(sz, 1, g.nz, g.los, az);
      float wx[3], wy[3], wz[3];
      int ox[3], oy[3], oz[3];
      stage_axis32(ax, x0, ex, tg.px, wx, ox);
      stage_axis32(ay, y0, ey, tg.py, wy, oy);
      stage_axis32(az, z0, ez, 1, wz, oz);
#pragma unroll
      for (int a = 0; a < K; a++)
#pragma unroll
        for (int b2 = 0; b2 < K; b2++) {
          const float wxy = wx[a] * wy[b2];
          if (wxy == 0.0f) continue;
          const float pa = va * wxy, pb = vb * wxy;
          const int oxy = ox[a] + oy[b2];
#pragma unroll
          for (int c = 0; c < K; c++)
            if (wz[c] != 0.0f) det_add<NF>(d, oxy + oz[c], pa * wz[c], pb * wz[c]);
        }
    }
    __syncthreads();
    // write this stencil's slots: pairs of cells along z as float2 (rows start 8-byte aligned in global
    // memory: the padded row length 2*(NZ/2+1) is even); the slots' integer DC sums at the global scale
    const int npair = (tg.tx * tg.ty * tg.tz) >> 1;
#pragma unroll
    for (int f = 0; f < NF; f++) {
      const int slot = stn * NF + f;
      float *gp = (float *)grids.g[slot];
      const double inv = fast ? ldexp(1.0, -(f ? SB : SA)) : 1.0 / (f ? G1 : G0);
      long long isum = 0;
      for (int q = threadIdx.x; q < npair; q += blockDim.x) {
        const int c = q << 1;
        const int rz = c & (tg.tz - 1), ly = (c >> tg.lz) & (tg.ty - 1), lx = c >> (tg.lz + tg.ly);
        if (lx >= ex || ly >= ey || rz >= ez) continue;
        const int sidx = lx * tg.px + ly * tg.py + rz;
        long long a0, a1;
        if (fast) {
          const int *lo = smd + 2 * f * slotw, *hi = lo + slotw;
          a0 = (long long)hi[sidx] * (1ll << k) + (long long)lo[sidx];
          a1 = (long long)hi[sidx + 1] * (1ll << k) + (long long)lo[sidx + 1];
        } else {
          const unsigned long long *u = reinterpret_cast<const unsigned long long *>(smd) + f * slotw;
          a0 = (long long)u[sidx];
          a1 = (long long)u[sidx + 1];
        }
        const bool two = rz + 1 < ez;
        isum += a0 + (two ? a1 : 0ll);
        float *dst = gp + (long long)(x0 + lx) * g.slice + (long long)(y0 + ly) * g.row + z0 + rz;
        if (two) *reinterpret_cast<float2 *>(dst) = make_float2((float)((double)a0 * inv), (float)((double)a1 * inv));
        else dst[0] = (float)((double)a0 * inv);
      }
      for (int o = 16; o > 0; o >>= 1) isum += __shfl_xor_sync(FULL_MASK, isum, o);
      if ((threadIdx.x & 31) == 0 && isum) {
        // to the global scale: exact (a power of two) where it is the finer one, else rounded once
        const long long gsum = fast ? __double2ll_rn((double)isum * ((f ? G1 : G0) * inv)) : isum;
        atomicAdd(&st->dc_fixed[slot], (unsigned long long)gsum);
      }
    }
    __syncthreads();
  }
  const double vals[2] = {d_grid + (double)f_grid, d_out + (double)f_out};
  double *const dst[2] = {&st->ngrid, &st->nout};
  block_add<2>(vals, dst);
  if (fatal) atomicOr(&st->fatal, 1);
}

// Bucket mode: records that found their tile's bucket full, deposited after the tiles were written
// (FP32 global atomics), each restricted to the taps inside its own tile, with their DC sums.
template <int K, int NF, bool IL>
__global__ void __launch_bounds__(128) k_ovf_paint(Geom g, FieldSpec fs, TileGeo tg, const float4 *ovf_recs,
                                                   const float *ovf_w, const unsigned *ovf_tile,
                                                   const unsigned *ovf_count, unsigned long long ovf_cap,
                                                   GridPtrs grids, DevStats *st) {
  constexpr int NS = IL ? 2 : 1;
  const unsigned long long no = min((unsigned long long)*ovf_count, ovf_cap);
  if (blockIdx.x * (unsigned long long)blockDim.x >= no) return;  // (most calls have none: no block sums then)
  double l_dc[4] = {0, 0, 0, 0};
  for (unsigned long long o = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; o < no;
       o += (unsigned long long)gridDim.x * blockDim.x) {
    const float4 rec = ovf_recs[o];
    const float w = ovf_w ? ovf_w[o] : 1.0f;
    const int tile = (int)ovf_tile[o];
    const int bz = tile % tg.nbz, by = (tile / tg.nbz) % tg.nby, bx = tile / (tg.nbz * tg.nby);
    const int x0 = bx * tg.tx, y0 = by * tg.ty, z0 = bz * tg.tz;
    const int ex = min(tg.tx, g.nx - x0), ey = min(tg.ty, g.ny - y0), ez = min(tg.tz, g.nz - z0);
    float va = w, vb = w;
    for (int e = 0; e < fs.ea; e++) va *= rec.w;
    for (int e = 0; e < fs.eb; e++) vb *= rec.w;
#pragma unroll
    for (int s = 0; s < NS; s++) {
      const float sx = s ? __fadd_rn(rec.x, 0.5f) : rec.x, sy = s ? __fadd_rn(rec.y, 0.5f) : rec.y,
                  sz = s ? __fadd_rn(rec.z, 0.5f) : rec.z;
      if (!accept32(g, sx, sy, sz)) continue;
      AxisTapsF ax, ay, az;
      axis32k<K>(sx, 0, g.nx, g.los, ax);
      axis32k<K>(sy, 1, g.ny, g.los, ay);
      axis32k<K>(sz, 1, g.nz, g.los, az);
      float wx[3], wy[3], wz[3];
      int lx[3], ly[3], lz[3];
      stage_axis32(ax, x0, ex, 1, wx, lx);
      stage_axis32(ay, y0, ey, 1, wy, ly);
      stage_axis32(az, z0, ez, 1, wz, lz);
#pragma unroll
      for (int a = 0; a < K; a++)
#pragma unroll
        for (int b2 = 0; b2 < K; b2++) {
          const float wxy = wx[a] * wy[b2];
          const long long rowb = ((long long)(x0 + lx[a]) * g.ny + (y0 + ly[b2])) * g.row + z0;
#pragma unroll
          for (int c = 0; c < K; c++) {
            if (wxy == 0.0f || wz[c] == 0.0f) continue;
            const float da = (va * wxy) * wz[c];
            atomicAdd((float *)grids.g[s * NF] + rowb + lz[c], da);
            l_dc[s * NF] += (double)da;
            if (NF == 2) {
              const float db = (vb * wxy) * wz[c];
              atomicAdd((float *)grids.g[s * NF + 1] + rowb + lz[c], db);
              l_dc[s * NF + 1] += (double)db;
            }
          }
        }
    }
  }
  const double vals[4] = {l_dc[0], l_dc[1], l_dc[2], l_dc[3]};
  double *const dst[4] = {&st->dc[0], &st->dc[1], &st->dc[2], &st->dc[3]};
  block_add<4>(vals, dst);
}

// Particles near an edge of the reference's rules, painted after the tiles with the exact FP64
// rules and global atomics into the FP32 grids; their exact statistics (NGRID, the out-of-box
// count, the LOS == 0 error) are added here. One warp per particle: lanes 0-2 take the taps of the
// three axes, then lane t deposits tap t (each a serial chain of FP64 steps otherwise).
template <typename T>
__global__ void __launch_bounds__(128) k_edge_fixup(Geom g, FieldSpec fs, PIn<T> in, const unsigned *edge_list,
                                                    const unsigned *edge_count, GridPtrs grids, DevStats *st) {
  const unsigned ne = *edge_count;
  if (blockIdx.x * (blockDim.x >> 5) >= ne) return;  // nothing for this CTA: no block sums
  const int nf = fs.nfields, nst = g.interlace ? 2 : 1;
  const int lane = threadIdx.x & 31;
  const unsigned warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarp = (gridDim.x * blockDim.x) >> 5;
  double d_grid = 0.0, d_out = 0.0, l_dc[4] = {0, 0, 0, 0};
  int fatal = 0;
  for (unsigned k = warp; k < ne; k += nwarp) {
    const unsigned idx = edge_list[k];
    double x, y, z, v, w;
    exact_pos(g, fs, in, idx, x, y, z, v, w);
    if (outside_box(g, x, y, z)) {  // src/read_data.c:81-88
      if (lane == 0) d_out += 1.0;
      if (g.los == 0) {
        fatal = 1;
        if (lane == 0) atomicMax(&st->fatal_inv, ~0ULL - (unsigned long long)idx);
        continue;
      }
    }
    const double val[2] = {wpow64(w, v, fs.ea), wpow64(w, v, fs.eb)};
    for (int stn = 0; stn < nst; stn++) {
      const double px = stn ? DADD(x, g.hx) : x, py = stn ? DADD(y, g.hy) : y, pz = stn ? DADD(z, g.hz) : z;
      AxisTaps t;
      t.n = 0;
      bool acc = true;
      if (lane < 3) acc = exact_axis(g, lane, lane == 0 ? px : (lane == 1 ? py : pz), t);
      if (__ballot_sync(FULL_MASK, !acc)) continue;  // rejected by some axis
      if (stn == 0 && lane == 0) d_grid += w;
      // this lane's tap (a, b, c) of a 3 x 3 x 3 block; the axes' taps from lanes 0, 1, 2
      const int ta = lane / 9, tb = (lane / 3) % 3, tc = lane % 3;
      const int nx_ = __shfl_sync(FULL_MASK, t.n, 0), ny_ = __shfl_sync(FULL_MASK, t.n, 1),
                nz_ = __shfl_sync(FULL_MASK, t.n, 2);
      int ix = 0, iy = 0, iz = 0, on = 1;
      double wx = 0.0, wy = 0.0, wz = 0.0;
#pragma unroll
      for (int q = 0; q < 3; q++) {
        const int i0 = __shfl_sync(FULL_MASK, t.idx[q], 0), i1 = __shfl_sync(FULL_MASK, t.idx[q], 1),
                  i2 = __shfl_sync(FULL_MASK, t.idx[q], 2);
        const int o0 = __shfl_sync(FULL_MASK, (int)t.on[q], 0), o1 = __shfl_sync(FULL_MASK, (int)t.on[q], 1),
                  o2 = __shfl_sync(FULL_MASK, (int)t.on[q], 2);
        const double w0 = __shfl_sync(FULL_MASK, t.w[q], 0), w1 = __shfl_sync(FULL_MASK, t.w[q], 1),
                     w2 = __shfl_sync(FULL_MASK, t.w[q], 2);
        if (ta == q) { ix = i0; wx = w0; on &= o0; }
        if (tb == q) { iy = i1; wy = w1; on &= o1; }
        if (tc == q) { iz = i2; wz = w2; on &= o2; }
      }
      if (lane >= 27 || ta >= nx_ || tb >= ny_ || tc >= nz_ || !on) continue;
      const long long L = canon_index(g, ix, iy, iz);
      if (L < 0) continue;
      const double tw = DMUL(DMUL(wx, wy), wz);
      for (int f = 0; f < nf; f++) {
        const float dep = (float)DMUL(val[f], tw);
        atomicAdd((float *)grids.g[stn * nf + f] + L, dep);
        l_dc[stn * nf + f] += (double)dep;
      }
    }
  }
  const double vals[6] = {d_grid, d_out, l_dc[0], l_dc[1], l_dc[2], l_dc[3]};
  double *const dst[6] = {&st->ngrid, &st->nout, &st->dc[0], &st->dc[1], &st->dc[2], &st->dc[3]};
  block_add<6>(vals, dst);
  if (fatal) atomicOr(&st->fatal, 1);
}

static int pow2_at_least(int n) {
  int p = 1;
  while (p < n) p <<= 1;
  return p;
}

static int log2i(int p) {
  int l = 0;
  while ((1 << l) < p) l++;
  return l;
}

TileGeo choose_tiles(const Geom &g, int nslots, int deterministic) {
  // 4 grid slots x 8x16x32 floats = 64 KB (three CTAs per SM). The deterministic kernel holds one stencil's
  // fields at a time, as 8-byte cells: the same tiles for two fields (or one field interlaced), the
  // 16x16x32 ones for a single field otherwise.
  if (deterministic) return make_tiles(g, nslots == 1 ? 16 : 8, 16, 32);
  return make_tiles(g, nslots <= 2 ? 16 : 8, 16, 32);
}

// The FP32 tiles of a context: the default ones, or for a small grid smaller ones, so that there is about one
// tile for each SM (rec_split then adds CTAs). (Edges below 8 would put a footprint in three tiles along an axis.)
TileGeo fit_tiles(const Geom &g, int nslots) {
  static const int edge[5][3] = {{16, 16, 32}, {16, 16, 16}, {8, 16, 16}, {8, 8, 16}, {8, 8, 8}};
  TileGeo t = choose_tiles(g, nslots, 0);
  for (int k = nslots <= 2 ? 1 : 2; k < 5 && t.ntiles < 152; k++) t = make_tiles(g, edge[k][0], edge[k][1], edge[k][2]);
  return t;
}

// Tile edges are powers of two (tile coordinates are shifts); a grid edge shorter than the tile
// uses the next power of two and the tile is partial.
TileGeo make_tiles(const Geom &g, int tx, int ty, int tz) {
  TileGeo t;
  t.tx = tx;
  t.ty = ty;
  t.tz = tz;
  t.tz = t.tz < pow2_at_least(g.nz) ? t.tz : pow2_at_least(g.nz);
  t.ty = t.ty < pow2_at_least(g.ny) ? t.ty : pow2_at_least(g.ny);
  t.tx = t.tx < pow2_at_least(g.nx) ? t.tx : pow2_at_least(g.nx);
  t.lx = log2i(t.tx);
  t.ly = log2i(t.ty);
  t.lz = log2i(t.tz);
  t.nbx = (g.nx + t.tx - 1) / t.tx;
  t.nby = (g.ny + t.ty - 1) / t.ty;
  t.nbz = (g.nz + t.tz - 1) / t.tz;
  t.ntiles = t.nbx * t.nby * t.nbz;
  t.py = t.tz + 1;  // >= tz + 1 so a z pair never straddles rows; = 3 (mod 32)
  while (t.py % 32 != 3) t.py++;
  t.px = t.ty * t.py;
  while (t.px % 32 != 9) t.px++;
  t.slot = t.px * t.tx;
  return t;
}

size_t tile_smem_bytes(const TileGeo &tg, int nslots, int deterministic) {
  return ((size_t)nslots * tg.slot * (deterministic ? 8 : 4) + 15) & ~(size_t)15;
}

// k_tile_rec's cells: every slot, or (dense) where a tile may be dense the two limbs of one slot if they are more.
size_t rec_smem_bytes(const TileGeo &tg, int nslots, bool dense) {
  return (size_t)(dense && nslots < 2 ? 2 : nslots) * tg.slot * 4;
}

double tile_dup_estimate(const Geom &g, const TileGeo &tg) {
  // a footprint spans 4 (TSC, CIC) or 2 (NN) cells plus the margin; it crosses into the next tile
  // with probability (span - 1) / tile edge
  const double span = (g.order == 1 ? 2.0 : (g.order == 2 ? 3.0 : 4.0)) + 2.0 * g.margin;
  return (1.0 + (span - 1.0) / tg.tx) * (1.0 + (span - 1.0) / tg.ty) * (1.0 + (span - 1.0) / tg.tz);
}

// CTAs per tile, a power of two up to 8 (a cluster shares the tile's records): the one whose busiest SM is done first. A CTA
// costs a fixed time (its cells cleared and written, in a cluster also its barriers and the reading of the others' cells) and
// its share of the deposits; an SM works through its CTAs' deposits 1.9 and 2.4 times as fast with two and with three of them
// as with one. The times (us, fitted to 1080 launches: NN to TSC, one to four slots, 64 to 512 tiles, 80 to 200,000 records a
// tile) only rank the four; a cluster has to win by 4 %, one of eight by 15 %. 128^3, two slots, 60,000 to 600,000 CIC
// particles: one CTA 17 to 29 us, two 31 to 44; 48^3, two slots, TSC, 600,000: 160 us by one, 107 by two, 113 by four; 32^3,
// 200,000: 158, 88, 60 and 72 us by one to eight.
static int rec_split(const TileGeo &tg, int K, int slots, double records, unsigned dense) {
  const double r = records / tg.ntiles, kwords = (double)tg.tx * tg.ty * tg.tz * std::max(slots, 2) / 1024.0;
  const double dep = 0.18e-3 * r * (22.0 + (r > dense ? 2.2 : 1.0) * K * K * K * slots);
  const double bias[4] = {1.0, 1.04, 1.04, 1.15};
  int best = 0;
  double best_t = 0.0;
  for (int k = 0; k < 4 && (k == 0 || tg.ntiles << k <= 152 * 6); k++) {
    const double ctas = std::max(1.0, ceil((double)(tg.ntiles << k) / 152.0 - 0.1));  // of the busiest SM
    const double fix = 1.4 + 0.07 * kwords + (k ? 1.25 + 0.09 * kwords : 0.0);
    const double t = bias[k] * (8.0 + ctas * fix + ctas / (1 << k) * dep / (ctas <= 1.0 ? 1.0 : (ctas <= 2.0 ? 1.9 : 2.4)));
    if (k == 0 || t < best_t) {
      best = k;
      best_t = t;
    }
  }
  return 1 << best;
}

template <int K, int NF, bool IL>
static void launch_rec(cudaStream_t s, const Geom &g, const FieldSpec &fs, const TileGeo &tg, const PaintBufs &b,
                       bool weights, long long n, const GridPtrs &grids, DevStats *st) {
  const float *recw = weights ? b.recw : nullptr;
  const TileGeo def = choose_tiles(g, NF * (IL ? 2 : 1), 0);
  const unsigned dense = (unsigned)((double)TILE_DENSE_RECORDS * std::min(1.0, (double)tg.tx * tg.ty * tg.tz /
                                                                               ((double)def.tx * def.ty * def.tz)));
  const int split = rec_split(tg, K, NF * (IL ? 2 : 1), tile_dup_estimate(g, tg) * (double)n, dense);
  // (buckets that end below the dense limit: no tile needs the limbs' second slot. One slot, 512x256x256, TSC, 0.24M
  // particles: 58 -> 57 us with 40 instead of 80 KB a CTA, 52 with the fourth CTA per SM that this leaves room for)
  const bool may_dense = b.bucket_cap == 0 || b.bucket_cap > dense;
  const size_t smem = rec_smem_bytes(tg, NF * (IL ? 2 : 1), may_dense);
  if (split > 1) {
    allow_smem(k_tile_rec<K, NF, IL, true>, 4096);
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)split;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tg.ntiles * split));
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k_tile_rec<K, NF, IL, true>, g, fs, tg, (const unsigned *)b.offsets,
                       (const unsigned *)b.counts, b.bucket_cap, (const float4 *)b.recs, recw, b.capacity, split, dense,
                       grids, st);
  } else {
    allow_smem(k_tile_rec<K, NF, IL, false>, 4096);
    k_tile_rec<K, NF, IL, false><<<tg.ntiles, 256, smem, s>>>(g, fs, tg, b.offsets, b.counts, b.bucket_cap, b.recs,
                                                                   recw, b.capacity, 1, dense, grids, st);
  }
  if (b.bucket_cap)
    k_ovf_paint<K, NF, IL><<<152 * 2, 128, 0, s>>>(g, fs, tg, b.ovf_recs, weights ? b.ovf_w : nullptr, b.ovf_tile,
                                                   b.ovf_count, b.ovf_cap, grids, st);
}

template <int K>
static void launch_rec_k(cudaStream_t s, const Geom &g, const FieldSpec &fs, const TileGeo &tg, const PaintBufs &b,
                         bool weights, long long n, const GridPtrs &grids, DevStats *st) {
  if (fs.nfields == 2) {
    if (g.interlace) launch_rec<K, 2, true>(s, g, fs, tg, b, weights, n, grids, st);
    else launch_rec<K, 2, false>(s, g, fs, tg, b, weights, n, grids, st);
  } else {
    if (g.interlace) launch_rec<K, 1, true>(s, g, fs, tg, b, weights, n, grids, st);
    else launch_rec<K, 1, false>(s, g, fs, tg, b, weights, n, grids, st);
  }
}

template <typename T, int K, int NF, bool IL>
static void launch_det(cudaStream_t s, const Geom &g, const FieldSpec &fs, const TileGeo &tg, const PIn<T> &in,
                       long long n, const PaintBufs &b, const GridPtrs &grids, DevStats *st) {
  const size_t smem = tile_smem_bytes(tg, NF, 1);
  allow_smem(k_tile_rec_det<T, K, NF, IL>, 4096);
  k_tile_rec_det<T, K, NF, IL><<<tg.ntiles, 256, smem, s>>>(g, fs, tg, in, n, b.offsets, b.recs,
                                                            in.w ? b.recw : nullptr, b.capacity, grids, b.fixed_scale,
                                                            st);
}

template <typename T, int K>
static void launch_det_k(cudaStream_t s, const Geom &g, const FieldSpec &fs, const TileGeo &tg, const PIn<T> &in,
                         long long n, const PaintBufs &b, const GridPtrs &grids, DevStats *st) {
  if (fs.nfields == 2) {
    if (g.interlace) launch_det<T, K, 2, true>(s, g, fs, tg, in, n, b, grids, st);
    else launch_det<T, K, 2, false>(s, g, fs, tg, in, n, b, grids, st);
  } else {
    if (g.interlace) launch_det<T, K, 1, true>(s, g, fs, tg, in, n, b, grids, st);
    else launch_det<T, K, 1, false>(s, g, fs, tg, in, n, b, grids, st);
  }
}

template <typename T>
static void run_paint32(cudaStream_t s, const Geom &g, const FieldSpec &fs, const TileGeo &tg, int det, PIn<T> in,
                        long long n, const GridPtrs &grids, const PaintBufs &b, DevStats *st, long long *launches) {
  const int th = 256;
  long long nbl = (n + th - 1) / th;
  const int nb = (int)(nbl < 1 ? 1 : (nbl > 152 * 8 ? 152 * 8 : nbl));  // one resident wave of 256-thread blocks
  const bool split = !det;  // FP32: edge particles go to k_edge_fixup; deterministic: exact rules in the tiles
  cudaMemsetAsync(b.counts, 0, sizeof(unsigned) * tg.ntiles, s);
  if (split) cudaMemsetAsync(b.edge_count, 0, sizeof(unsigned), s);
  if (!det && b.bucket_cap) {  // bucket mode: one pass to the tiles' buckets, overflow after the tiles
    cudaMemsetAsync(b.ovf_count, 0, sizeof(unsigned), s);
    const int nch = b.nchunk > 1 ? b.nchunk : 1;
    for (int k = 0; k < nch; k++) {  // one launch per copied chunk of a host catalogue (else one)
      const long long c0 = n * k / nch, c1 = n * (k + 1) / nch;
      if (nch > 1) cudaStreamWaitEvent(s, b.chunk_ev[k], 0);
      PIn<T> ink{in.x + c0, in.y + c0, in.z + c0, in.v ? in.v + c0 : nullptr, in.w ? in.w + c0 : nullptr};
      launch_bucket<T>(s, g, fs, tg, ink, c1 - c0, c0, b, st);
    }
    *launches += nch - 1;
    const bool wts = in.w != nullptr;
    if (b.tile_ev0) cudaEventRecord(b.tile_ev0, s);
    if (g.order == 3) launch_rec_k<3>(s, g, fs, tg, b, wts, n, grids, st);
    else if (g.order == 2) launch_rec_k<2>(s, g, fs, tg, b, wts, n, grids, st);
    else launch_rec_k<1>(s, g, fs, tg, b, wts, n, grids, st);
    if (b.tile_ev1) cudaEventRecord(b.tile_ev1, s);
    k_edge_fixup<T><<<152 * 2, 128, 0, s>>>(g, fs, in, b.edge_list, b.edge_count, grids, st);
    *launches += 4;
    return;
  }
  k_count<T><<<nb, th, 0, s>>>(g, fs, tg, in, n, b.counts, st, split ? 1 : 0);
  k_scan<<<1, 1024, 0, s>>>(b.counts, tg.ntiles, b.offsets, b.cursor, st, b.capacity, b.fixed_scale);
  k_scatter<T><<<nb, th, 0, s>>>(g, fs, tg, in, n, b.cursor, b.recs, in.w ? b.recw : nullptr, b.capacity,
                                 split ? b.edge_list : nullptr, b.edge_count);
  if (det) {
    if (b.tile_ev0) cudaEventRecord(b.tile_ev0, s);
    if (g.order == 3) launch_det_k<T, 3>(s, g, fs, tg, in, n, b, grids, st);
    else if (g.order == 2) launch_det_k<T, 2>(s, g, fs, tg, in, n, b, grids, st);
    else launch_det_k<T, 1>(s, g, fs, tg, in, n, b, grids, st);
    if (b.tile_ev1) cudaEventRecord(b.tile_ev1, s);
    *launches += 4;
  } else {
    const bool wts = in.w != nullptr;
    if (b.tile_ev0) cudaEventRecord(b.tile_ev0, s);
    if (g.order == 3) launch_rec_k<3>(s, g, fs, tg, b, wts, n, grids, st);
    else if (g.order == 2) launch_rec_k<2>(s, g, fs, tg, b, wts, n, grids, st);
    else launch_rec_k<1>(s, g, fs, tg, b, wts, n, grids, st);
    if (b.tile_ev1) cudaEventRecord(b.tile_ev1, s);
    k_edge_fixup<T><<<152 * 2, 128, 0, s>>>(g, fs, in, b.edge_list, b.edge_count, grids, st);
    *launches += 5;
  }
}

void launch_paint32(cudaStream_t s, const Geom &g, const FieldSpec &fs, const TileGeo &tg, int deterministic,
                    int dtype, const void *x, const void *y, const void *z, const void *v, const void *w,
                    long long n, const GridPtrs &grids, const PaintBufs &b, DevStats *st, long long *launches) {
  if (dtype == CAPOW_F64) {
    PIn<double> in{(const double *)x, (const double *)y, (const double *)z, (const double *)v, (const double *)w};
    run_paint32<double>(s, g, fs, tg, deterministic, in, n, grids, b, st, launches);
  } else {
    PIn<float> in{(const float *)x, (const float *)y, (const float *)z, (const float *)v, (const float *)w};
    run_paint32<float>(s, g, fs, tg, deterministic, in, n, grids, b, st, launches);
  }
}
