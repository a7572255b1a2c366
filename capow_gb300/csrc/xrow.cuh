// The fused x axis + binning kernel of the blocked path (xbin.cu) and its launch templates; the instances are
// spread over xrow_*.cu.
#pragma once
#include <cuda_runtime.h>

#include "bin.cuh"
#include "fft_dev.cuh"
#include "launch.cuh"

#define FULL_MASK 0xffffffffu

// Products and multipoles that the instance for bp accumulates: |A|^2, Im A*B, |B|^2 (dd + dp + pp) or all four; even
// multipoles or all.
inline bool xrow_full(const BinParams &bp) { return bp.odd || !bp.interlace || (bp.nfields == 2 && (bp.pmask & ~0xD) != 0); }
inline int xrow_products(const BinParams &bp) { return bp.nfields == 1 ? 1 : (xrow_full(bp) ? 4 : 3); }
inline int xrow_multipoles(const BinParams &bp) { return xrow_full(bp) ? 5 : 3; }

CAPOW_HD constexpr unsigned xr_align(unsigned x) { return (x + 15u) & ~15u; }

// The binning layout of a block: per ky column the frequencies in natural order, its slots in 16-byte pairs (A, B),
// (A, B interlaced) or (A, A interlaced), so that a mode is one or two wide loads and neighbouring modes lie on
// other banks. Bytes of one column of one pair array (a pad spreads the columns over the banks).
CAPOW_HD constexpr unsigned xr_col_bytes(int log2n, int ns) { return (ns == 1 ? 8u : 16u) * (1u << log2n) + 16u; }

// Values of the row buffer that RowFft exchanges through, and lanes per row (fft_dev.cuh).
CAPOW_HD constexpr unsigned xr_lanes(int log2n) { return log2n >= 9 ? 32u : (log2n == 8 ? 16u : (log2n == 5 ? 4u : 8u)); }
// Threads of a CTA (two CTAs per SM): 64 registers a thread for 8 or 16 values, 128 for the 32 of NX = 1024; half as
// many for NX = 32, whose grids have few blocks.
CAPOW_HD constexpr int xr_threads(int log2n) { return log2n == 10 || log2n == 5 ? 256 : 512; }
CAPOW_HD constexpr unsigned xr_rowbuf(int log2n) { return ((1u << log2n) / xr_lanes(log2n)) * (xr_lanes(log2n) + 1u); }

// Per-column quantities of the block being binned: everything of a mode that does not depend on kx.
struct XrCol {
  float syz;    // fy^2 + fz^2 (FP32)
  float cyzn;   // y, z deconvolution factors, x 0.25 when interlaced, x 2 off the kz = 0 plane (NM)
  float flos;   // mu numerator when the LOS is y or z (fy or fz)
  int j;        // ky index
  float2 eyz;   // y, z interlace phase
  int kz;
  int r;        // |kx| index beyond which no mode reaches the top bin edge (-1: none does)
};

struct XrowSmem {
  unsigned sd, stw, sxt, sfx, sb, sbd, scol, sE, sElo, sEhi, total;
};

CAPOW_HD XrowSmem xrow_smem_layout(int log2n, int ns, int npu, int nl, int nk, int nbc) {
  const unsigned n = 1u << log2n, ncol = (unsigned)xr_threads(log2n) / xr_lanes(log2n), kc = ncol / (unsigned)ns;
  XrowSmem L;
  unsigned o = 0;
  const unsigned a = 8u * ncol * xr_rowbuf(log2n), f = (ns == 4 ? 2u : 1u) * kc * xr_col_bytes(log2n, ns);
  L.sd = o;    o = xr_align(o + (a > f ? a : f));
  L.stw = o;   o = xr_align(o + 8u * n);
  L.sxt = o;   o = xr_align(o + 16u * (n / 2 + 1));
  L.sfx = o;   o = xr_align(o + 4u * (n / 2 + 1));
  L.sb = o;    o = xr_align(o + 4u * npu * nl * nk * nbc);
  L.sbd = o;   o = xr_align(o + 8u * npu * nl * nk);
  L.scol = o;  o = xr_align(o + (unsigned)sizeof(XrCol) * kc);
  L.sE = o;    o = xr_align(o + 8u * (nk + 3));
  L.sElo = o;  o = xr_align(o + 4u * (nk + 3));
  L.sEhi = o;  o = xr_align(o + 4u * (nk + 3));
  L.total = o;
  return L;
}

// c + a b
__device__ __forceinline__ float2 cfma(float2 a, float2 b, float2 c) {
  return make_float2(fmaf(a.x, b.x, fmaf(-a.y, b.y, c.x)), fmaf(a.x, b.y, fmaf(a.y, b.x, c.y)));
}

// The columns of a block along x: T lanes of a warp transform a column in registers (RowFft: one exchange, no block
// barrier) and, when the whole block is through its exchange, write the binning layout.
template <int LN, int NS>
__device__ __forceinline__ void xr_columns(const float2 *g0, const float2 *g1, const float2 *g2, const float2 *g3,
                                           long long off, unsigned char *sd, const float2 *stw) {
  typedef RowFft<LN> F;
  constexpr int N = F::N, T = F::T, R1 = F::R1, KC = xr_threads(LN) / T / NS;
  const int t = threadIdx.x % T, col = threadIdx.x / T, sl = col / KC, c = col - sl * KC;
  const float2 *g = NS == 1 ? g0 : (NS == 2 ? (sl ? g1 : g0) : (sl < 2 ? (sl ? g1 : g0) : (sl == 2 ? g2 : g3)));
  const float2 *src = g + off + c * N + t;
  float2 v[R1];
#pragma unroll
  for (int q = 0; q < R1; q++) v[q] = __ldcs(src + q * T);
  F::run(v, (float2 *)sd + col * F::BUF, stw, t);
  __syncthreads();
  constexpr unsigned COLB = xr_col_bytes(LN, NS);
  unsigned char *dst = sd + c * COLB + (NS == 4 ? (sl >> 1) * (KC * COLB) + 8 * (sl & 1) : (NS == 2 ? 8 * sl : 0));
#pragma unroll
  for (int j = 0; j < R1; j++) *(float2 *)(dst + F::freq(t, j) * (NS == 1 ? 8 : 16)) = v[j];
  __syncthreads();
}

// The k-bin of the mode (i, column) with |f|^2 = s (src/main.c:355, 369-375); nk beyond the column's last |kx|. sE,
// sElo, sEhi: the edges in shared memory.
__device__ __forceinline__ int xr_mode_bin(const BinParams &bp, const BinTables &t, const double *sE, const float *sElo,
                                           const float *sEhi, const XrCol &col, int i, float s) {
  const int nk = bp.nk;
  int b = nk;
  if (i <= col.r) {
    if (!bp.lg) {
      const float v = (s > 0.0f ? s * rsqrtf(s) : 0.0f) * bp.kscale + bp.koff;
      b = v < 0.0f ? -1 : (v >= (float)nk ? nk : (int)v);
    } else {
      int a = 0, z = nk + 2;  // sElo[a] <= s < sElo[z]
      while (z - a > 1) {
        const int mid = (a + z) >> 1;
        if (sElo[mid] <= s) a = mid;
        else z = mid;
      }
      b = a - 1;
    }
    while (b < nk && s >= sElo[b + 2]) b++;
    while (b > -1 && s < sEhi[b + 1]) b--;
    if (!(s >= sElo[b + 1] && s < sEhi[b + 2]))  // within a few ulps of an edge: the exact FP64 s decides
      b = exact_bin(sE, nk, __dadd_rn(__dadd_rn(t.fx2d[i], t.fy2d[col.j]), t.fz2d[col.kz]), b);
  }
  return b;
}

// Add each lane's NA sums to row q of dst ([NA][nk]) at its bin b (in: b is a bin; lanes of one bin are a run): the sum of
// a run is gathered to its first lane, which adds it.
template <int NA>
__device__ __forceinline__ void xr_add_runs(float (&acc)[NA], int b, bool in, int lane, float *dst, int nk) {
  const int prev = __shfl_up_sync(FULL_MASK, b, 1);
  for (int o = 1; o < 32; o <<= 1) {
    const int b2 = __shfl_down_sync(FULL_MASK, b, o);
    const bool same = lane + o < 32 && b2 == b;
    if (!__any_sync(FULL_MASK, same && in)) break;
#pragma unroll
    for (int q = 0; q < NA; q++) {
      const float v = __shfl_down_sync(FULL_MASK, acc[q], o);
      if (same) acc[q] += v;
    }
  }
  if (in && (lane == 0 || prev != b)) {
#pragma unroll
    for (int q = 0; q < NA; q++) atomicAdd(&dst[q * nk + b], acc[q]);
  }
}

// First block at or after blk (in steps of the grid) that reaches below the top edge: fz^2 grows with kz; fy^2 rises to
// ky = NY/2 and falls after it, so over a run of KC ky it is smallest at an end.
template <int KC>
__device__ __forceinline__ int xr_next_live(const BinTables &t, const XbinGeo &xg, float top, int blk) {
  for (; blk < xg.nblocks; blk += gridDim.x) {
    const int kz = blk / xg.nkb, j0 = (blk - kz * xg.nkb) * KC;
    if (!(t.fz2f[kz] + fminf(t.fy2f[j0], t.fy2f[j0 + KC - 1]) > top)) break;
  }
  return blk;
}

// The kx-independent quantities of the column (ky j, kz) (src/main.c:335-389 for the y, z factors).
template <bool IL>
__device__ __forceinline__ XrCol xr_column(const BinParams &bp, const BinTables &t, int j, int kz, float top, float inv_fx) {
  XrCol col;
  col.syz = t.fy2f[j] + t.fz2f[kz];
  float cyz = t.cyf[j] * t.czf[kz];
  if (IL) cyz *= 0.25f;
  col.cyzn = kz != 0 ? 2.0f * cyz : cyz;  // Hermitian multiplicity off the kz = 0 plane (:422-429)
  col.eyz = IL ? cmulf(t.eyf[j], t.ezf[kz]) : make_float2(0.0f, 0.0f);
  col.flos = bp.los == 2 ? t.fyf[j] : t.fzf[kz];
  col.j = j;
  col.kz = kz;
  const float rest = top - col.syz;
  col.r = rest > 0.0f ? min(bp.nx / 2, (int)(sqrtf(rest) * inv_fx) + 1) : -1;
  return col;
}

// FP32 block bins (nbc copies) to the CTA's FP64 bins.
__device__ __forceinline__ void xr_flush(float *sb, double *sbd, int nbins, int nbc) {
  for (int c = threadIdx.x; c < nbins; c += blockDim.x) {
    float v = 0.0f;
    for (int k = 0; k < nbc; k++) {
      v += sb[c + k * nbins];
      sb[c + k * nbins] = 0.0f;
    }
    sbd[c] += (double)v;
  }
}

// The fused pass. Blocks of kc columns of every slot (16 columns of 512 values: 64 KB, two CTAs per SM, so that one
// computes while the other waits for its block, whose lines an L2 prefetch of contiguous runs has brought near).
//
// Binning: a warp takes 32 consecutive kx >= 0 of one column, a lane one kx and -kx together (their bin, weights and
// Legendre factors agree). Along kx the bin is monotone, so each bin is a run of lanes: the sums of a run are
// gathered to its first lane by shuffles (as many steps as the longest run of the warp needs), which adds them
// to the block bins (shared-memory float additions, compare-and-swap loops). That is one addition per bin, column
// and warp, from lanes that never meet on an address, by warps with equal work; runs of 4 kx per thread used to
// flush every second mode, at addresses that met.
// FP32 block bins go to the CTA's FP64 bins every 16 blocks (a few hundred modes per bin), then to global.
//
// What bounds it: shared memory (63% of its cycles: the column exchange, the layout, the modes' 16-byte reads) and issue
// (48%) together, with the two block barriers between the phases. 512^3, four slots, dd + dp + pp: 0.76 ms (1.7 GB read,
// 443M warp instructions; HBM alone would take 0.25 ms) against 1.47 ms of the strided x pass of bin.cu; 256^3 0.11
// against 0.18 ms. A warp per (bin range, columns), gathering its bins' kx, took 1.19 ms: bins near the Nyquist edge hold
// most modes, and the warps that owned them kept the others waiting.
// PM: the products accumulated (bit q: |A|^2, Re A*B, Im A*B, |B|^2): a superset of what the spectra read. LN: log2 NX.
template <int NF, bool IL, bool ODD, int PM, int LN>
__global__ void __launch_bounds__(xr_threads(LN), 2)
    k_xrow_bin(BinParams bp, BinTables t, XbinGeo xg, const float2 *g0, const float2 *g1, const float2 *g2,
               const float2 *g3, const double *dcv, double *bins) {
  static_assert(RowFft<LN>::T == (int)xr_lanes(LN) && RowFft<LN>::BUF == (int)xr_rowbuf(LN), "row transform");
  constexpr int NS = NF * (IL ? 2 : 1);
  constexpr int NPU = NF == 1 ? 1 : ((PM & 1) + ((PM >> 1) & 1) + ((PM >> 2) & 1) + ((PM >> 3) & 1));
  constexpr int NL = ODD ? 5 : 3;  // stored multipoles: l = 0, 2, 4 (+ 1, 3)
  constexpr int N = 1 << LN, HALF = N / 2, XR_THREADS = xr_threads(LN), KC = XR_THREADS / RowFft<LN>::T / NS;
  constexpr unsigned COLB = xr_col_bytes(LN, NS);
  extern __shared__ __align__(16) unsigned char smraw[];
  const int nk = bp.nk;
  const XrowSmem L = xrow_smem_layout(LN, NS, NPU, NL, nk, xg.nbc);
  unsigned char *sd = smraw + L.sd;
  float2 *stw = (float2 *)(smraw + L.stw);
  float4 *sxt = (float4 *)(smraw + L.sxt);  // per kx >= 0: fx^2, deconvolution factor, interlace phase
  float *sfx = (float *)(smraw + L.sfx);    // per kx >= 0: fx (the mu numerator when LOS = x)
  float *sb = (float *)(smraw + L.sb);      // block bins, FP32, xg.nbc copies
  double *sbd = (double *)(smraw + L.sbd);  // the CTA's bins, FP64
  XrCol *scol = (XrCol *)(smraw + L.scol);
  double *sE = (double *)(smraw + L.sE);
  float *sElo = (float *)(smraw + L.sElo);
  float *sEhi = (float *)(smraw + L.sEhi);
  __shared__ int s_next;
  const int nbins = NPU * NL * nk;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int c = threadIdx.x; c < nbins * xg.nbc; c += XR_THREADS) sb[c] = 0.0f;
  for (int c = threadIdx.x; c < nbins; c += XR_THREADS) sbd[c] = 0.0;
  for (int c = threadIdx.x; c < nk + 3; c += XR_THREADS) {
    sE[c] = t.E[c];
    sElo[c] = t.Elo[c];
    sEhi[c] = t.Ehi[c];
  }
  for (int i = threadIdx.x; i <= HALF; i += XR_THREADS) {
    const float2 e = IL ? t.exf[i] : make_float2(0.0f, 0.0f);
    sxt[i] = make_float4(t.fx2f[i], t.cxf[i], e.x, e.y);
    sfx[i] = t.fxf[i];
  }
  RowFft<LN>::load_twiddles(stw, t.twx);
  const float topf32 = (float)t.E[nk + 1] * 1.0001f;
  const float inv_fx = 1.0f / bp.fx_step;
  const long long blk_elems = (long long)N * KC;
  float *sbw = sb + (warp & (xg.nbc - 1)) * nbins;  // this warp's copy
  int nproc = 0;
  if (threadIdx.x == 0) s_next = xr_next_live<KC>(t, xg, topf32, blockIdx.x);
  __syncthreads();
  int blk = s_next;
  __syncthreads();  // s_next is read before the loop writes it again
  while (blk < xg.nblocks) {
    const int kz = blk / xg.nkb, j0 = (blk - kz * xg.nkb) * KC;
    if (warp == XR_THREADS / 32 - 1) {  // the next block (read after the barriers below), and its runs towards L2
      const int nxt = xr_next_live<KC>(t, xg, topf32, blk + gridDim.x);
      if (lane == 0) s_next = nxt;
      if (lane < NS && nxt < xg.nblocks) {
        const float2 *q = (lane == 0 ? g0 : (lane == 1 ? g1 : (lane == 2 ? g2 : g3))) + (long long)nxt * blk_elems;
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(q), "r"((unsigned)(blk_elems * 8)) : "memory");
      }
    }
    if (threadIdx.x < KC) scol[threadIdx.x] = xr_column<IL>(bp, t, j0 + threadIdx.x, kz, sElo[nk + 1], inv_fx);
    xr_columns<LN, NS>(g0, g1, g2, g3, (long long)blk * blk_elems, sd, stw);
    constexpr int NJ = (HALF + 32) / 32;  // warps' worth of kx = 0 .. NX/2
    for (int task = warp; task < KC * NJ; task += XR_THREADS / 32) {
      const int c = task % KC, i = task / KC * 32 + lane;
      const XrCol col = scol[c];
      if (i - lane > col.r) continue;
      const unsigned char *F0 = sd + c * COLB, *F1 = F0 + KC * COLB;
      const int ic = min(i, HALF);
      const float4 xt = sxt[ic];
      const float s = xt.x + col.syz;
      const int b = xr_mode_bin(bp, t, sE, sElo, sEhi, col, i, s);
      const bool in = b >= 0 && b < nk;
      float acc[NPU * NL];
      {
        const bool pair = i != 0 && i != HALF;  // kx = 0 and NX/2 have no mirror
        float Pe[NPU], Po[NPU];  // products summed over the pair, and with the mirror's sign of mu
#pragma unroll
        for (int m = 0; m < 2; m++) {
          const int ii = m ? (N - ic) & (N - 1) : ic;  // (the single modes read themselves again)
          float2 A, B = make_float2(0.0f, 0.0f), Ai, Bi;
          if (NS == 4) {
            const float4 u = *(const float4 *)(F0 + 16 * ii), w = *(const float4 *)(F1 + 16 * ii);
            A = make_float2(u.x, u.y);
            B = make_float2(u.z, u.w);
            Ai = make_float2(w.x, w.y);
            Bi = make_float2(w.z, w.w);
          } else if (NS == 2) {
            const float4 u = *(const float4 *)(F0 + 16 * ii);
            A = make_float2(u.x, u.y);
            if (NF == 2) B = make_float2(u.z, u.w);
            else Ai = make_float2(u.z, u.w);
          } else {
            A = *(const float2 *)(F0 + 8 * ii);
          }
          if (i == 0 && col.j == 0 && col.kz == 0) {  // the slots' exact DC values replace F(0)
            A = make_float2((float)dcv[0], 0.0f);
            if (NF == 2) B = make_float2((float)dcv[1], 0.0f);
            if (IL) Ai = make_float2((float)dcv[NF], 0.0f);
            if (IL && NF == 2) Bi = make_float2((float)dcv[NS - 1], 0.0f);
          }
          if (IL) {
            const float2 e = cmulf(make_float2(xt.z, m ? -xt.w : xt.w), col.eyz);
            A = cfma(Ai, e, A);
            if (NF == 2) B = cfma(Bi, e, B);
          }
          float P[4];
          P[0] = A.x * A.x + A.y * A.y;
          if (NF == 2) {
            P[1] = A.x * B.x + A.y * B.y;
            P[2] = A.x * B.y - A.y * B.x;
            P[3] = B.x * B.x + B.y * B.y;
          }
          int k = 0;
#pragma unroll
          for (int q = 0; q < 4; q++)
            if (NF == 1 ? q == 0 : ((PM >> q) & 1)) {
              if (m == 0) {
                Pe[k] = P[q];
                if (ODD) Po[k] = P[q];
              } else {
                const float p = pair ? P[q] : 0.0f;
                Pe[k] += p;
                if (ODD) Po[k] += bp.los == 1 ? -p : p;
              }
              k++;
            }
        }
        float gc = col.cyzn * xt.y;
        // NM on the kz = 0 plane: 1, except 2 at kx = NX/2 and, on ky = 0, at kx = 0 (src/main.c:422-429)
        if (col.kz == 0 && (i == HALF || (i == 0 && col.j == 0))) gc *= 2.0f;
        const float fl = bp.los == 1 ? sfx[ic] : col.flos;
        const float mu = s > 0.0f ? fl * rsqrtf(s) : 0.0f;
        const float mu2 = mu * mu;
        const float L2 = 1.5f * mu2 - 0.5f;
        const float L4 = (4.375f * mu2 - 3.75f) * mu2 + 0.375f;
#pragma unroll
        for (int q = 0; q < NPU; q++) {
          const float p = in ? Pe[q] * gc : 0.0f;  // (columns beyond the top edge hold no values)
          acc[q * NL] = p;
          acc[q * NL + 1] = p * L2;
          acc[q * NL + 2] = p * L4;
          if (ODD) {
            const float o = in ? Po[q] * gc : 0.0f;
            acc[q * NL + NL - 2] = o * mu;
            acc[q * NL + NL - 1] = o * ((2.5f * mu2 - 1.5f) * mu);
          }
        }
      }
      xr_add_runs<NPU * NL>(acc, b, in, lane, sbw, nk);
    }
    blk = s_next;
    __syncthreads();  // the binning has read sd and scol
    if ((++nproc & 15) == 0) xr_flush(sb, sbd, nbins, xg.nbc);
  }
  __syncthreads();
  // CTA bins (FP64) -> global FP64 bins [product][5][nk]; stored product and multipole index -> q, l
  for (int c = threadIdx.x; c < nbins; c += XR_THREADS) {
    double v = sbd[c];
    for (int k = 0; k < xg.nbc; k++) v += (double)sb[c + k * nbins];
    if (v == 0.0) continue;
    const int b = c % nk, ql = c / nk, qu = ql / NL, li = ql - qu * NL;
    int q = 0;
    if (NF == 2)
      for (int left = qu; q < 4; q++)
        if ((PM >> q) & 1)
          if (left-- == 0) break;
    const int l = li == 0 ? 0 : (li == 1 ? 2 : (li == 2 ? 4 : (li == 3 ? 1 : 3)));
    atomicAdd(&bins[(q * 5 + l) * nk + b], v);
  }
}

template <int NF, bool IL, bool ODD, int PM, int LN>
static void launch_xrow_n(cudaStream_t s, const BinParams &bp, const BinTables &t, const XbinGeo &xg,
                          void *const slots[4], const double *dcv, double *bins) {
  constexpr int NS = NF * (IL ? 2 : 1);
  const size_t smem = xrow_smem_layout(LN, NS, xrow_products(bp), xrow_multipoles(bp), bp.nk, xg.nbc).total;
  int grid = resident_ctas((const void *)k_xrow_bin<NF, IL, ODD, PM, LN>, xr_threads(LN), smem, 64);
  if (grid > xg.nblocks) grid = xg.nblocks;
  k_xrow_bin<NF, IL, ODD, PM, LN><<<grid, xr_threads(LN), smem, s>>>(bp, t, xg, (const float2 *)slots[0],
                                                                 (const float2 *)slots[1], (const float2 *)slots[2],
                                                                 (const float2 *)slots[3], dcv, bins);
}

template <int NF, bool IL, bool ODD, int PM>
static void launch_xrow_t(cudaStream_t s, const BinParams &bp, const BinTables &t, const XbinGeo &xg,
                          void *const slots[4], const double *dcv, double *bins) {
  switch (xg.log2n) {
    case 5: return launch_xrow_n<NF, IL, ODD, PM, 5>(s, bp, t, xg, slots, dcv, bins);
    case 6: return launch_xrow_n<NF, IL, ODD, PM, 6>(s, bp, t, xg, slots, dcv, bins);
    case 7: return launch_xrow_n<NF, IL, ODD, PM, 7>(s, bp, t, xg, slots, dcv, bins);
    case 8: return launch_xrow_n<NF, IL, ODD, PM, 8>(s, bp, t, xg, slots, dcv, bins);
    case 9: return launch_xrow_n<NF, IL, ODD, PM, 9>(s, bp, t, xg, slots, dcv, bins);
    default: return launch_xrow_n<NF, IL, ODD, PM, 10>(s, bp, t, xg, slots, dcv, bins);
  }
}

// The instances: two fields interlaced, one field interlaced, not interlaced.
void launch_xrow_f2i(cudaStream_t s, const BinParams &bp, const BinTables &t, const XbinGeo &xg, void *const slots[4],
                     const double *dcv, double *bins);
void launch_xrow_f1i(cudaStream_t s, const BinParams &bp, const BinTables &t, const XbinGeo &xg, void *const slots[4],
                     const double *dcv, double *bins);
void launch_xrow_plain(cudaStream_t s, const BinParams &bp, const BinTables &t, const XbinGeo &xg, void *const slots[4],
                       const double *dcv, double *bins);
