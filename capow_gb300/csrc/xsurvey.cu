// The fused x axis + assign_survey_power of the FP32 survey estimator (src/main.c:781-967) for power-of-two NX: the
// columns along x of one FFT set, transformed and multiplied with the monopole field from shared memory, so that the
// x-transformed term grids never go to HBM.
#include <string.h>

#include "harm.cuh"
#include "xrow.cuh"

// Sums of a mode: P0, P2, P4 for the l = 0 pass, one otherwise.
CAPOW_HD constexpr int xs_sums(bool lz) { return lz ? 3 : 1; }

// One FFT set (l, m): blocks, columns and binning as in k_xrow_bin; the power forms are those of k_sv_assign. A lane takes
// kx and -kx together: h_lm(k^) is even or odd in kx (S.xodd).
//  LZ: the l = 0 pass, which writes the monopole fields F0 (and F0m), [kz][ky][kx] like the term grids, for the others.
//
// What bounds it: shared memory and the two block barriers between its phases, as in k_xrow_bin. 512^3, two slots, bins up
// to 0.62 of the Nyquist frequency: 0.150 ms a set (0.167 for l = 0) where the strided cuFFT pass along x and k_sv_assign
// took 0.60 + 0.24; with the y pass (0.20 against 0.30) 30.2 -> 18.0 ms for the 15 sets of a call.
template <int NF, bool IL, bool LZ, int LN>
__global__ void __launch_bounds__(xr_threads(LN), 2)
    k_xrow_survey(BinParams bp, BinTables t, XbinGeo xg, const float2 *g0, const float2 *g1, const float2 *g2,
                  const float2 *g3, SvSet S, double *bins) {
  constexpr int NS = NF * (IL ? 2 : 1);
  constexpr bool CROSS = NF == 2;
  constexpr int NA = xs_sums(LZ);
  constexpr int N = 1 << LN, HALF = N / 2, XR_THREADS = xr_threads(LN), KC = XR_THREADS / RowFft<LN>::T / NS;
  constexpr unsigned COLB = xr_col_bytes(LN, NS);
  extern __shared__ __align__(16) unsigned char smraw[];
  const int nk = bp.nk;
  const XrowSmem L = xrow_smem_layout(LN, NS, 1, NA, nk, xg.nbc);
  unsigned char *sd = smraw + L.sd;
  float2 *stw = (float2 *)(smraw + L.stw);
  float4 *sxt = (float4 *)(smraw + L.sxt);  // per kx >= 0: fx^2, deconvolution factor, interlace phase
  float *sfx = (float *)(smraw + L.sfx);    // per kx >= 0: fx
  float *sb = (float *)(smraw + L.sb);
  double *sbd = (double *)(smraw + L.sbd);
  XrCol *scol = (XrCol *)(smraw + L.scol);
  double *sE = (double *)(smraw + L.sE);
  float *sElo = (float *)(smraw + L.sElo);
  float *sEhi = (float *)(smraw + L.sEhi);
  __shared__ int s_next;
  const int nbins = NA * nk;
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
  float o[4] = {0.0f, 0.0f, 0.0f, 0.0f};            // painted values at the observer's cell, by slot
  if (LZ && S.origin)
    for (int q = 0; q < NS; q++) o[q] = S.a[q][S.oind];
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
      const unsigned char *D0 = sd + c * COLB, *D1 = D0 + KC * COLB;
      const int ic = min(i, HALF);
      const float4 xt = sxt[ic];
      const float s = xt.x + col.syz;
      const int b = xr_mode_bin(bp, t, sE, sElo, sEhi, col, i, s);
      const bool in = b >= 0 && b < nk;
      const bool kzero = i == 0 && col.j == 0 && col.kz == 0;
      const bool pair = i != 0 && i != HALF;  // kx = 0 and NX/2 have no mirror
      const long long f = (long long)blk * blk_elems + c * N;
      float acc[NA];
#pragma unroll
      for (int q = 0; q < NA; q++) acc[q] = 0.0f;
#pragma unroll
      for (int m = 0; m < 2; m++) {
        const int ii = m ? (N - ic) & (N - 1) : ic;
        const bool on = in && (m == 0 || pair);
        float2 F = make_float2(0.0f, 0.0f), Fm = F;
        if (!LZ && on) {
          F = S.F0[f + ii];
          if (CROSS) Fm = S.F0m[f + ii];
        }
        float2 X, M = make_float2(0.0f, 0.0f), Xi, Mi;
        if (NS == 4) {
          const float4 u = *(const float4 *)(D0 + 16 * ii), w = *(const float4 *)(D1 + 16 * ii);
          X = make_float2(u.x, u.y);
          M = make_float2(u.z, u.w);
          Xi = make_float2(w.x, w.y);
          Mi = make_float2(w.z, w.w);
        } else if (NS == 2) {
          const float4 u = *(const float4 *)(D0 + 16 * ii);
          X = make_float2(u.x, u.y);
          if (CROSS) M = make_float2(u.z, u.w);
          else Xi = make_float2(u.z, u.w);
        } else {
          X = *(const float2 *)(D0 + 8 * ii);
        }
        if (LZ && kzero) {  // the slots' exact DC values replace F(0)
          X = make_float2((float)S.dc[0], 0.0f);
          if (CROSS) M = make_float2((float)S.dc[1], 0.0f);
          if (IL) Xi = make_float2((float)S.dc[NF], 0.0f);
          if (IL && CROSS) Mi = make_float2((float)S.dc[NS - 1], 0.0f);
        }
        float2 e = make_float2(0.0f, 0.0f);
        if (IL) {
          e = cmulf(make_float2(xt.z, m ? -xt.w : xt.w), col.eyz);
          X = cfma(Xi, e, X);
          if (CROSS) M = cfma(Mi, e, M);
        }
        if (LZ) {
          if (on) {
            S.F0[f + ii] = X;
            if (CROSS) S.F0m[f + ii] = M;
          }
          const float p = CROSS ? X.x * M.y - X.y * M.x : X.x * X.x + X.y * X.y;
          float pc = CROSS || kzero ? p : 0.0f;  // enters P2 with -1/2 and P4 with 3/8
          if (S.origin && !kzero) {  // the observer cell's closed-form field (f_o + e f_o,interlaced) e^{-i k.r_o}
            const float2 ph = cmulf(S.ox[ii], cmulf(S.oy[col.j], S.oz[col.kz]));
            const float2 O = cmulf(IL ? make_float2(o[0] + o[NF] * e.x, o[NF] * e.y) : make_float2(o[0], 0.0f), ph);
            if (CROSS) {
              const float2 Om = cmulf(IL ? make_float2(o[1] + o[NS - 1] * e.x, o[NS - 1] * e.y) : make_float2(o[1], 0.0f), ph);
              pc += 0.5f * ((O.x * M.y - O.y * M.x) + (Om.x * X.y - Om.y * X.x));
            } else {
              pc += O.x * X.x + O.y * X.y;
            }
          }
          if (on) {
            acc[0] += p;
            acc[NA > 1 ? 1 : 0] += -0.5f * pc;
            acc[NA > 2 ? 2 : 0] += 0.375f * pc;
          }
        } else {
          float v;
          if (!CROSS) v = (S.l & 1) ? X.x * F.y - X.y * F.x : X.x * F.x + X.y * F.y;
          else if (S.l & 1) v = 0.5f * ((X.x * Fm.x + X.y * Fm.y) + (M.x * F.x + M.y * F.y));
          else v = 0.5f * ((X.x * Fm.y - X.y * Fm.x) + (M.x * F.y - M.y * F.x));
          if (on && !kzero) acc[0] += m && S.xodd ? -v : v;
        }
      }
      float gc = col.cyzn * xt.y;
      // NM on the kz = 0 plane: 1, except 2 at kx = NX/2 and, on ky = 0, at kx = 0 (src/main.c:422-429)
      if (col.kz == 0 && (i == HALF || (i == 0 && col.j == 0))) gc *= 2.0f;
      if (!LZ) {
        const float inv = kzero ? 0.0f : rsqrtf(s);
        gc *= S.coef * harm<float>(S.l, S.m, sfx[ic] * inv, t.fyf[col.j] * inv, t.fzf[col.kz] * inv);
      }
#pragma unroll
      for (int q = 0; q < NA; q++) acc[q] *= gc;
      xr_add_runs<NA>(acc, b, in, lane, sbw, nk);
    }
    blk = s_next;
    __syncthreads();  // the binning has read sd and scol
    if ((++nproc & 15) == 0) xr_flush(sb, sbd, nbins, xg.nbc);
  }
  __syncthreads();
  // CTA bins (FP64) -> global FP64 bins [5][nk]
  for (int c = threadIdx.x; c < nbins; c += XR_THREADS) {
    double v = sbd[c];
    for (int k = 0; k < xg.nbc; k++) v += (double)sb[c + k * nbins];
    if (v != 0.0) atomicAdd(&bins[(LZ ? 2 * (c / nk) : S.l) * nk + c % nk], v);
  }
}

bool xrow_survey_plan(const BinParams &bp, const BinTables &t, int nslot, XbinGeo &xg) {
  if (!xrow_geo(bp, t, nslot, xg)) return false;
  // (512 bins at most: three rows of FP32 and FP64 sums fit beside two copies)
  xg.nbc = 2;
  if (xrow_smem_layout(xg.log2n, nslot, 1, 3, bp.nk, 2).total > 112 * 1024) xg.nbc = 1;
  return xrow_smem_layout(xg.log2n, nslot, 1, 3, bp.nk, xg.nbc).total <= 220 * 1024;
}

template <int NF, bool IL, bool LZ, int LN>
static void launch_xs_n(cudaStream_t s, const BinParams &bp, const BinTables &t, const XbinGeo &xg, const float2 *u,
                        long long uslot, const SvSet &set, double *bins) {
  constexpr int NS = NF * (IL ? 2 : 1);
  const size_t smem = xrow_smem_layout(LN, NS, 1, xs_sums(LZ), bp.nk, xg.nbc).total;
  int grid = resident_ctas((const void *)k_xrow_survey<NF, IL, LZ, LN>, xr_threads(LN), smem, 64);
  if (grid > xg.nblocks) grid = xg.nblocks;
  k_xrow_survey<NF, IL, LZ, LN><<<grid, xr_threads(LN), smem, s>>>(bp, t, xg, u, u + uslot, u + 2 * uslot, u + 3 * uslot, set,
                                                                bins);
}

template <int NF, bool IL>
static void launch_xs_t(cudaStream_t s, const BinParams &bp, const BinTables &t, const XbinGeo &xg, const float2 *u,
                        long long uslot, const SvSet &set, double *bins) {
  switch (xg.log2n * 2 + (set.l == 0)) {
    case 10: return launch_xs_n<NF, IL, false, 5>(s, bp, t, xg, u, uslot, set, bins);
    case 11: return launch_xs_n<NF, IL, true, 5>(s, bp, t, xg, u, uslot, set, bins);
    case 12: return launch_xs_n<NF, IL, false, 6>(s, bp, t, xg, u, uslot, set, bins);
    case 13: return launch_xs_n<NF, IL, true, 6>(s, bp, t, xg, u, uslot, set, bins);
    case 14: return launch_xs_n<NF, IL, false, 7>(s, bp, t, xg, u, uslot, set, bins);
    case 15: return launch_xs_n<NF, IL, true, 7>(s, bp, t, xg, u, uslot, set, bins);
    case 16: return launch_xs_n<NF, IL, false, 8>(s, bp, t, xg, u, uslot, set, bins);
    case 17: return launch_xs_n<NF, IL, true, 8>(s, bp, t, xg, u, uslot, set, bins);
    case 18: return launch_xs_n<NF, IL, false, 9>(s, bp, t, xg, u, uslot, set, bins);
    case 19: return launch_xs_n<NF, IL, true, 9>(s, bp, t, xg, u, uslot, set, bins);
    case 20: return launch_xs_n<NF, IL, false, 10>(s, bp, t, xg, u, uslot, set, bins);
    default: return launch_xs_n<NF, IL, true, 10>(s, bp, t, xg, u, uslot, set, bins);
  }
}

void launch_xrow_survey(cudaStream_t s, const BinParams &bp, const BinTables &t, const XbinGeo &xg, int nf, const float2 *u,
                        long long uslot, SvSet set, double *bins) {
  // h_lm of harm.cuh that change sign with x
  static const unsigned odd[5] = {0, 0x1, 0x5, 0x19, 0x99};
  set.xodd = (int)((odd[set.l] >> set.m) & 1u);
  if (nf == 2) {
    if (bp.interlace) launch_xs_t<2, true>(s, bp, t, xg, u, uslot, set, bins);
    else launch_xs_t<2, false>(s, bp, t, xg, u, uslot, set, bins);
  } else {
    if (bp.interlace) launch_xs_t<1, true>(s, bp, t, xg, u, uslot, set, bins);
    else launch_xs_t<1, false>(s, bp, t, xg, u, uslot, set, bins);
  }
}
