// The y axis and the fused x axis + binning of the power stage for power-of-two NX, NY and NZ (FP32).
//
// k_zfft (bin.cu) leaves [NX][NZ/2+1][NY] complex per slot (z transformed, transposed). Here:
//  * k_yfft transforms the rows along y and stores them transposed once more, [kz][ky][NX] per slot, so that the
//    columns along x of the next pass are contiguous;
//  * k_xrow_bin (xrow.cuh) transforms a block's columns along x and bins the modes from shared memory (the
//    binning of k_bin, src/main.c:302-468), so that the x-transformed grids never go to HBM.
// Columns and rows beyond the top k-bin edge are neither written nor read.
#include <cuda_runtime.h>
#include <math.h>
#include <string.h>

#include "bin.cuh"
#include "fft_dev.cuh"
#include "launch.cuh"
#include "xrow.cuh"

// ------------------------------------------------------------------------------------------- y axis
struct YfftGeo {
  int nx, nzc;              // planes of this call, kz rows per plane of the input
  int x0, nx_out;           // first plane's place in the output, NX of the output
  int kzmax;
  int ns;
  long long in_slot, out_slot;
  float top, fz_step, inv_fy;  // just above the top bin edge in |f|^2; f of kz = 1; 1 / f of ky = 1
};

// Threads of a CTA: 16 rows, so that 128 contiguous bytes are written per ky (512: 64 registers and two CTAs per SM;
// 1024: 128 registers and one).
template <int LOGN>
struct YfftShape {
  typedef RowFft<LOGN> F;
  static constexpr int THREADS = LOGN >= 9 ? 512 : 256;
  static constexpr int RP = THREADS / F::T;
  static constexpr int PITCH = (F::BUF > F::N ? F::BUF : F::N) | 1;  // odd: lanes across rows meet no bank conflict
  static constexpr unsigned SMEM = 8u * (RP * PITCH + F::N);
};

// Blocks of RP planes at one kz that follow each other in the block order: 4 x 128 bytes of the same output rows are
// written at about the same time (1 and 8 blocks were slower).
constexpr int YF_XG = 4;

// A CTA transforms the rows (x, kz) of RP consecutive x at one kz (T lanes a row, RowFft): rows straight from
// HBM into registers, one exchange within the warp, then through shared memory to RP * 8 contiguous bytes per ky.
// Rows kz > kzmax and frequencies beyond the top bin edge are left out.
// What bounds it: HBM, at 5.3 TB/s of its reads and writes (512^3, four slots: 0.73 ms for 2.2 GB read and the 1.7 GB
// below the top k-bin written; cuFFT's C2C took 0.60 ms in place, but left the columns along x 4 KB apart, for a binning
// pass of 1.47 ms that now takes 0.76).
template <int LOGN>
__global__ void __launch_bounds__(YfftShape<LOGN>::THREADS, LOGN == 10 ? 1 : (LOGN == 9 ? 2 : 4))
    k_yfft(YfftGeo yg, BinTables t, const float2 *in, float2 *out) {
  typedef YfftShape<LOGN> S;
  typedef typename S::F F;
  constexpr int N = F::N, T = F::T, R1 = F::R1, RP = S::RP;
  extern __shared__ __align__(16) unsigned char smy[];
  float2 *sd = (float2 *)smy;
  float2 *stw = sd + RP * S::PITCH;
  F::load_twiddles(stw, t.twy);
  const int tl = threadIdx.x % T, row = threadIdx.x / T;
  const int orow = threadIdx.x % RP, ok = threadIdx.x / RP;  // output phase: row, first ky
  float2 *srow = sd + row * S::PITCH;
  // order of the blocks of RP planes: (slot, group of YF_XG blocks, kz, block)
  const int nxb = (yg.nx + RP - 1) / RP, nxg = (nxb + YF_XG - 1) / YF_XG, nkz = yg.kzmax + 1;
  const long long nblk = (long long)yg.ns * nkz * nxg * YF_XG;
  for (long long b = blockIdx.x; b < nblk; b += gridDim.x) {
    const long long r = b / YF_XG, r2 = r / nkz;
    const int kz = (int)(r - r2 * nkz), sl = (int)(r2 / nxg), xb = (int)(r2 - (long long)sl * nxg) * YF_XG + (int)(b - r * YF_XG);
    if (xb >= nxb) continue;
    const int x = min(xb * RP + row, yg.nx - 1), ox = xb * RP + orow;
    const float2 *src = in + sl * yg.in_slot + ((long long)x * yg.nzc + kz) * N + tl;
    float2 v[R1];
#pragma unroll
    for (int q = 0; q < R1; q++) v[q] = __ldcs(src + T * q);
    __syncthreads();  // twiddles written; the previous rows' output has read sd
    F::run(v, srow, stw, tl);
#pragma unroll
    for (int j = 0; j < R1; j++) srow[F::freq(tl, j)] = v[j];
    __syncthreads();
    const float fz = yg.fz_step * (float)kz, rest = yg.top - fz * fz;
    // |ky| beyond kym has fy^2 + fz^2 above the top edge (two rows to spare)
    const int kym = rest > 0.0f ? min(N / 2, (int)(sqrtf(rest) * yg.inv_fy) + 2) : 1;
    if (ox < yg.nx) {
      const float2 *zr = sd + orow * S::PITCH;
      float2 *dst = out + sl * yg.out_slot + (long long)kz * N * yg.nx_out + yg.x0 + ox;
#pragma unroll 4
      for (int ky = ok; ky < N; ky += T)
        if (min(ky, N - ky) <= kym) dst[(long long)ky * yg.nx_out] = zr[ky];
    }
  }
}

bool yfft_supported(const BinParams &bp, const BinTables &t) {
  return t.twy && bp.ny >= 16 && bp.ny <= 1024 && (bp.ny & (bp.ny - 1)) == 0;
}

template <int LOGN>
static void launch_yfft_t(cudaStream_t s, const YfftGeo &yg, const BinTables &t, const float2 *in, float2 *out) {
  typedef YfftShape<LOGN> S;
  const size_t smem = S::SMEM;
  const int resident = resident_ctas((const void *)k_yfft<LOGN>, S::THREADS, smem);
  const long long nblk = (long long)yg.ns * (yg.kzmax + 1) * ((yg.nx + S::RP * YF_XG - 1) / (S::RP * YF_XG)) * YF_XG;
  long long grid = resident;
  if (grid > nblk) grid = nblk;
  k_yfft<LOGN><<<(unsigned)grid, S::THREADS, smem, s>>>(yg, t, in, out);
}

void launch_yfft(cudaStream_t s, const BinParams &bp, const BinTables &t, int nslot, int x0, int nx,
                 const float2 *in, long long in_slot, float2 *out, long long out_slot) {
  YfftGeo yg;
  memset(&yg, 0, sizeof yg);
  yg.nx = nx;
  yg.nzc = bp.nzc;
  yg.x0 = x0;
  yg.nx_out = bp.nx;
  yg.kzmax = bp.kzmax;
  yg.ns = nslot;
  yg.in_slot = in_slot;
  yg.out_slot = out_slot;
  yg.top = bp.ftop2 * 1.0002f;
  yg.fz_step = bp.fz_step;
  yg.inv_fy = 1.0f / bp.fy_step;
  switch (bp.ny) {
    case 16: launch_yfft_t<4>(s, yg, t, in, out); break;
    case 32: launch_yfft_t<5>(s, yg, t, in, out); break;
    case 64: launch_yfft_t<6>(s, yg, t, in, out); break;
    case 128: launch_yfft_t<7>(s, yg, t, in, out); break;
    case 256: launch_yfft_t<8>(s, yg, t, in, out); break;
    case 512: launch_yfft_t<9>(s, yg, t, in, out); break;
    default: launch_yfft_t<10>(s, yg, t, in, out); break;
  }
}

// ---------------------------------------------------------------------------------- x axis + binning
bool xrow_geo(const BinParams &bp, const BinTables &t, int nslot, XbinGeo &xg) {
  const int n = bp.nx;
  if (n < 32 || n > 1024 || (n & (n - 1)) != 0 || bp.out2d || !yfft_supported(bp, t) || nslot == 3) return false;
  memset(&xg, 0, sizeof xg);
  while ((1 << xg.log2n) < n) xg.log2n++;
  xg.ncol = xr_threads(xg.log2n) / (int)xr_lanes(xg.log2n);
  xg.kc = xg.ncol / nslot;
  if (xg.kc > bp.ny) return false;
  while ((1 << xg.log2ncol) < xg.ncol) xg.log2ncol++;
  while ((1 << xg.log2kc) < xg.kc) xg.log2kc++;
  xg.tr = 2;
  xg.n_outer = bp.kzmax + 1;
  xg.n_inner = bp.ny;
  xg.nkb = bp.ny >> xg.log2kc;
  xg.nblocks = xg.n_outer * xg.nkb;
  return true;
}

bool xrow_plan(const BinParams &bp, const BinTables &t, int nslot, XbinGeo &xg) {
  if (!xrow_geo(bp, t, nslot, xg)) return false;
  const int np = xrow_products(bp), nl = xrow_multipoles(bp);
  // two copies of the block bins while two CTAs fit an SM, else one
  xg.nbc = 2;
  if (xrow_smem_layout(xg.log2n, nslot, np, nl, bp.nk, 2).total > 112 * 1024) xg.nbc = 1;
  return xrow_smem_layout(xg.log2n, nslot, np, nl, bp.nk, xg.nbc).total <= 220 * 1024;
}

void launch_xrow(cudaStream_t s, const BinParams &bp, const BinTables &t, const XbinGeo &xg, void *const slots[4],
                 const double *dcv, double *bins, long long *launches) {
  if (bp.interlace) {
    if (bp.nfields == 2) launch_xrow_f2i(s, bp, t, xg, slots, dcv, bins);
    else launch_xrow_f1i(s, bp, t, xg, slots, dcv, bins);
  } else {
    launch_xrow_plain(s, bp, t, xg, slots, dcv, bins);
  }
  (*launches)++;
}
