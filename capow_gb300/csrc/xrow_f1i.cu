// Instances of k_xrow_bin: one field, interlaced: even multipoles, or all.
#include "xrow.cuh"

void launch_xrow_f1i(cudaStream_t s, const BinParams &bp, const BinTables &t, const XbinGeo &xg, void *const slots[4],
        const double *dcv, double *bins) {
  if (xrow_full(bp)) launch_xrow_t<1, true, true, 1>(s, bp, t, xg, slots, dcv, bins);
  else launch_xrow_t<1, true, false, 1>(s, bp, t, xg, slots, dcv, bins);
}
