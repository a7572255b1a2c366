// Instances of k_xrow_bin: two fields, interlaced. dd + dp + pp (|A|^2, Im A*B, |B|^2) with even multipoles, or all four products
// and all multipoles.
#include "xrow.cuh"

void launch_xrow_f2i(cudaStream_t s, const BinParams &bp, const BinTables &t, const XbinGeo &xg, void *const slots[4],
        const double *dcv, double *bins) {
  if (xrow_full(bp)) launch_xrow_t<2, true, true, 0xF>(s, bp, t, xg, slots, dcv, bins);
  else launch_xrow_t<2, true, false, 0xD>(s, bp, t, xg, slots, dcv, bins);
}
