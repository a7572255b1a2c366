// Instances of k_xrow_bin: one or two fields, not interlaced, all multipoles.
#include "xrow.cuh"

void launch_xrow_plain(cudaStream_t s, const BinParams &bp, const BinTables &t, const XbinGeo &xg, void *const slots[4],
        const double *dcv, double *bins) {
  if (bp.nfields == 2) launch_xrow_t<2, false, true, 0xF>(s, bp, t, xg, slots, dcv, bins);
  else launch_xrow_t<1, false, true, 1>(s, bp, t, xg, slots, dcv, bins);
}
