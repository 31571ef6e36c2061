// The tree walk's form of a cell type (pc::host_walk_type, exported by libprocell.so), for
// tests/test_walk.py: out[0..4] = mean, sd, eps, band per generation, band; cum = the ratio
// threshold on 53-bit integers. Returns whether the walk serves the type.
#include <vector_types.h>

#include "../cuda-pro-cell_gb300/csrc/pc_engine.h"

extern "C" int walk_type(double mean, double sd, double t_max, double cumulative, float* out, uint64_t* cum) {
  pc::TypeDev t = {};
  t.cum = cumulative;
  t.mode = mean < 0.0 ? pc::kModeQuiescent : (mean == 0.0 ? pc::kModeZeroMean : pc::kModeNormal);
  const bool ok = pc::host_walk_type(t, mean, sd, t_max);
  out[0] = t.w_mean;
  out[1] = t.w_sd;
  out[2] = t.w_eps;
  out[3] = t.w_band_gen;
  out[4] = t.w_band;
  *cum = t.w_cum;
  return ok ? 1 : 0;
}
