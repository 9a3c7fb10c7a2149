// lgpu_replay.cpp - replays on given data that no solve needs, in a translation unit of
// their own: with this one in lgpu_engine.cpp the compiler inlined less of the rest of it
// (lgpu_get_distributions 595 us, 740 then).
#include "lgpu_engine.h"

extern "C" {

int lgpu_replay_rebin(lgpu_ctx* ctx, int n_cells, int n_cos, int n_phases, double old_max, double new_max,
                      double* eedf, double* eadf, double* eedf_per) {
  if (!ctx || !ctx->e || n_cells < 1 || n_cells > lgpu::kMaxEnergyCells || n_cos < 0 || n_cos > 65536 || n_phases < 0 ||
      n_phases > 65536 || !(old_max > 0) || !(new_max > old_max) || !eedf || (n_cos && !eadf) || (n_phases && !eedf_per))
    return LGPU_ERR_BAD_ARG;
  return ctx->e->replay_rebin(n_cells, n_cos, n_phases, old_max, new_max, eedf, eadf, eedf_per);
}

}  // extern "C"
