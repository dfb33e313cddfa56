// The frequency integrals of ComputeTs on the device (rg_freq.cu).
#pragma once

#include "rg_internal.h"
#include "rg_xray.h"

namespace rg {

// Start the frequency tables of a snapshot's shells on the context's side stream (they need only
// scalars, so they overlap the transforms), then wait for them and fill *out.
int ts_freq_start(rg_context* ctx, const rg_params* p, const TsShells& sh, double zp, double x_e_ave,
                  double collapse_fraction, const double* ZZ, const double* stored_fcoll, int snapshot);
int ts_freq_finish(rg_context* ctx, const rg_params* p, const TsShells& sh, double zp, TsTables* out);

}  // namespace rg
