// float32.h -- what the drop-in libraries (legacy.cu) call in libwind and its
// public header does not show: one declaration for both sides.
#pragma once

#include "../../include/wind.h"

// wind_integrate on float32 host arrays of a builtin network, in place on y: the
// arrays are widened and the results narrowed on the device.
extern "C" int wind_integrate_f32(const wind_options* opt, int32_t kind, int32_t n_eq, int32_t n_const, double tnow,
                                  double tend, int32_t n_integration_steps, const float* constants, float* y,
                                  int64_t nsys, double atol, double rtol, int64_t* total_nsteps);
