// pm_adjoint.h -- the differentiation form on a PM handle (internal).
#pragma once

#include <string>

#include <cuda_runtime.h>

#include "hyowon_adjoint.h"

namespace hyowon::adj {

// Adjoint engines (plans and work arrays) a handle keeps between VJP calls.
struct Cache;
void destroy_cache(Cache* c);
// Gives the work arrays of the engines back (they are taken again when used).
void trim_cache(Cache* c);
// Device bytes that gradients of this cache may keep forward potentials in.
int limit_potentials(Cache** c, size_t bytes);
// hyowon_vjp_1lpt_pm on stream s with the engine of *cache (created, or
// re-created when the geometry changed). Returns a hyowon_status code.
int run_cached(Cache** cache, const VjpConfig& cfg, cudaStream_t s, const double* noise,
               const double* target_delta, double* loss, double* grad_noise,
               double* final_delta, double* timings, std::string* err);

}  // namespace hyowon::adj
