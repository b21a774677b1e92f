// Passes that the library's own step drivers share, beside the C entry points.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "dpf_gb300.h"

namespace dpf {

// Doubles a bond of the linearisation that residual_pass stores.
constexpr int kLinear = 46;

// dpf_residual that also stores the linearisation of the midpoint force at y
// (kLinear planes of n_bonds doubles) when `linear` is given; *general becomes 1
// when a committed normal is not a unit vector (the stored form does not hold).
int residual_pass(const dpf_graph *g, const dpf_stiffness *k, const dpf_history *h, const double *y, const double *v,
                  const double *external, const double *mass, const uint8_t *fixed, double dt,
                  const dpf_trial_out *trial, const double *preconditioner, const double *units, double *residual,
                  double *norms, double *wrench, double *partials, int *status, double *linear, double *general,
                  cudaStream_t stream);

// out = P (J d) / units from a stored linearisation; d in the coordinates of y.
int jacobian_pass(const dpf_graph *g, const double *linear, const double *direction, const double *mass,
                  const uint8_t *fixed, double dt, const double *units, const double *preconditioner, double *out,
                  double *wrench, cudaStream_t stream);

// One CGS2 Arnoldi step in one cooperative launch (dpf_arnoldi_cgs2_fused).
int arnoldi_pass(int64_t length, double *basis, int64_t ld, int j, double *w, double *h, double *partials,
                 unsigned *barrier, int *status, cudaStream_t stream);

// What the elastic PCG reads and writes:
//   kElastic    r = block (units vector), out = x / units (dpf_elastic_precondition);
//   kElasticRaw r the same, out = x;
//   kElasticT   r = vector / units, out = units (block x): the transposed preconditioner.
enum ElasticForm { kElastic = 0, kElasticRaw = 1, kElasticT = 2 };

int elastic_pass(const dpf_graph *g, const dpf_stiffness *k, const dpf_tangent *t, const double *mass,
                 const uint8_t *fixed, const double *block, const double *preconditioner, const double *units,
                 const double *vector, double dt, double tolerance, int max_iterations, double *out, int *iterations,
                 double *wrench, double *workspace, unsigned *barrier, int *status, ElasticForm form,
                 cudaStream_t stream);

}  // namespace dpf
