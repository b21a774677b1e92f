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

// The bonds' wrenches of the committed state (dpf_loads without the sites' sums).
int loads_bonds_pass(const dpf_graph *g, const dpf_history *h, double *wrench, cudaStream_t stream);

// A step driver's launches write what the host decides on straight to pinned memory
// (`host` pointers, read after the stream is waited for).  Report: words that the last
// block of a pass copies there beside its own results.
struct Report {
    const double *from = nullptr;
    double *to = nullptr;
    int count = 0;
    const int *status = nullptr;
    int *status_to = nullptr;
    __device__ void send() const {
        for (int k = 0; k < count; ++k) to[k] = from[k];
        if (status) *status_to = *status;
    }
};

// One CGS2 Arnoldi step in one cooperative launch (dpf_arnoldi_cgs2_fused); h may be
// pinned host memory.  clear: the next cooperative launch's barrier word, which this
// launch clears; with it the own word is clean already, without it a memset cleans it.
int arnoldi_pass(int64_t length, double *basis, int64_t ld, int j, double *w, double *h, double *partials,
                 unsigned *barrier, unsigned *clear, int *status, cudaStream_t stream);

// dpf_scale_residual with a report.
int scale_residual64_pass(int64_t n_sites, const double *preconditioner, const double *units, const double *residual,
                          double *scaled, double *norms, double *partials, const Report &report, cudaStream_t stream);

// What the elastic PCG reads and writes:
//   kElastic    r = block (units vector), out = x / units (dpf_elastic_precondition);
//   kElasticRaw r the same, out = x;
//   kElasticT   r = vector / units, out = units (block x): the transposed preconditioner.
// clear as arnoldi_pass.
enum ElasticForm { kElastic = 0, kElasticRaw = 1, kElasticT = 2 };

int elastic_pass(const dpf_graph *g, const dpf_stiffness *k, const dpf_tangent *t, const double *mass,
                 const uint8_t *fixed, const double *block, const double *preconditioner, const double *units,
                 const double *vector, double dt, double tolerance, int max_iterations, double *out, int *iterations,
                 double *wrench, double *workspace, unsigned *barrier, unsigned *clear, int *status, ElasticForm form,
                 cudaStream_t stream);

// ---- passes of the mixed-precision step driver -------------------------------
//
// The driver's launches are shared or joined where the entry points of the same
// passes each read and write whole vectors; every entry gets the same arithmetic
// in the same order, so a step gives the same bits either way.

// dpf_mixed_begin, and the start of a step whose records come from the last
// commit: y = y32 = 0, residual = r0 on free sites, cleared status, counter and
// barrier words.
int mixed_start_pass(int64_t n_sites, const double *loads, const double *mass, const double *v, const double *external,
                     const uint8_t *fixed, double dt, double *r0, double *scales, double *partials, double *y,
                     float *y32, double *residual, int *status, int *inner, unsigned *barrier, cudaStream_t stream);

// dpf_mixed_scale_residual with a report.
int scale_residual_pass(int64_t n_sites, const float *preconditioner, const float *units32, const double *residual,
                        double *scaled, double *norms, double *partials, const Report &report, cudaStream_t stream);

// dpf_mixed_jacobian_vector_f32 with d32 = units * direction already written.
int jvp32_pass(const dpf_graph *g, float *bond_data, const float *y32, const float *mass32, const uint8_t *fixed,
               double dt, const float *units32, const float *preconditioner, float *out, const float *d32,
               float *wrench, cudaStream_t stream);

// dpf_end_precondition_f32 that also writes direction = units * out; the barrier
// words are clean at the launch, and the launch clears `clear` for the next one.
int end_precondition32_pass(const dpf_graph *g, const float *ends, const float *site4, const uint8_t *fixed,
                            const float *block32, const float *P24, const float *units32, const float *vector,
                            double tolerance, int max_iterations, float *out, float *direction, int *iterations,
                            float *workspace, double *partials, unsigned *barrier, unsigned *clear, int *status,
                            int variant, cudaStream_t stream);

// dpf_arnoldi_cgs2_f32, barrier and clear as above; h may be pinned host memory.
int arnoldi32_pass(int64_t length, float *basis, int64_t ld, int j, const float *v, float *w, double *h,
                   double *partials, unsigned *barrier, unsigned *clear, int *status, cudaStream_t stream);

// The end of a restart cycle: x = sum c_k z_k and the true residual res = -scaled -
// sum c_k (J z_k), or with `add` (a later cycle) x += sum c_k z_k and res -= sum c_k
// (J z_k); the residual's norm in norm[1], the Newton correction (units x, zero rows
// on fixed sites), the full step y + correction and its float32 copy; clears the
// status word.
int mixed_correction_pass(int64_t n_sites, const float *transformed, const float *products, int count,
                          const double *coefficients, bool add, const double *scaled, const double *units,
                          const uint8_t *fixed, const double *y, double *x, double *res, double *correction,
                          double *candidate, float *y32, double *norm, double *partials, int *status,
                          cudaStream_t stream);

// The commit's bond and site passes (dpf_mixed_commit, or with corrections
// dpf_mixed_commit_lazy) for end positions already written.
int mixed_commit_pass(const dpf_graph *g, float *bond_data, const dpf_history *h, const float *y32,
                      const double *x_end, double *normal_end, double *offset_end, double *fn_end, double *fs_end,
                      double *mt_end, double *mb_end, float *corrections, float *dloads, double *loads,
                      cudaStream_t stream);

}  // namespace dpf
