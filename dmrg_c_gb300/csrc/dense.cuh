// dense.cuh -- one step of the dense path (systems below dense_below states: a Lanczos recurrence
// fully reorthogonalised against its whole basis) as a single kernel on one thread-block cluster.
#pragma once

#include "apply.cuh"

struct dg_matrix;

namespace dg {

// Largest system the cluster step takes (64 rows a CTA on 16 CTAs).
constexpr int kDenseMaxN = 1024;

struct DenseStep {
  int n, b;                  // states; the step
  const int64_t *row;        // CRS operator
  const int *col;
  const double *val;
  double *V;                 // basis, v_j at V + j n; v_b is written
  double *w;                 // in: unnormalised w_b; out: w_{b+1}
  double *D, *O, *hD, *hO;   // recurrence scalars of step b and their host mirrors
  Norm2 *r2;                 // in: <w_b,w_b>; out: <w_{b+1},w_{b+1}>
};

// Enqueues the step; false (nothing enqueued) when the system is too large for it.
bool launch_dense_step(const dg_matrix *m, DenseStep a, cudaStream_t st);

}  // namespace dg
