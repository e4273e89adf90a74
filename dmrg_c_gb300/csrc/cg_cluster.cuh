// cg_cluster.cuh -- conjugate-gradient iterations of a small system as one kernel on one thread-block
// cluster.
#pragma once

#include "apply.cuh"

struct dg_matrix;

namespace dg {

struct Scalars;
struct Progress;

struct CgCluster {
  int n;
  const int64_t *row;        // CRS operator
  const int *col;
  const double *val;
  double sigma;
  double *x, *r, *p;         // in: the state entering iteration it0; out: after the last one run
  Scalars *S;
  Progress *prog;
  int it0, it1, max_step;    // iterations it0..it1, ended by convergence or by the iteration limit
  double acc;
};

// Whether the cluster form takes the system.
bool cg_cluster_takes(const dg_matrix *m);
// Enqueues the iterations (of a system it takes).
void launch_cg_cluster(const dg_matrix *m, CgCluster a, cudaStream_t st);

}  // namespace dg
