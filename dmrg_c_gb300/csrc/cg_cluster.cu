// cg_cluster.cu -- conjugate gradients of a small system (cg_cluster.cuh).
//
// An iteration is a product, two vector updates and two dot products: three launches, and for a
// few thousand rows nearly all of it is what lies between them.  Here one cluster of up to
// 16 CTAs keeps the solve: a CTA owns a contiguous range of rows with its parts of x, r and y in
// shared memory, every CTA holds the whole direction p there (the product gathers from it), and
// the dot products and the new direction go through distributed shared memory, three cluster
// barriers an iteration.  The recurrences are those of k_cg_update and k_cg_direction.
#include <algorithm>
#include <cstring>

#include <cooperative_groups.h>

#include "cg_cluster.cuh"
#include "krylov.cuh"
#include "matrix.cuh"

namespace dg {
namespace {

constexpr int kCgThreads = 512;
// Sizes up to which the cluster is faster than the three kernels on the whole GPU, whose 11 - 12 us an
// iteration do not depend on the size there.  Measured, us an iteration on the cluster (n, elements):
// 5.8 (100, 1 k), 6.5 (924, 8 k), 9.0 (3,432, 31 k), 10.1 (2,000, 62 k); past the limits 13.9 (8,000, 72 k) and
// 16.2 (3,696, 245 k; 4.4 of it FP64 issue of 16 SMs, the rest their gathers and barriers).  At 3,432 rows the
// FP64 pipe is 31 % busy and most stalls are at barriers.
constexpr int kCgClusterN = 4096;
constexpr long kCgClusterNnz = 1L << 16;

template <int L>
__global__ void __launch_bounds__(kCgThreads) k_cg_cluster(CgCluster a, int rows) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int cs = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  extern __shared__ double cg_smem[];
  double *const p = cg_smem, *const x = p + a.n, *const r = x + rows, *const y = r + rows;
  __shared__ double s_py[16], s_rr[16], s_sc[2];
  const int tid = threadIdx.x, lane = tid & 31;
  const int n = a.n, r0 = min(n, rank * rows), nloc = min(n, r0 + rows) - r0;
  pdl_wait();
  // (written only behind the first barrier, so the same in every CTA)
  if (*((volatile const int *)&a.S->done)) return;
  for (int i = tid; i < n; i += kCgThreads) p[i] = a.p[i];
  for (int i = tid; i < nloc; i += kCgThreads) {
    x[i] = a.x[r0 + i];
    r[i] = a.r[r0 + i];
  }
  double rr = a.S->rrs[a.it0 & 1];
  cluster.sync();   // every CTA runs: its shared memory may be written
  // the cluster's sum of v, in the first warp of every CTA, the same bits in each
  auto cluster_sum = [&](double v, double *slots) {
    double t[1] = {v};
    block_sums<kCgThreads, 1>(t);
    if (tid < cs) cluster.map_shared_rank(slots, tid)[rank] = t[0];
    cluster.sync();
    double c = tid < cs ? slots[tid] : 0.0;
    if (tid < 32) c = lanes_sum<16>(c);
    return c;
  };
  int it = a.it0, done = 0;
  for (;; ++it) {
    // y = (H + sigma) p on this CTA's rows, L lanes a row
    double dot = 0.0;
    for (int i0 = 0; i0 < nloc; i0 += kCgThreads / L) {
      const int i = i0 + tid / L;
      double q = 0.0;
      if (i < nloc) {
        const int64_t e = a.row[r0 + i + 1];
#pragma unroll 4
        for (int64_t k = a.row[r0 + i] + tid % L; k < e; k += L) q += a.val[k] * p[a.col[k]];
      }
      q = lanes_sum<L>(q);
      if (i < nloc && tid % L == 0) {
        const double pi = p[r0 + i];
        if (a.sigma != 0.0) q += a.sigma * pi;
        y[i] = q;
        dot += q * pi;
      }
    }
    const double py = cluster_sum(dot, s_py);
    if (tid == 0) s_sc[0] = rr / py;
    __syncthreads();
    const double alpha = s_sc[0];
    double nn = 0.0;
    for (int i = tid; i < nloc; i += kCgThreads) {
      x[i] += alpha * p[r0 + i];
      const double rn = r[i] - alpha * y[i];
      r[i] = rn;
      nn += rn * rn;
    }
    const double t = cluster_sum(nn, s_rr);
    if (tid == 0) {
      s_sc[0] = t;
      s_sc[1] = t / rr;
    }
    __syncthreads();
    const double beta = s_sc[1];
    rr = s_sc[0];
    done = rr < a.acc ? 1 : it >= a.max_step - 1 ? 2 : 0;
    if (done) break;
    for (int i = tid; i < nloc; i += kCgThreads) {
      const double pn = r[i] + beta * p[r0 + i];
      for (int c = 0; c < cs; ++c) cluster.map_shared_rank(p, c)[r0 + i] = pn;
    }
    cluster.sync();
    if (it >= a.it1) break;
  }
  for (int i = tid; i < nloc; i += kCgThreads) {
    a.x[r0 + i] = x[i];
    a.r[r0 + i] = r[i];
    a.p[r0 + i] = p[r0 + i];
  }
  if (rank == 0 && tid == 0) {
    a.S->rrs[(it + 1) & 1] = rr;
    if (done) {
      a.S->done = done;
      a.S->iters = done == 1 ? it : a.max_step;
    }
    a.prog->done = done;
    a.prog->stamp = it;
  }
}

}  // namespace

bool cg_cluster_takes(const dg_matrix *m) { return m->n <= kCgClusterN && m->nnz <= kCgClusterNnz; }

void launch_cg_cluster(const dg_matrix *m, CgCluster a, cudaStream_t st) {
  a.n = m->n;
  a.row = m->row.get();
  a.col = m->col.get();
  a.val = m->val.get();
  auto kernel = m->nnz > 16L * a.n ? k_cg_cluster<8> : k_cg_cluster<4>;
  constexpr int kSmem = (int)sizeof(double) * (kCgClusterN + 3 * (kCgClusterN / 8));
  DG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
  // a device that runs no cluster of 16 gets 8
  const bool wide = runs_cluster16((const void *)kernel, kCgThreads, kSmem);
  int cs = 1;
  while (cs < (wide ? 16 : 8) && cs * 32 < a.n) cs <<= 1;
  const int rows = (a.n + cs - 1) / cs;
  cudaLaunchConfig_t cfg;
  std::memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)cs);
  cfg.blockDim = dim3(kCgThreads);
  cfg.dynamicSmemBytes = sizeof(double) * ((size_t)a.n + 3 * (size_t)rows);
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  DG_CUDA(cudaLaunchKernelEx(&cfg, kernel, a, rows));
  count_launch();
}

}  // namespace dg
