// dense.cu -- the dense path's step kernel (dense.cuh).
//
// A step is the product y = H v_b, alpha_b = <y, v_b>, the three-term recurrence and two classical
// Gram-Schmidt passes against v_0..v_b: six kernels and four reductions over vectors of a few
// hundred elements, all of it latency.  Here one cluster of up to 16 CTAs keeps the step: each CTA
// owns a contiguous range of rows, holds its part of the basis in shared memory (read once for the
// four passes over it, and before the kernel waits for its predecessor, except for the newest
// vector), and the reductions are exchanged through distributed shared memory, one cluster barrier
// each: alpha, the coefficients of each pass, the norm.  What is left is latency: barriers, the
// chains of dependent FP64 operations and loads (the FP64 pipe of a CTA's SM is 31 % busy, at 19 cycles a
// warp instruction): the dot products are summed by transposing through shared memory (one add a
// lane and vector instead of a five-step shuffle tree), the subtraction by four threads a row.
//
// Measured on the XXZ chain of 924 states (59 steps): 37 us a step as six kernels, 18 like this (build and solve 2.70 -> 1.45 ms).
#include <algorithm>
#include <cstring>

#include <cooperative_groups.h>

#include "dense.cuh"
#include "matrix.cuh"

namespace dg {
namespace {

constexpr int kDenseRows = kDenseMaxN / 16;   // rows a CTA, at most (four threads a row)
constexpr int kDenseChunk = 128;              // vectors whose coefficients are exchanged at once
constexpr size_t kDenseBasisBytes = 128 * 1024;   // shared memory for a CTA's part of the basis
constexpr size_t kDenseFixedBytes = sizeof(double) * kDenseChunk * (33 + 2 * 16);

template <int L>
__global__ void __launch_bounds__(kThreads) k_dense_step(DenseStep a, int rows, int cap) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int cs = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  extern __shared__ double dense_smem[];
  double (*const tile)[33] = reinterpret_cast<double (*)[33]>(dense_smem);   // kDenseChunk dot products by lane
  // the CTAs' coefficient sums [2][16][kDenseChunk], alternating, then cap vectors of ld elements
  double (*const part)[16][kDenseChunk] = reinterpret_cast<double (*)[16][kDenseChunk]>(dense_smem + kDenseChunk * 33);
  double *const basis = dense_smem + kDenseChunk * (33 + 2 * 16);
  __shared__ double coef[kDenseMaxN];
  __shared__ double w_s[kDenseRows], v_s[kDenseRows];
  __shared__ double s_alpha[16], s_norm[16];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = a.n, b = a.b, ld = rows | 1;
  const int r0 = min(n, rank * rows), nloc = min(n, r0 + rows) - r0;
  // this CTA's rows of the stored vectors: from shared memory up to vector cap, else from L2
  auto keep = [&](int j) {
    if (j < cap)
      for (int i = lane; i < nloc; i += 32) basis[j * ld + i] = a.V[(size_t)j * n + r0 + i];
  };
  auto vec = [&](int j) -> const double * { return j < cap ? basis + j * ld : a.V + (size_t)j * n + r0; };
  // v_0..v_{b-2} were complete when the predecessor began: they need no wait
  for (int j = warp; j < b - 1; j += kWarps) keep(j);
  pdl_wait();
  if (b > 0 && warp == (b - 1) % kWarps) keep(b - 1);
  const double s = a.r2->rs, o = b > 0 ? sqrt(a.r2->v) : 0.0;
  // v_b, y = H v_b = s (H w) on this CTA's rows, L lanes a row
  double dot = 0.0;
  for (int i0 = 0; i0 < nloc; i0 += kThreads / L) {
    const int i = i0 + tid / L;
    double y = 0.0;
    if (i < nloc) {
      const int64_t e = a.row[r0 + i + 1];
      for (int64_t k = a.row[r0 + i] + tid % L; k < e; k += L) y += a.val[k] * a.w[a.col[k]];
    }
    y = lanes_sum<L>(y) * s;
    if (i < nloc && tid % L == 0) {
      const double v = a.w[r0 + i] * s;
      a.V[(size_t)b * n + r0 + i] = v;
      if (b < cap) basis[b * ld + i] = v;
      v_s[i] = v;
      w_s[i] = y;
      dot += y * v;
    }
  }
  pdl_trigger();
  dot = block_sum(dot);
  if (tid < 32) {
    dot = __shfl_sync(0xffffffffu, dot, 0);
    if (lane < cs) cluster.map_shared_rank(s_alpha, lane)[rank] = dot;
  }
  cluster.sync();   // every CTA's alpha part is here, and w has been read by all
  double alpha = 0.0;
  for (int c = 0; c < cs; ++c) alpha += s_alpha[c];
  if (rank == 0 && tid == 0) {
    a.D[b] = alpha;
    a.O[b] = o;
    a.hD[b] = alpha;
    a.hO[b] = o;
  }
  for (int i = tid; i < nloc; i += kThreads) {
    double r = w_s[i] - alpha * v_s[i];
    if (b > 0) r = r - o * vec(b - 1)[i];
    w_s[i] = r;
  }
  __syncthreads();
  const int nvec = b + 1;
  int buf = 0;
  for (int pass = 0; pass < 2; ++pass) {
    // coef_j = <v_j, w>
    for (int j0 = 0; j0 < nvec; j0 += kDenseChunk, buf ^= 1) {
      const int cnt = min(kDenseChunk, nvec - j0);
      for (int j = warp; j < cnt; j += kWarps) {
        const double *v = vec(j0 + j);
        double p = 0.0;
        if (lane < nloc) p = v[lane] * w_s[lane];
        if (lane + 32 < nloc) p += v[lane + 32] * w_s[lane + 32];
        tile[j][lane] = p;
      }
      __syncthreads();
      if (tid < cnt) {
        double q[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int l = 0; l < 32; l += 4)
#pragma unroll
          for (int u = 0; u < 4; ++u) q[u] += tile[tid][l + u];
        const double c = (q[0] + q[1]) + (q[2] + q[3]);
        for (int r = 0; r < cs; ++r) (*cluster.map_shared_rank(&part[buf][rank], r))[tid] = c;
      }
      cluster.sync();
      if (tid < cnt) {
        double c = 0.0;
        for (int r = 0; r < cs; ++r) c += part[buf][r][tid];
        coef[j0 + tid] = c;
      }
    }
    __syncthreads();
    // w -= sum_j coef_j v_j, four threads a row
    const int i = tid >> 2;
    double r = 0.0;
    if (i < nloc)
      for (int j = tid & 3; j < nvec; j += 4) r += coef[j] * vec(j)[i];
    r += __shfl_xor_sync(0xffffffffu, r, 1);
    r += __shfl_xor_sync(0xffffffffu, r, 2);
    if (i < nloc && (tid & 3) == 0) w_s[i] -= r;
    __syncthreads();
  }
  double nn = 0.0;
  for (int i = tid; i < nloc; i += kThreads) {
    const double r = w_s[i];
    a.w[r0 + i] = r;
    nn += r * r;
  }
  nn = block_sum(nn);
  if (tid == 0) cluster.map_shared_rank(s_norm, 0)[rank] = nn;
  cluster.sync();
  if (rank == 0 && tid == 0) {
    double t = 0.0;
    for (int c = 0; c < cs; ++c) t += s_norm[c];
    set_norm2(a.r2, t);
  }
}

}  // namespace

bool launch_dense_step(const dg_matrix *m, DenseStep a, cudaStream_t st) {
  a.n = m->n;
  a.row = m->row.get();
  a.col = m->col.get();
  a.val = m->val.get();
  if (a.n > kDenseMaxN) return false;
  auto kernel = m->nnz > 16L * a.n ? k_dense_step<8> : k_dense_step<4>;
  constexpr size_t kMost = kDenseFixedBytes + kDenseBasisBytes;
  DG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMost));
  // a device that runs no cluster of 16 takes systems of up to 8 CTAs' rows
  const bool wide = runs_cluster16((const void *)kernel, kThreads, kMost);
  // about 32 rows a CTA, so that a row's four threads and the barrier's cost both count little
  int cs = 1;
  while (cs < 16 && cs * 32 < a.n) cs <<= 1;
  if (cs == 16 && !wide) cs = 8;
  const int rows = (a.n + cs - 1) / cs;
  if (rows > kDenseRows) return false;
  const int cap = (int)std::min<size_t>(kDenseBasisBytes / sizeof(double) / (rows | 1), kDenseMaxN);
  cudaLaunchConfig_t cfg;
  std::memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)cs);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kDenseFixedBytes + sizeof(double) * (size_t)(rows | 1) * std::min(cap, (a.b / 32 + 1) * 32);
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
  DG_CUDA(cudaLaunchKernelEx(&cfg, kernel, a, rows, cap));
  count_launch();
  return true;
}

}  // namespace dg
