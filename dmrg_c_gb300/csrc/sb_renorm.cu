// sb_renorm.cu -- operator renormalisation Out = M1 (M2 M3) (CRS_CRS_CCS_PRODUCT,
// sml/CRS_CRS_CCS_PRODUCT.c:6-124), the product TRANSFORM_MATRIX and DMRG_EXTEND_AND_REDUCE apply
// to every block operator of a DMRG step (T^dagger O T: M1 = Trans_Matrix_Dagger in CRS, M2 the
// operator on the LLLR basis in CRS, M3 = Trans_Matrix in CCS).
//
// The reference forms W = M2 M3 column by column (the column of M3 scattered into a dense vector,
// each row of M2 summed against it in storage order, |value| > 1e-15 kept, CCS), then Out = M1 W row
// by row (the row of M1 scattered, each column of W summed in its storage order, |value| > 1e-15
// kept, CRS).  On the device both products are one thread per output entry over dense copies of the
// scattered operand -- M3 by columns, M1 by columns -- with the sums in the reference's order and
// rounded as written, so every kept value is bitwise the reference's (entries whose operands' supports
// lie apart are zero and cost no sum); an ordered compaction (a
// block per column of W / row of Out, prefix sums of the keep flags) writes CCS / CRS in the
// reference's element order.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <vector>

#include "common.cuh"

namespace dg {
namespace {

constexpr double kZero = 1e-15;   // |value| above this is kept (pow(10,-15) in the reference)

// Support of a line (a column of M3, a row of M1 or M2): the smallest and largest index stored,
// (INT_MAX, -1) for an empty one.
struct Span {
  int lo, hi;
};
__device__ __forceinline__ bool apart(Span a, Span b) { return a.lo > b.hi || a.hi < b.lo; }

// The spans of n lines and, with D, their dense copy: entry e of line l goes to
// D[l * lstride + idx[e] * estride], in storage order (the last of repeated indices wins, as in the
// reference's scatter; within 32 entries the highest lane of an index writes).  *odd is set when a
// value is infinite or NaN.  A warp per line: with one thread a line, each walking its entries
// through two dependent L2 round trips, the scatters of T (512 lines of ~36) took 109 and 101 us;
// now about 5.
__global__ void __launch_bounds__(kThreads) k_lines(int n, const int64_t *__restrict__ ptr, const int *__restrict__ idx,
                                                   const double *__restrict__ val, Span *__restrict__ span, double *__restrict__ D,
                                                   int64_t lstride, int64_t estride, int *__restrict__ odd) {
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  for (int l = warp; l < n; l += nw) {
    const int64_t b = ptr[l], e = ptr[l + 1];
    unsigned lo = INT_MAX;
    int hi = -1;
    bool bad = false;
    for (int64_t k0 = b; k0 < e; k0 += 32) {
      const int64_t k = k0 + lane;
      const int i = k < e ? idx[k] : -1;
      const double v = k < e ? val[k] : 0.0;
      if (k < e) {
        lo = min(lo, (unsigned)i);
        hi = max(hi, i);
        bad = bad || !isfinite(v);
      }
      if (D) {
        const unsigned same = __match_any_sync(0xffffffffu, i);
        if (k < e && 31 - __clz(same) == lane) D[(int64_t)l * lstride + (int64_t)i * estride] = v;
        __syncwarp();   // the next 32 entries' stores come after these
      }
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if (lane == 0) span[l] = Span{(int)lo, hi};
    if (__any_sync(0xffffffffu, bad) && lane == 0) *odd = 1;
  }
}

// W[c * rows + i] = sum over row i of M2 (storage order) of D3[c * ld3 + col] * val.  A block per
// column, a thread per row.  Where the row's columns lie apart from the support of M3's column every
// product is a zero, which changes no sum: the entry is 0 without walking the row.  The operands of a
// renormalisation conserve the block labels, so that is nine entries of ten, and the FP64 work (two
// instructions a term, rounded apart) is what bounds the rest: Hubbard m=512 (2048 x 512 entries,
// 74 k stored in M2) 213 us with every row walked; the whole call from host arrays 0.95 -> 0.55 ms.  A product of zero and an infinity is not zero:
// when M2 holds a non-finite value (odd) every row is walked.
__global__ void __launch_bounds__(kThreads) k_rows_times_dense(int rows, int ncols, const int64_t *__restrict__ rp, const int *__restrict__ ci,
                                                              const double *__restrict__ cv, const Span *__restrict__ rspan,
                                                              const Span *__restrict__ cspan, const int *__restrict__ odd,
                                                              const double *__restrict__ D, int64_t ld, double *__restrict__ W,
                                                              int *__restrict__ w_odd) {
  const bool walk_all = *odd != 0;
  for (int c = blockIdx.y; c < ncols; c += gridDim.y) {
    const double *__restrict__ d = D + (int64_t)c * ld;
    const Span sc = cspan[c];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < rows; i += gridDim.x * blockDim.x) {
      double acc = 0.0;
      if (walk_all || !apart(rspan[i], sc)) {
        int64_t k = rp[i];
        const int64_t e = rp[i + 1];
        for (; k + 8 <= e; k += 8) {   // eight gathers in flight, summed in storage order
          int cc[8];
          double a[8], v[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            cc[u] = ci[k + u];
            v[u] = cv[k + u];
          }
#pragma unroll
          for (int u = 0; u < 8; ++u) a[u] = d[cc[u]];
#pragma unroll
          for (int u = 0; u < 8; ++u) acc = __dadd_rn(acc, __dmul_rn(a[u], v[u]));
        }
        for (; k < e; ++k) acc = __dadd_rn(acc, __dmul_rn(d[ci[k]], cv[k]));
        if (!isfinite(acc)) *w_odd = 1;
      }
      W[(int64_t)c * rows + i] = acc;
    }
  }
}

// O[c * rows + r] = sum over the stored entries of column c of W (storage order, rows ascending) of
// D1[row * rows + r] * value; 0 where the column's rows lie apart from row r of M1's columns (as
// k_rows_times_dense; w_odd: W holds a non-finite value).
__global__ void __launch_bounds__(kThreads) k_dense_times_cols(int rows, int ncols, const int64_t *__restrict__ cp,
                                                              const int *__restrict__ ri, const double *__restrict__ rv,
                                                              const Span *__restrict__ rspan, const int *__restrict__ w_odd,
                                                              const double *__restrict__ D1, double *__restrict__ O) {
  const bool walk_all = *w_odd != 0;
  for (int c = blockIdx.y; c < ncols; c += gridDim.y) {
    const int64_t b = cp[c], e = cp[c + 1];
    const Span sc = e > b ? Span{ri[b], ri[e - 1]} : Span{INT_MAX, -1};
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x) {
      double acc = 0.0;
      if (walk_all || !apart(rspan[r], sc)) {
        int64_t k = b;
        for (; k + 8 <= e; k += 8) {
          double a[8], v[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            a[u] = D1[(int64_t)ri[k + u] * rows + r];
            v[u] = rv[k + u];
          }
#pragma unroll
          for (int u = 0; u < 8; ++u) acc = __dadd_rn(acc, __dmul_rn(a[u], v[u]));
        }
        for (; k < e; ++k) acc = __dadd_rn(acc, __dmul_rn(D1[(int64_t)ri[k] * rows + r], rv[k]));
      }
      O[(int64_t)c * rows + r] = acc;
    }
  }
}

// Ordered compaction of a dense matrix along its lines: line l holds len values at
// A[l * lstride + j * estride]; count[l] = kept values (pass 0), or the kept values' positions and
// values written from off[l] on (pass 1).  One block a line.
__global__ void __launch_bounds__(kThreads) k_compact_lines(int nlines, int len, const double *__restrict__ A, int64_t lstride,
                                                           int64_t estride, int pass, int64_t *__restrict__ count,
                                                           const int64_t *__restrict__ off, int *__restrict__ pos,
                                                           double *__restrict__ out) {
  __shared__ int warp_sum[kWarps];
  __shared__ int64_t base;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int l = blockIdx.x; l < nlines; l += gridDim.x) {
    if (threadIdx.x == 0) base = pass ? off[l] : 0;
    __syncthreads();
    for (int j0 = 0; j0 < len; j0 += blockDim.x) {
      const int j = j0 + threadIdx.x;
      const double v = j < len ? A[(int64_t)l * lstride + (int64_t)j * estride] : 0.0;
      const bool keep = j < len && fabs(v) > kZero;
      const unsigned bal = __ballot_sync(0xffffffffu, keep);
      if (lane == 0) warp_sum[warp] = __popc(bal);
      __syncthreads();
      int before = 0, all = 0;
      for (int w = 0; w < kWarps; ++w) {
        if (w < warp) before += warp_sum[w];
        all += warp_sum[w];
      }
      if (pass && keep) {
        const int64_t at = base + before + __popc(bal & ((1u << lane) - 1u));
        pos[at] = j;
        out[at] = v;
      }
      __syncthreads();
      if (threadIdx.x == 0) base += all;
      __syncthreads();
    }
    if (!pass && threadIdx.x == 0) count[l] = base;
    __syncthreads();
  }
}

[[noreturn]] void fatal(const char *msg) {
  printf("error in CRS_CRS_CCS_PRODUCT\n%s\n", msg);
  fflush(stdout);
  exit(1);
}

// The reference checks the capacity before every candidate entry, so it stops as soon as the count
// reaches max and another candidate follows.
void check_capacity(const char *what, int64_t kept, int64_t max, int64_t candidates, bool last_kept) {
  if (candidates == 0) return;
  if (max == 0 || kept > max || (kept == max && !last_kept)) {
    char msg[160];
    snprintf(msg, sizeof(msg), "Need more %s->max_val = %lld", what, (long long)std::min(kept, max));
    fatal(msg);
  }
}

template <class T>
void upload(DevBuf<T> &b, const T *h, size_t n, cudaStream_t st) {
  b.alloc(std::max<size_t>(n, 1));
  if (n) DG_CUDA(cudaMemcpyAsync(b.get(), h, sizeof(T) * n, cudaMemcpyHostToDevice, st));
}

void crs_crs_ccs(CRS1 *M1, CRS1 *M2, CCS1 *M3, CRS1 *Out, CCS1 *Work, double *Work_Vec) {
  const int row_m1 = M1->row_dim, row_m2 = M2->row_dim, row_m3 = M3->row_dim, col_m3 = M3->col_dim;
  // operand indices are checked here: the device never addresses outside its dense copies
  auto check_idx = [&](const char *name, long n_lines, const long *ptr, const int *idx, int limit) {
    for (long l = 0; l < n_lines; ++l) {
      if (ptr[l + 1] < ptr[l]) fatal("decreasing offsets");
      for (long e = ptr[l]; e < ptr[l + 1]; ++e)
        if (idx[e] < 0 || idx[e] >= limit) {
          char msg[160];
          snprintf(msg, sizeof(msg), "%s index %d outside [0, %d)", name, idx[e], limit);
          fatal(msg);
        }
    }
  };
  if ((double)std::max(row_m3, row_m2) * col_m3 > 2147483647.0 || (double)row_m2 * row_m1 > 2147483647.0)
    fatal("the operands are too large for the dense-column product (more than 2^31 dense entries)");
  check_idx("M1 column", row_m1, M1->Row, M1->Col, row_m2);
  check_idx("M2 column", row_m2, M2->Row, M2->Col, row_m3);
  check_idx("M3 row", col_m3, M3->Col, M3->Row, row_m3);
  const long nnz1 = M1->Row[row_m1] - M1->Row[0], nnz2 = M2->Row[row_m2] - M2->Row[0], nnz3 = M3->Col[col_m3] - M3->Col[0];
  std::vector<double> Wval, Oval;
  std::vector<int> Wrow, Ocol;
  std::vector<int64_t> Wcnt(col_m3), Ocnt(row_m1);
  bool w_last = false, o_last = false;
  const int rc = guarded([&] {
    require_device();
    cudaStream_t st = stream();
    // operands (offsets rebased to their first entry)
    std::vector<int64_t> p1(M1->Row, M1->Row + row_m1 + 1), p2(M2->Row, M2->Row + row_m2 + 1), p3(M3->Col, M3->Col + col_m3 + 1);
    for (auto &x : p1) x -= M1->Row[0];
    for (auto &x : p2) x -= M2->Row[0];
    for (auto &x : p3) x -= M3->Col[0];
    DevBuf<int64_t> d_p1, d_p2, d_p3;
    DevBuf<int> d_c1, d_c2, d_r3;
    DevBuf<double> d_v1, d_v2, d_v3;
    upload(d_p1, p1.data(), p1.size(), st);
    upload(d_p2, p2.data(), p2.size(), st);
    upload(d_p3, p3.data(), p3.size(), st);
    upload(d_c1, M1->Col + M1->Row[0], nnz1, st);
    upload(d_v1, M1->Val + M1->Row[0], nnz1, st);
    upload(d_c2, M2->Col + M2->Row[0], nnz2, st);
    upload(d_v2, M2->Val + M2->Row[0], nnz2, st);
    upload(d_r3, M3->Row + M3->Col[0], nnz3, st);
    upload(d_v3, M3->Val + M3->Col[0], nnz3, st);
    const int sms = sm_count();
    auto grid = [&](int64_t work) { return (int)std::max<int64_t>(1, std::min<int64_t>((work + kThreads - 1) / kThreads, (int64_t)sms * 8)); };
    // a block per column of the result, its threads over the rows
    auto grid2 = [&](int rows, int cols) { return dim3((unsigned)grid(rows), (unsigned)std::max(1, std::min(cols, 65535))); };
    DevBuf<Span> s1(std::max(row_m1, 1)), s2(std::max(row_m2, 1)), s3(std::max(col_m3, 1));
    DevBuf<int> odd(3);   // a non-finite value in M2 / in W / in M1 or M3 (not needed)
    DG_CUDA(cudaMemsetAsync(odd.get(), 0, sizeof(int) * 3, st));
    // W = M2 M3 (dense, by columns), then its CCS
    DevBuf<double> D3((size_t)row_m3 * col_m3), Wd((size_t)row_m2 * col_m3);
    DG_CUDA(cudaMemsetAsync(D3.get(), 0, sizeof(double) * D3.n, st));
    k_lines<<<grid((int64_t)col_m3 * 32), kThreads, 0, st>>>(col_m3, d_p3.get(), d_r3.get(), d_v3.get(), s3.get(), D3.get(), row_m3, 1,
                                                             odd.get() + 2);
    count_launch();
    k_lines<<<grid((int64_t)row_m2 * 32), kThreads, 0, st>>>(row_m2, d_p2.get(), d_c2.get(), d_v2.get(), s2.get(), nullptr, 0, 0,
                                                             odd.get());
    count_launch();
    k_rows_times_dense<<<grid2(row_m2, col_m3), kThreads, 0, st>>>(row_m2, col_m3, d_p2.get(), d_c2.get(), d_v2.get(), s2.get(), s3.get(),
                                                                   odd.get(), D3.get(), row_m3, Wd.get(), odd.get() + 1);
    count_launch();
    DevBuf<int64_t> wcnt(col_m3), woff(col_m3);
    k_compact_lines<<<grid((int64_t)col_m3 * kThreads), kThreads, 0, st>>>(col_m3, row_m2, Wd.get(), row_m2, 1, 0, wcnt.get(), nullptr,
                                                                          nullptr, nullptr);
    count_launch();
    DG_CUDA(cudaGetLastError());
    DG_CUDA(cudaMemcpyAsync(Wcnt.data(), wcnt.get(), sizeof(int64_t) * col_m3, cudaMemcpyDeviceToHost, st));
    DG_CUDA(cudaStreamSynchronize(st));
    std::vector<int64_t> wo(col_m3 + 1, 0);
    for (int c = 0; c < col_m3; ++c) wo[c + 1] = wo[c] + Wcnt[c];
    const int64_t nnzW = wo[col_m3];
    DevBuf<int> Wr(nnzW);
    DevBuf<double> Wv(nnzW);
    DevBuf<int64_t> d_wo;
    upload(d_wo, wo.data(), wo.size(), st);
    k_compact_lines<<<grid((int64_t)col_m3 * kThreads), kThreads, 0, st>>>(col_m3, row_m2, Wd.get(), row_m2, 1, 1, nullptr, d_wo.get(),
                                                                          Wr.get(), Wv.get());
    count_launch();
    // Out = M1 W (dense, by columns), then its CRS
    DevBuf<double> D1((size_t)row_m2 * row_m1), Od((size_t)row_m1 * col_m3);
    DG_CUDA(cudaMemsetAsync(D1.get(), 0, sizeof(double) * D1.n, st));
    k_lines<<<grid((int64_t)row_m1 * 32), kThreads, 0, st>>>(row_m1, d_p1.get(), d_c1.get(), d_v1.get(), s1.get(), D1.get(), 1, row_m1,
                                                             odd.get() + 2);
    count_launch();
    k_dense_times_cols<<<grid2(row_m1, col_m3), kThreads, 0, st>>>(row_m1, col_m3, d_wo.get(), Wr.get(), Wv.get(), s1.get(),
                                                                   odd.get() + 1, D1.get(), Od.get());
    count_launch();
    DevBuf<int64_t> ocnt(row_m1);
    k_compact_lines<<<grid((int64_t)row_m1 * kThreads), kThreads, 0, st>>>(row_m1, col_m3, Od.get(), 1, row_m1, 0, ocnt.get(), nullptr,
                                                                          nullptr, nullptr);
    count_launch();
    DG_CUDA(cudaGetLastError());
    DG_CUDA(cudaMemcpyAsync(Ocnt.data(), ocnt.get(), sizeof(int64_t) * row_m1, cudaMemcpyDeviceToHost, st));
    DG_CUDA(cudaStreamSynchronize(st));
    std::vector<int64_t> oo(row_m1 + 1, 0);
    for (int r = 0; r < row_m1; ++r) oo[r + 1] = oo[r] + Ocnt[r];
    const int64_t nnzO = oo[row_m1];
    DevBuf<int> Oc(nnzO);
    DevBuf<double> Ov(nnzO);
    DevBuf<int64_t> d_oo;
    upload(d_oo, oo.data(), oo.size(), st);
    k_compact_lines<<<grid((int64_t)row_m1 * kThreads), kThreads, 0, st>>>(row_m1, col_m3, Od.get(), 1, row_m1, 1, nullptr, d_oo.get(),
                                                                          Oc.get(), Ov.get());
    count_launch();
    DG_CUDA(cudaGetLastError());
    Wrow.resize(nnzW);
    Wval.resize(nnzW);
    Ocol.resize(nnzO);
    Oval.resize(nnzO);
    if (nnzW) {
      DG_CUDA(cudaMemcpyAsync(Wrow.data(), Wr.get(), sizeof(int) * nnzW, cudaMemcpyDeviceToHost, st));
      DG_CUDA(cudaMemcpyAsync(Wval.data(), Wv.get(), sizeof(double) * nnzW, cudaMemcpyDeviceToHost, st));
    }
    if (nnzO) {
      DG_CUDA(cudaMemcpyAsync(Ocol.data(), Oc.get(), sizeof(int) * nnzO, cudaMemcpyDeviceToHost, st));
      DG_CUDA(cudaMemcpyAsync(Oval.data(), Ov.get(), sizeof(double) * nnzO, cudaMemcpyDeviceToHost, st));
    }
    DG_CUDA(cudaStreamSynchronize(st));
    // was the final candidate of each product kept?  (for the capacity rule)
    w_last = nnzW > 0 && Wcnt[col_m3 - 1] > 0 && Wrow[nnzW - 1] == row_m2 - 1;
    o_last = nnzO > 0 && Ocnt[row_m1 - 1] > 0 && Ocol[nnzO - 1] == col_m3 - 1;
  });
  if (rc != DG_OK) {
    char msg[1100];
    snprintf(msg, sizeof(msg), "GPU path failed (status %d): %s", rc, dg_last_error());
    fatal(msg);
  }
  // the reference's results, capacity rule included
  check_capacity("Work", (int64_t)Wval.size(), Work->max_val, (int64_t)row_m2 * col_m3, w_last);
  long e = 0;
  for (int c = 0; c < col_m3; ++c) {
    for (int64_t k = 0; k < Wcnt[c]; ++k, ++e) {
      Work->Val[e] = Wval[e];
      Work->Row[e] = Wrow[e];
    }
    Work->Col[c + 1] = e;
  }
  Work->row_dim = row_m2;
  Work->col_dim = col_m3;
  for (int i = 0; i < std::max(row_m3, row_m2); ++i) Work_Vec[i] = 0.0;
  check_capacity("Out", (int64_t)Oval.size(), Out->max_val, (int64_t)row_m1 * col_m3, o_last);
  e = 0;
  for (int r = 0; r < row_m1; ++r) {
    for (int64_t k = 0; k < Ocnt[r]; ++k, ++e) {
      Out->Val[e] = Oval[e];
      Out->Col[e] = Ocol[e];
    }
    Out->Row[r + 1] = e;
  }
  Out->row_dim = row_m1;
  Out->col_dim = col_m3;
}

}  // namespace
}  // namespace dg

extern "C" {

// include/SML.h:181
void CRS_CRS_CCS_PRODUCT(CRS1 *M1, CRS1 *M2, CCS1 *M3, CRS1 *Out, CCS1 *Work, double *Work_Vec) {
  if (M1->col_dim != M2->row_dim || M2->col_dim != M3->row_dim) {
    char msg[200];
    snprintf(msg, sizeof(msg), "M1_col = %d, M2_row = %d, M2_col = %d, M3_col = %d", M1->col_dim, M2->row_dim, M2->col_dim,
             M3->row_dim);
    dg::fatal(msg);
  }
  if (Work->max_col <= M3->col_dim) {
    char msg[200];
    snprintf(msg, sizeof(msg), "Need more Work->max_col = %d <= %d", Work->max_col, M3->col_dim);
    dg::fatal(msg);
  }
  if (Out->max_row <= M1->row_dim) {
    char msg[200];
    snprintf(msg, sizeof(msg), "Need more Out->max_row = %d <= %d", Out->max_row, M1->row_dim);
    dg::fatal(msg);
  }
  dg::crs_crs_ccs(M1, M2, M3, Out, Work, Work_Vec);
}

}  // extern "C"
