// sb_build.cu -- superblock Hamiltonian CRS (lower triangle, diagonal last) on the device.
//
// Reference: GET_HAM_LLLRRRRL (main/dmrg/xxz_vf/src/allocations/GET_HAM_LLLRRRRL.c:11-123)
// loops over superblock rows; MAKE_ELEMENT_HAM_LLLRRRRL applies the model's terms in a fixed
// order through DMRG_MAKE_ELEM_*_LLLRRRRL (dmrg/), which append a new target or add to an
// existing one (generation order), then DMRG_MAKE_ELEM_ZERO_LLLRRRRL adds a zero diagonal if
// absent; the row keeps (0 <= col <= row and |v| > 1e-15) or col == row, and
// SORT_COLUMN_CRS1 orders the columns.
//
// GB300 form: one warp per row.  The lanes read the row's term list 32 terms at a time (a lane
// per term: operator rows, fermion sign, target offsets), then walk the generated elements of all
// of them together (element k of a two-operator term is op1 entry k / c2 times op2 entry k % c2,
// the reference's loop order), compute value and target column in parallel, and compact the
// accepted ones (|v| > 1e-15, target in the sector and in the lower triangle, the only ones the
// row can keep) into shared memory with key (column << 22 | generation position).  A bitonic sort
// of the keys puts every column's contributions together in generation order, so summing each run
// left to right reproduces the reference's accumulation bit for bit; the sorted runs are already in
// column order.  The rows are generated once, into a scratch with room for every row's generated
// elements, and compacted behind a scan of the kept counts; where that scratch would be too large
// a count pass and a fill pass generate them twice.
//
// Measured on the Hubbard m=512 superblock of a DMRG run (238 k rows, 325 generated elements a row,
// 28.2 M kept): two passes of 8.96 ms with every term walked by itself (22 terms of ~15 elements:
// most lanes idle, a chain of four dependent loads a term), the upper triangle sorted along and 12
// warps a SM (16 KB of buffer a warp, sized by the operators' widest rows instead of the rows
// themselves).  Term list to solver operator and first product: 22.3 -> 6.4 ms.
#include <algorithm>
#include <cmath>
#include <vector>

#include "dmrg_gb300_sb.h"
#include "matrix.cuh"
#include "sb_basis.cuh"
#include "scan.cuh"

namespace dg {
namespace {

struct SbTermDev {
  int pos1, pos2, op1, op2, sign_mask, sign_even;
  double coef;
};

struct SbDev {
  int n, dim_RR, d, n_terms;
  const short *st[4];             // LL, LR, RR, RL per superblock state
  const int *inv;
  const SbTermDev *terms;
  const int64_t *op_row;          // concatenated row offsets (relative to the op's first element)
  const int *op_row_base;         // first row-offset entry of each op
  const int *op_first;            // first element of each op
  const int *op_col;
  const double *op_val;
  const int *ele[4];
  double zero;
};

constexpr int kGenBits = 22;      // generation position bits of a sort key
constexpr int kSbWarps = 4;       // warps a block, at most
constexpr int kSbTerms = 32;      // terms a warp holds at once: a lane each
constexpr size_t kSbScratchBytes = size_t(2) << 30;   // scratch of the single-pass build, at most

// A term of the row at hand.
struct SbRowTerm {
  int64_t sup, m1, m2;            // target position: sup + col1 * m1 + col2 * m2
  double sc;                      // sign * coefficient
  int e1, e2, c2, first;          // first elements of op1 and op2 (e2 < 0: one operator), op2's
                                  // row length, first generated element of the term
};

// bound[b] = generated elements of row b; *most = the largest.
__global__ void __launch_bounds__(kThreads) k_sb_bounds(SbDev m, long long *__restrict__ bound, int *__restrict__ most) {
  int mx = 0;
  for (long b = (long)blockIdx.x * blockDim.x + threadIdx.x; b < m.n; b += (long)gridDim.x * blockDim.x) {
    long long g = 0;
    for (int t = 0; t < m.n_terms; ++t) {
      const SbTermDev T = m.terms[t];
      if (fabs(T.coef) < m.zero) continue;
      const int64_t *r1 = m.op_row + m.op_row_base[T.op1] + m.st[T.pos1][b];
      long long c = r1[1] - r1[0];
      if (T.pos2 >= 0) {
        const int64_t *r2 = m.op_row + m.op_row_base[T.op2] + m.st[T.pos2][b];
        c *= r2[1] - r2[0];
      }
      g += c;
    }
    bound[b] = g + 1;   // + the zero diagonal
    mx = max(mx, (int)g);
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  if ((threadIdx.x & 31) == 0) atomicMax(most, mx);
}

// Rows of the lower triangle.  soff set: row b's kept elements to col/val[soff[b] ...] (room for its
// bound), their number to counts[b]; else row set: the fill pass, to col/val[row[b] ...]; else the
// count pass.  err: 1 buffer overflow, 2 fill pass and count pass disagree.
__global__ void __launch_bounds__(kSbWarps * 32) k_sb_rows(SbDev m, int cap, const int64_t *__restrict__ soff,
                                                           long long *__restrict__ counts, const int64_t *__restrict__ row,
                                                           int *__restrict__ col, double *__restrict__ val, int *err) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ SbRowTerm s_term[kSbWarps][kSbTerms];
  const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint64_t *keys = reinterpret_cast<uint64_t *>(smem) + (size_t)warp * cap;
  double *vals = reinterpret_cast<double *>(smem + (size_t)warps * cap * sizeof(uint64_t)) + (size_t)warp * cap;
  SbRowTerm *const rt = s_term[warp];
  const unsigned FULL = 0xffffffffu;
  const unsigned lt = (1u << lane) - 1u;
  const int64_t mult[4] = {(int64_t)m.d * m.dim_RR * m.d, (int64_t)m.dim_RR * m.d, m.d, 1};
  for (long b = (long)blockIdx.x * warps + warp; b < m.n; b += (long)gridDim.x * warps) {
    int st[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) st[p] = m.st[p][b];
    const int64_t sup0 = st[0] * mult[0] + st[1] * mult[1] + st[2] * mult[2] + st[3];
    int nitems = 0;
    for (int t0 = 0; t0 < m.n_terms; t0 += kSbTerms) {
      // the terms' operator rows, signs and target offsets: a lane per term
      const int nt = min(kSbTerms, m.n_terms - t0);
      int mine = 0;
      SbRowTerm R{};
      if (lane < nt) {
        const SbTermDev T = m.terms[t0 + lane];
        if (!(fabs(T.coef) < m.zero)) {
          int s1 = 0, s2 = 0;
#pragma unroll
          for (int p = 0; p < 4; ++p) {
            if (T.pos1 == p) {
              s1 = st[p];
              R.m1 = mult[p];
            }
            if (T.pos2 == p) {
              s2 = st[p];
              R.m2 = mult[p];
            }
          }
          const int64_t *r1 = m.op_row + m.op_row_base[T.op1] + s1;
          R.e1 = m.op_first[T.op1] + (int)r1[0];
          mine = (int)(r1[1] - r1[0]);
          R.sup = sup0 - s1 * R.m1 - s2 * R.m2;
          R.c2 = 1;
          R.e2 = -1;
          R.sc = T.coef;
          if (T.pos2 >= 0) {
            const int64_t *r2 = m.op_row + m.op_row_base[T.op2] + s2;
            R.e2 = m.op_first[T.op2] + (int)r2[0];
            R.c2 = (int)(r2[1] - r2[0]);
            mine *= R.c2;
            int sign = 1;
            if (T.sign_mask) {
              int ne = 0;
#pragma unroll
              for (int p = 0; p < 4; ++p)
                if (T.sign_mask & (1 << p)) ne += m.ele[p][st[p]];
              sign = (ne % 2 == 0) ? T.sign_even : -T.sign_even;
            }
            R.sc = __dmul_rn((double)sign, T.coef);
          }
        }
      }
      int incl = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += v;
      }
      const int total = __shfl_sync(FULL, incl, 31);
      R.first = incl - mine;
      __syncwarp();   // the previous terms' readers are done
      rt[lane] = R;   // lanes past nt: first = total, never selected
      __syncwarp();
      // the generated elements of these terms, 32 at a time
      for (int k0 = 0; k0 < total; k0 += 32) {
        const int k = k0 + lane;
        bool acc = false;
        int64_t tgt = -1;
        double v = 0.0;
        if (k < total) {
          int lo = 0;   // the last term whose first element is at or before k (empty terms: the last of equals)
#pragma unroll
          for (int step = kSbTerms / 2; step > 0; step >>= 1)
            if (rt[lo + step].first <= k) lo += step;
          const SbRowTerm &T = rt[lo];
          const int r = k - T.first;
          const int i = T.c2 == 1 ? r : r / T.c2, j = T.c2 == 1 ? 0 : r - i * T.c2;
          const int e1 = T.e1 + i;
          int64_t sup = T.sup + m.op_col[e1] * T.m1;
          v = __dmul_rn(T.sc, m.op_val[e1]);
          if (T.e2 >= 0) {
            sup += m.op_col[T.e2 + j] * T.m2;
            v = __dmul_rn(v, m.op_val[T.e2 + j]);
          }
          tgt = m.inv[sup];
          acc = tgt >= 0 && tgt <= b && fabs(v) > m.zero;
        }
        const unsigned bal = __ballot_sync(FULL, acc);
        const int pos = nitems + __popc(bal & lt);
        if (acc && pos < cap) {
          keys[pos] = ((uint64_t)tgt << kGenBits) | (uint64_t)pos;
          vals[pos] = v;
        }
        nitems += __popc(bal);
      }
    }
    if (nitems > cap) {
      if (lane == 0) {
        atomicExch(err, 1);
        if (counts) counts[b] = 0;
      }
      continue;
    }
    // bitonic sort of the keys, padded to a power of two (the values stay where they are)
    int P = 1;
    while (P < nitems) P <<= 1;
    for (int p = nitems + lane; p < P; p += 32) keys[p] = ~0ull;
    __syncwarp();
    for (int kk = 2; kk <= P; kk <<= 1) {
      for (int j = kk >> 1; j > 0; j >>= 1) {
        for (int i = lane; i < P / 2; i += 32) {
          const int lo = ((i & ~(j - 1)) << 1) | (i & (j - 1)), hi = lo | j;   // the pair's lower index has bit j clear
          const uint64_t ka = keys[lo], kb = keys[hi];
          if ((ka > kb) == ((lo & kk) == 0)) {
            keys[lo] = kb;
            keys[hi] = ka;
          }
        }
        __syncwarp();
      }
    }
    // runs of equal column, summed in generation order
    const int64_t start = soff ? soff[b] : (row ? row[b] : 0), end = soff ? soff[b + 1] : (row ? row[b + 1] : 0);
    const bool write = soff || row;
    const uint64_t gen = (1ull << kGenBits) - 1;
    int kept = 0;
    bool have_diag = false;
    for (int c0 = 0; c0 < nitems; c0 += 32) {
      const int p = c0 + lane;
      bool keep = false, diag = false;
      int64_t t = -1;
      double sum = 0.0;
      if (p < nitems) {
        const uint64_t key = keys[p];
        t = (int64_t)(key >> kGenBits);
        const bool head = (p == 0) || ((int64_t)(keys[p - 1] >> kGenBits) != t);
        if (head) {
          sum = vals[key & gen];
          for (int q = p + 1; q < nitems && (int64_t)(keys[q] >> kGenBits) == t; ++q) sum = __dadd_rn(sum, vals[keys[q] & gen]);
          keep = fabs(sum) > m.zero || t == b;
          diag = t == b;
        }
      }
      const unsigned kb = __ballot_sync(FULL, keep);
      if (write && keep) {
        const int64_t pos = start + kept + __popc(kb & lt);
        if (pos < end) {
          col[pos] = (int)t;
          val[pos] = sum;
        }
      }
      kept += __popc(kb);
      have_diag = have_diag || __any_sync(FULL, diag);
    }
    if (!have_diag) {   // DMRG_MAKE_ELEM_ZERO_LLLRRRRL: a zero diagonal, the row's largest column
      if (write && lane == 0 && start + kept < end) {
        col[start + kept] = (int)b;
        val[start + kept] = 0.0;
      }
      ++kept;
    }
    if (lane == 0) {
      if (counts) counts[b] = kept;
      if (row && !soff && start + kept != end) atomicExch(err, 2);
    }
    __syncwarp();
  }
}

// Row b's kept elements from the scratch (at soff[b]) to col/val[row[b] ...].  One warp a row.
__global__ void __launch_bounds__(kThreads) k_sb_compact(int n, const int64_t *__restrict__ soff, const int64_t *__restrict__ row,
                                                        const int *__restrict__ scol, const double *__restrict__ sval,
                                                        int *__restrict__ col, double *__restrict__ val) {
  const int lane = threadIdx.x & 31;
  const long nw = (long)gridDim.x * kWarps;
  for (long b = blockIdx.x * (long)kWarps + (threadIdx.x >> 5); b < n; b += nw) {
    const int64_t src = soff[b], dst = row[b];
    const int cnt = (int)(row[b + 1] - dst);
    for (int k = lane; k < cnt; k += 32) {
      col[dst + k] = scol[src + k];
      val[dst + k] = sval[src + k];
    }
  }
}

int position_dim(const dg_sb_model *m, int p) {
  return (p == DG_SB_LL) ? m->dim_LL : (p == DG_SB_RR) ? m->dim_RR : m->dim_onsite;
}

}  // namespace
}  // namespace dg

struct dg_sb {
  int n = 0;
  long nnz = 0;
  dg::DevBuf<int64_t> row;
  dg::DevBuf<int> col;
  dg::DevBuf<double> val;
};

namespace dg {
namespace {

// bv: the states and Inv table already on the device (a dg_sb_basis); null: the model's host arrays.
dg_sb *sb_build(const dg_sb_model *m, const SbBasisView *bv) {
  DG_REQUIRE(m, DG_ERR_ARG, "null model");
  const int n = bv ? bv->n : m->n, d = m->dim_onsite;
  DG_REQUIRE(n > 0 && m->dim_LL > 0 && m->dim_RR > 0 && m->dim_onsite > 0, DG_ERR_ARG, "dimensions must be positive");
  if (bv)
    DG_REQUIRE(bv->dim_LL == m->dim_LL && bv->dim_RR == m->dim_RR && bv->d == m->dim_onsite, DG_ERR_ARG,
               "the model's dimensions (%d, %d, %d) differ from the basis' (%d, %d, %d)", m->dim_LL, m->dim_RR, m->dim_onsite,
               bv->dim_LL, bv->dim_RR, bv->d);
  else
    DG_REQUIRE(m->LL && m->LR && m->RR && m->RL && m->inv, DG_ERR_ARG, "null basis arrays");
  DG_REQUIRE(m->n_ops >= 1 && m->ops && m->n_terms >= 0 && (m->n_terms == 0 || m->terms), DG_ERR_ARG, "null operators/terms");
  const long dim_whole = (long)m->dim_LL * d * m->dim_RR * d;
  DG_REQUIRE(dim_whole < (1L << 40), DG_ERR_ARG, "Inv_LLLRRRRL too large");
  // basis states inside their position ranges (a device basis is in range by construction)
  for (int b = 0; !bv && b < n; ++b) {
    DG_REQUIRE(m->LL[b] >= 0 && m->LL[b] < m->dim_LL && m->LR[b] >= 0 && m->LR[b] < d && m->RR[b] >= 0 &&
                   m->RR[b] < m->dim_RR && m->RL[b] >= 0 && m->RL[b] < d,
               DG_ERR_ARG, "superblock state %d out of range", b);
  }
  // operators: validated against the dimension of every position they are used on
  std::vector<int> op_dim(m->n_ops, -1);
  long gen_bound = 0;
  auto width = [&](int o) {
    int w = 0;
    for (int r = 0; r < op_dim[o]; ++r) w = std::max(w, (int)(m->ops[o].Row[r + 1] - m->ops[o].Row[r]));
    return w;
  };
  for (int k = 0; k < m->n_terms; ++k) {
    const dg_sb_term &t = m->terms[k];
    DG_REQUIRE(t.pos1 >= 0 && t.pos1 < 4 && t.pos2 >= -1 && t.pos2 < 4 && t.pos1 != t.pos2, DG_ERR_ARG, "term %d: bad positions", k);
    DG_REQUIRE(t.op1 >= 0 && t.op1 < m->n_ops && (t.pos2 < 0 || (t.op2 >= 0 && t.op2 < m->n_ops)), DG_ERR_ARG,
               "term %d: operator index out of range", k);
    DG_REQUIRE((t.sign_mask & ~15) == 0 && (t.sign_mask == 0 || t.sign_even == 1 || t.sign_even == -1), DG_ERR_ARG,
               "term %d: bad sign", k);
    for (int p = 0; p < 4; ++p)
      if (t.sign_mask & (1 << p)) DG_REQUIRE(m->ele[p], DG_ERR_ARG, "term %d: sign needs ele[%d]", k, p);
    const int uses[2][2] = {{t.op1, t.pos1}, {t.pos2 >= 0 ? t.op2 : -1, t.pos2}};
    for (auto &u : uses) {
      if (u[0] < 0) continue;
      const int dim = position_dim(m, u[1]);
      DG_REQUIRE(op_dim[u[0]] < 0 || op_dim[u[0]] == dim, DG_ERR_ARG, "operator %d used on positions of different dimension", u[0]);
      op_dim[u[0]] = dim;
    }
  }
  for (int o = 0; o < m->n_ops; ++o) {
    if (op_dim[o] < 0) continue;
    const CRS1 &O = m->ops[o];
    DG_REQUIRE(O.Row && O.Row[0] == 0, DG_ERR_ARG, "operator %d: bad row offsets", o);
    for (int r = 0; r < op_dim[o]; ++r) {
      DG_REQUIRE(O.Row[r] <= O.Row[r + 1], DG_ERR_ARG, "operator %d: decreasing row offsets", o);
      for (long e = O.Row[r]; e < O.Row[r + 1]; ++e)
        DG_REQUIRE(O.Col[e] >= 0 && O.Col[e] < op_dim[o], DG_ERR_ARG, "operator %d: column out of range", o);
    }
  }
  for (int k = 0; k < m->n_terms; ++k) {
    const dg_sb_term &t = m->terms[k];
    gen_bound += (long)width(t.op1) * (t.pos2 >= 0 ? width(t.op2) : 1);
  }
  DG_REQUIRE(gen_bound < (1L << kGenBits), DG_ERR_ARG, "a row can generate %ld elements (limit %ld)", gen_bound, 1L << kGenBits);
  const int cap_need = (int)std::min<long>(gen_bound + 1, 1L << 30);
  DG_REQUIRE(cap_need <= 4096, DG_ERR_ARG, "a row can keep %d elements; at most 4096 are supported", cap_need);

  cudaStream_t st = stream();
  // device copies
  std::vector<int64_t> op_row;
  std::vector<int> op_row_base(m->n_ops, 0), op_first(m->n_ops, 0), op_col;
  std::vector<double> op_val;
  for (int o = 0; o < m->n_ops; ++o) {
    op_row_base[o] = (int)op_row.size();
    op_first[o] = (int)op_col.size();
    if (op_dim[o] < 0) {
      op_row.push_back(0);
      continue;
    }
    const CRS1 &O = m->ops[o];
    for (int r = 0; r <= op_dim[o]; ++r) op_row.push_back(O.Row[r]);
    for (long e = 0; e < O.Row[op_dim[o]]; ++e) {
      op_col.push_back(O.Col[e]);
      op_val.push_back(O.Val[e]);
    }
  }
  if (op_col.empty()) {
    op_col.push_back(0);
    op_val.push_back(0.0);
  }
  std::vector<SbTermDev> terms(m->n_terms);
  for (int k = 0; k < m->n_terms; ++k) {
    const dg_sb_term &t = m->terms[k];
    terms[k] = SbTermDev{t.pos1, t.pos2, t.op1, t.pos2 >= 0 ? t.op2 : 0, t.sign_mask, t.sign_even, t.coef};
  }
  DevBuf<short> sst[4];
  DevBuf<int> inv;
  if (!bv) {
    const short *hst[4] = {m->LL, m->LR, m->RR, m->RL};
    for (int p = 0; p < 4; ++p) {
      sst[p].alloc(n);
      DG_CUDA(cudaMemcpyAsync(sst[p].get(), hst[p], sizeof(short) * n, cudaMemcpyHostToDevice, st));
    }
    inv.alloc(dim_whole);
    DG_CUDA(cudaMemcpyAsync(inv.get(), m->inv, sizeof(int) * dim_whole, cudaMemcpyHostToDevice, st));
  }
  DevBuf<int> orb(op_row_base.size()), of(op_first.size()), oc(op_col.size()), err(1);
  DevBuf<int64_t> orow(op_row.size());
  DevBuf<double> ov(op_val.size());
  DevBuf<SbTermDev> td(std::max<size_t>(terms.size(), 1));
  DevBuf<int> ele[4];
  DG_CUDA(cudaMemcpyAsync(orb.get(), op_row_base.data(), sizeof(int) * op_row_base.size(), cudaMemcpyHostToDevice, st));
  DG_CUDA(cudaMemcpyAsync(of.get(), op_first.data(), sizeof(int) * op_first.size(), cudaMemcpyHostToDevice, st));
  DG_CUDA(cudaMemcpyAsync(oc.get(), op_col.data(), sizeof(int) * op_col.size(), cudaMemcpyHostToDevice, st));
  DG_CUDA(cudaMemcpyAsync(orow.get(), op_row.data(), sizeof(int64_t) * op_row.size(), cudaMemcpyHostToDevice, st));
  DG_CUDA(cudaMemcpyAsync(ov.get(), op_val.data(), sizeof(double) * op_val.size(), cudaMemcpyHostToDevice, st));
  if (!terms.empty())
    DG_CUDA(cudaMemcpyAsync(td.get(), terms.data(), sizeof(SbTermDev) * terms.size(), cudaMemcpyHostToDevice, st));
  SbDev dev{};
  dev.n = n;
  dev.dim_RR = m->dim_RR;
  dev.d = d;
  dev.n_terms = m->n_terms;
  for (int p = 0; p < 4; ++p) {
    dev.st[p] = bv ? bv->st[p] : sst[p].get();
    dev.ele[p] = nullptr;
    if (m->ele[p]) {
      const int dim = position_dim(m, p);
      ele[p].alloc(dim);
      DG_CUDA(cudaMemcpyAsync(ele[p].get(), m->ele[p], sizeof(int) * dim, cudaMemcpyHostToDevice, st));
      dev.ele[p] = ele[p].get();
    }
  }
  dev.inv = bv ? bv->inv : inv.get();
  dev.terms = td.get();
  dev.op_row = orow.get();
  dev.op_row_base = orb.get();
  dev.op_first = of.get();
  dev.op_col = oc.get();
  dev.op_val = ov.get();
  dev.zero = std::pow(10.0, -15.0);
  DG_CUDA(cudaMemsetAsync(err.get(), 0, sizeof(int), st));

  dg_sb *s = new dg_sb();
  try {
    s->n = n;
    DevBuf<long long> counts(n), tmp((n + kScanTile - 1) / kScanTile + 2);
    DevBuf<int64_t> soff(n + 1);
    DevBuf<int> most(1);
    // every row's generated elements: the scratch offsets, and the largest row, which sizes a warp's
    // buffer (the operators' widest rows seldom meet in one superblock row: 490 against a bound of
    // 960 on the Hubbard m=512 superblock, which doubles the warps a SM holds)
    DG_CUDA(cudaMemsetAsync(most.get(), 0, sizeof(int), st));
    k_sb_bounds<<<(int)std::max(1L, std::min<long>((n + kThreads - 1) / kThreads, (long)sm_count() * 8)), kThreads, 0, st>>>(
        dev, counts.get(), most.get()); ::dg::count_launch();
    DG_CUDA(cudaGetLastError());
    exclusive_scan(counts.get(), n, soff.get(), tmp.get(), st);
    int64_t bound = 0;
    int hmost = 0;
    DG_CUDA(cudaMemcpyAsync(&bound, soff.get() + n, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    DG_CUDA(cudaMemcpyAsync(&hmost, most.get(), sizeof(int), cudaMemcpyDeviceToHost, st));
    DG_CUDA(cudaStreamSynchronize(st));
    int cap = 32;
    while (cap < hmost) cap <<= 1;
    // warps a block bounded by 192 KB of shared memory (cap <= 4096: three warps at least); the limit is
    // set to that for every superblock, since all threads that build one share it
    constexpr size_t kMost = 192 << 10;
    const size_t per_warp = (size_t)cap * (sizeof(uint64_t) + sizeof(double));
    const int warps = (int)std::min<size_t>(kSbWarps, kMost / per_warp);
    const size_t smem = per_warp * warps;
    DG_CUDA(cudaFuncSetAttribute(k_sb_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMost));
    const long blocks = std::max(1L, std::min<long>((n + warps - 1) / warps, (long)sm_count() * 32));
    DevBuf<int> scol;
    DevBuf<double> sval;
    bool single = (size_t)bound * (sizeof(int) + sizeof(double)) <= kSbScratchBytes;
    if (single) {
      try {
        scol.alloc(bound);
        sval.alloc(bound);
      } catch (const Error &e) {   // no room for the scratch: the two passes need none
        if (e.code != DG_ERR_NOMEM) throw;
        cudaGetLastError();
        scol.release();
        single = false;
      }
    }
    k_sb_rows<<<(int)blocks, warps * 32, smem, st>>>(dev, cap, single ? soff.get() : (const int64_t *)nullptr, counts.get(), nullptr,
                                                        scol.get(), sval.get(), err.get()); ::dg::count_launch();
    DG_CUDA(cudaGetLastError());
    s->row.alloc(n + 1);
    exclusive_scan(counts.get(), n, s->row.get(), tmp.get(), st);
    int64_t total = 0;
    int herr = 0;
    DG_CUDA(cudaMemcpyAsync(&total, s->row.get() + n, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    DG_CUDA(cudaMemcpyAsync(&herr, err.get(), sizeof(int), cudaMemcpyDeviceToHost, st));
    DG_CUDA(cudaStreamSynchronize(st));
    DG_REQUIRE(herr == 0, DG_ERR_INTERNAL, "superblock row generation overflowed its buffer");
    s->nnz = total;
    auto take_result = [&] {
      s->col.alloc(total);
      s->val.alloc(total);
    };
    try {
      take_result();
    } catch (const Error &e) {
      if (e.code != DG_ERR_NOMEM || !single) throw;
      // no room for the result beside the scratch: it takes the scratch's place (a row keeps no more than it
      // generates) and the fill pass generates the rows again
      cudaGetLastError();
      s->col.release();
      scol.release();
      sval.release();
      soff.release();
      single = false;
      take_result();
    }
    if (single) {
      k_sb_compact<<<(int)std::max(1L, std::min<long>((n + kWarps - 1) / kWarps, (long)sm_count() * 16)), kThreads, 0, st>>>(
          n, soff.get(), s->row.get(), scol.get(), sval.get(), s->col.get(), s->val.get()); ::dg::count_launch();
      DG_CUDA(cudaGetLastError());
      DG_CUDA(cudaStreamSynchronize(st));
    } else {
      k_sb_rows<<<(int)blocks, warps * 32, smem, st>>>(dev, cap, nullptr, nullptr, s->row.get(), s->col.get(), s->val.get(),
                                                          err.get()); ::dg::count_launch();
      DG_CUDA(cudaGetLastError());
      DG_CUDA(cudaMemcpyAsync(&herr, err.get(), sizeof(int), cudaMemcpyDeviceToHost, st));
      DG_CUDA(cudaStreamSynchronize(st));
      DG_REQUIRE(herr == 0, DG_ERR_INTERNAL, "superblock fill pass disagreed with the count pass (%d)", herr);
    }
  } catch (...) {
    delete s;
    throw;
  }
  return s;
}

}  // namespace
}  // namespace dg

using namespace dg;

extern "C" {

int dg_sb_build(const dg_sb_model *model, dg_sb **out) {
  return guarded([&] {
    require_device();
    DG_REQUIRE(out, DG_ERR_ARG, "null argument");
    *out = nullptr;
    *out = sb_build(model, nullptr);
  });
}

int dg_sb_build_with_basis(const dg_sb_model *model, const dg_sb_basis *basis, dg_sb **out) {
  return guarded([&] {
    require_device();
    DG_REQUIRE(out && basis, DG_ERR_ARG, "null argument");
    *out = nullptr;
    DG_REQUIRE(basis->inv_len == (long)basis->dim_LL * basis->d * basis->dim_RR * basis->d, DG_ERR_ARG,
               "the basis carries no full Inv_LLLRRRRL table");
    const SbBasisView bv{basis->n, basis->dim_LL, basis->dim_RR, basis->d,
                         {basis->st[0].get(), basis->st[1].get(), basis->st[2].get(), basis->st[3].get()}, basis->inv.get()};
    *out = sb_build(model, &bv);
  });
}

int dg_sb_info(const dg_sb *s, int *n, long *nnz) {
  return guarded([&] {
    DG_REQUIRE(s, DG_ERR_ARG, "null superblock");
    if (n) *n = s->n;
    if (nnz) *nnz = s->nnz;
  });
}

int dg_sb_download(const dg_sb *s, long *row, int *col, double *val) {
  return guarded([&] {
    DG_REQUIRE(s, DG_ERR_ARG, "null superblock");
    cudaStream_t st = stream();
    if (row) DG_CUDA(cudaMemcpyAsync(row, s->row.get(), sizeof(int64_t) * (s->n + 1), cudaMemcpyDeviceToHost, st));
    if (col) DG_CUDA(cudaMemcpyAsync(col, s->col.get(), sizeof(int) * s->nnz, cudaMemcpyDeviceToHost, st));
    if (val) DG_CUDA(cudaMemcpyAsync(val, s->val.get(), sizeof(double) * s->nnz, cudaMemcpyDeviceToHost, st));
    DG_CUDA(cudaStreamSynchronize(st));
  });
}

int dg_sb_matrix(const dg_sb *s, int values, dg_matrix **out) {
  return guarded([&] {
    require_device();
    DG_REQUIRE(s && out, DG_ERR_ARG, "null argument");
    *out = matrix_from_device(s->n, s->nnz, reinterpret_cast<const long *>(s->row.get()), s->col.get(), s->val.get(),
                              DG_STORE_LOWER_DIAG_LAST, values, stream(), true);
  });
}

void dg_sb_free(dg_sb *s) { delete s; }

}  // extern "C"
