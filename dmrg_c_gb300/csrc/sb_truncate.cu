// sb_truncate.cu -- truncation of the LL+LR block after a superblock solve
// (DMRG_GET_SYSTEM_INFO_Q1 / _Q2 / _Q3, dmrg/DMRG_GET_SYSTEM_INFO_Q1.c:8-213, with
// DMRG_GET_DENSITY_MATRIX_INFO_Q1..Q3 and DMRG_GET_DENSITY_MATRIX).
//
// The LLLR pairs come in blocks of equal quantum numbers.  Block g's density matrix is
// rho_g = X_g X_g^T, row p of X_g being the superblock-vector entries of the states of pair p
// (every pair of a block has the same number of states, listed with the same (RR, RL) pairs).
// On the device: every block's rho_g (entries summed in the reference's order, so bitwise its
// density matrices), then every block's eigen-decomposition at once -- a cyclic Jacobi
// eigensolver, one thread block per density block, the rotations of one round (a round-robin
// pairing of the indices) applied together.  On the host: the reference's ordering rules --
// eigenvalues in ascending order inside a block (as LAPACK's dsyev returns them), a stable sort
// of all of them in descending order, the kept dimension (no cut inside a degenerate multiplet,
// nothing at or below 1e-15), a stable sort of the kept states by their quantum numbers -- and
// the transformation matrix (CCS) and its transpose (CRS), allocated as the reference's
// GET_CCS1 / GET_CRS1 allocate them so that DMRG_FREE_SYSTEM_INFO releases them.
//
// Eigenvalues agree with LAPACK's to ~1e-16 * ||rho||; eigenvectors are the same up to sign (and
// to a rotation inside a degenerate multiplet, which the cut keeps whole).
#include <algorithm>
#include <chrono>
#include <climits>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <numeric>
#include <vector>

#include <cooperative_groups.h>

#include "common.cuh"

namespace dg {
namespace {

constexpr int kJacobiMaxN = 1024;    // bound of the per-round rotation arrays
constexpr int kJacobiSweeps = 60;    // cap on sweeps (convergence takes ~6-10)
constexpr size_t kJacobiSmem = 200 * 1024;   // dynamic shared memory a CTA may take for its rows
constexpr int kJacobiSmemN = 384;            // no block above it fits (n = 368 is the last)
constexpr int kJacobiAhead = 112;            // pairs from which the rotations are formed ahead
constexpr size_t kJacobiAlone = 116 * 1024;  // dynamic shared memory with which a CTA has its SM for itself

struct GramBlk {
  int64_t x_off, a_off;   // X_g (P x Q, row-major) and rho_g (P x P) offsets
  int P, Q;
};

__device__ __forceinline__ int find_blk(const int64_t *__restrict__ off, int B, int64_t e) {
  int lo = 0, hi = B - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (off[mid] <= e)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

// rho_g[p][q] = sum_t X_g[p][t] * X_g[q][t] for p <= q, in t order, rounded as written; mirrored.
__global__ void __launch_bounds__(kThreads) k_gram_batched(const double *__restrict__ X, const GramBlk *__restrict__ blks,
                                                          const int64_t *__restrict__ a_pre, int nb, double *__restrict__ A) {
  const int64_t total = a_pre[nb];
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int g = find_blk(a_pre, nb, e);
    const GramBlk b = blks[g];
    const int64_t loc = e - b.a_off;
    const int p = (int)(loc / b.P), q = (int)(loc - (int64_t)p * b.P);
    if (p > q) continue;
    const double *__restrict__ x = X + b.x_off + (int64_t)p * b.Q;
    const double *__restrict__ y = X + b.x_off + (int64_t)q * b.Q;
    double acc = 0.0;
    for (int t = 0; t < b.Q; ++t) acc = __dadd_rn(acc, __dmul_rn(x[t], y[t]));
    A[b.a_off + (int64_t)p * b.P + q] = acc;
    A[b.a_off + (int64_t)q * b.P + p] = acc;
  }
}

struct EigBlk {
  int64_t off;    // A_g and V_g (n x n, row-major)
  int64_t woff;   // eigenvalues
  int n;
};

// The plane rotation (c, s) of a pair (x, y), rounded the same wherever it is applied.
__device__ __forceinline__ double rot_p(double2 cs, double x, double y) { return __fma_rn(cs.x, x, -__dmul_rn(cs.y, y)); }
__device__ __forceinline__ double rot_q(double2 cs, double x, double y) { return __fma_rn(cs.y, x, __dmul_rn(cs.x, y)); }

// Round-robin pairing of m indices (m even) in round r of m - 1: pair 0 is (r, m-1), pair k the
// indices r + k and r - k modulo m - 1.
__device__ __forceinline__ int2 rr_pair(int m, int r, int k) {
  if (k == 0) return make_int2(r, m - 1);
  int p = r + k, q = r - k;
  if (p >= m - 1) p -= m - 1;
  if (q < 0) q += m - 1;
  return make_int2(min(p, q), max(p, q));
}
// (pair, partner) of index i.
__device__ __forceinline__ int2 rr_of(int m, int r, int i) {
  if (i == r) return make_int2(0, m - 1);
  if (i == m - 1) return make_int2(0, r);
  int k = i - r, o = 2 * r - i;
  if (k < 0) k += m - 1;
  if (o < 0) o += m - 1;
  if (o >= m - 1) o -= m - 1;
  return make_int2(k < m / 2 ? k : m - 1 - k, o);
}

// Cyclic Jacobi on every block, one thread-block cluster of cs CTAs a block: A_g -> diag
// (eigenvalues in W), V_g's columns the eigenvectors.  CTA c keeps rows [c*rp, (c+1)*rp) of A_g (two
// copies: the current one and the next) and of V_g in its shared memory (rp = ceil(n / cs)), so a
// block's FP64 work spreads over cs SMs.  A sweep is m-1 rounds (m = n rounded up to even) of the
// round-robin pairing; a round applies its m/2 disjoint rotations J at once, A' = J^T A J:
//   1. every CTA writes its rows of A' into the next copy -- row i of A' needs row i and the row
//      paired with i (read through distributed shared memory when another CTA keeps it) -- and
//      rotates the columns of its rows of V in place;
//   2. meanwhile (blocks of kJacobiAhead pairs or more) the last CTA, which keeps no rows (workers =
//      cs - 1), forms the next round's rotations, a thread each: the three entries of A' it needs, straight from the current copy
//      with the round's rotations (the same operations as 1, so the same bits), then the rotation,
//      written to every CTA of the cluster (small blocks: every CTA forms all rotations of a round
//      itself, before 1);
//   3. one cluster barrier, after which the copies swap.  A round without a rotation leaves A and V
//      as they are: it skips 1 and keeps the copy.
// FP64 issue bounds a round: 12 instructions a pair of entries, ~20 cycles each a warp; at n = 199
// that is ~10 k cycles a SM.  A rotation (three divisions, two square roots) is a chain of ~7 k cycles
// that every instruction of the update delays, so it has a SM of its own.  Measured per round at
// n = 199: 24 k cycles with every CTA forming every rotation before its update, 16 k with each CTA
// forming its share on a warp beside the update, ~14 k like this.
// Entries at or below 1e-18 of the Frobenius norm are not rotated away.  The sweep loop stops when
// the off-diagonal part is below 1e-16 of the norm or a sweep found nothing to rotate (decided by
// CTA 0 and broadcast, so every CTA leaves together), or after max_sweeps (sweeps[g] reports the
// count).  Blocks are in descending size.
constexpr int kJacThreads = 512;   // threads a CTA when a large block has its SMs for itself, else kThreads

template <bool GMEM, int threads>
__global__ void __launch_bounds__(threads, threads == kThreads ? 5 : 1) k_jacobi_cluster(const EigBlk *__restrict__ blks, const double *__restrict__ Ag,
                                                               double *__restrict__ Vg, double *__restrict__ Wg, int workers,
                                                               int max_sweeps, int *__restrict__ sweeps, double *gwork, int64_t gstride) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int cs = (int)cluster.num_blocks();
  const int rank = (int)cluster.block_rank();
  extern __shared__ double sm_jac[];
  constexpr int kMaxN = GMEM ? kJacobiMaxN : kJacobiSmemN;
  __shared__ double2 rot[2][kMaxN / 2];   // (c, s) of the pairs: this round's and the next's
  __shared__ int pair_pq[2][kMaxN / 2];   // the round's pairs, lower index + higher << 16
  __shared__ int of_index[2][kMaxN];      // each index's pair + partner << 16
  __shared__ const double *partner_row[2][kMaxN / 7 + 1];   // the rows paired with this CTA's
  __shared__ int s_any[3];                      // the round rotates something: this, next, the one after (cleared)
  __shared__ double s_part[2 * 16];
  __shared__ double s_sum[kThreads];
  __shared__ int s_done, s_rot;
  __shared__ double s_tol;
  const int tid = threadIdx.x, lane = tid & 31;
  const EigBlk b = blks[blockIdx.x / cs];
  const int n = b.n;
  if (n <= 0) return;   // the whole cluster sees the same block
  // rows over the first `workers` CTAs: cs - 1, or cs when the block fits no fewer
  const int rows = (n + workers - 1) / workers;
  const int r0 = min(n, rank * rows), r1 = min(n, r0 + rows), nloc = r1 - r0;
  const int64_t slab = (int64_t)rows * n;
  const bool ahead = workers < cs;
  const int owner_of = (1 << 20) / rows + 1;
  // this CTA's rows: in shared memory, or (GMEM, blocks too large for it) in the global workspace
  // gwork, gstride doubles a CTA
  double *const mine = GMEM ? gwork + (int64_t)blockIdx.x * gstride : sm_jac;
  double *V = mine + 2 * slab;
  for (int64_t e = tid; e < (int64_t)nloc * n; e += threads) {
    const int64_t i = r0 + e / n, j = e % n;
    mine[e] = Ag[b.off + i * n + j];
    V[e] = i == j ? 1.0 : 0.0;
  }
  int cur = 0;   // the copy holding the current A
  const int m = n + (n & 1), half = m / 2;
  auto row_at = [&](int i, int copy) -> const double * {   // row i of a copy of A, in whichever CTA keeps it
    const int owner = (i * owner_of) >> 20;   // i / rows for i < 1024
    const double *base =
        GMEM ? gwork + (int64_t)(blockIdx.x - rank + owner) * gstride : cluster.map_shared_rank(sm_jac, owner);
    return base + copy * slab + (int64_t)(i - owner * rows) * n;
  };
  auto row_ptr = [&](int i) { return row_at(i, cur); };
  // The tables of round r, whose current copy is `copy`, by all threads, the last first (in a small
  // block the row update leaves them idle): looked up they cost one shared-memory read an element,
  // worked out in the row update ~30 integer instructions (a 199-pair block 32 -> 45 ms).
  auto tables = [&](int r, int copy) {
    const int back = threads - 1 - tid;
    for (int i = back; i < m; i += threads) {
      const int2 o = rr_of(m, r, i);
      of_index[r & 1][i] = o.x | (o.y << 16);
    }
    for (int k = back; k < m / 2; k += threads) {
      const int2 o = rr_pair(m, r, k);
      pair_pq[r & 1][k] = o.x | (o.y << 16);
    }
    for (int li = back; li < nloc; li += threads) {
      const int o = rr_of(m, r, r0 + li).y;
      partner_row[r & 1][li] = row_at(o < n ? o : r0 + li, copy);
    }
  };
  // a value of another CTA's rows (global workspace: read from L2, where the writer's stores are
  // visible after the cluster barrier)
  auto rd = [&](const double *p) { return GMEM ? __ldcg(p) : *p; };
  // the sum of the first kThreads threads' values, valid in thread 0 (block_sum's order)
  auto sum = [&](double v) {
    __syncthreads();
    if (tid < kThreads) s_sum[tid] = v;
    __syncthreads();
    double r = 0.0;
    if (tid < 32) {
      const double *c = s_sum + tid;
      r = warp_sum(((c[0] + c[32]) + (c[64] + c[96])) + ((c[128] + c[160]) + (c[192] + c[224])));
    }
    return r;
  };
  // Entries (p, p), (q, q) and (p, q) of A' = J^T A J with the rotations of round r (of A itself when
  // r < 0), by the operations of the row update below.  Every operand is read up front and every
  // alternative selected, not branched to: the lanes' pairs take different ones, and this is the
  // head of the round's longest chain.
  auto entries = [&](int r, int p, int q, double &app, double &aqq, double &apq) {
    if (r < 0) {
      app = rd(row_ptr(p) + p);
      aqq = rd(row_ptr(q) + q);
      apq = rd(row_ptr(p) + q);
      return;
    }
    const int op = of_index[r & 1][p], oq = of_index[r & 1][q];
    const int2 kp = make_int2(op & 0xffff, op >> 16), kq = make_int2(oq & 0xffff, oq >> 16);
    const double2 *const rt = rot[r & 1];
    const double2 cp = rt[kp.x], cq = rt[kq.x];
    // each index with its partner of round r, lower index first (a dummy partner stands for itself)
    const int pp = kp.y < n ? kp.y : p, qq = kq.y < n ? kq.y : q;
    const int p0 = min(p, pp), p1 = max(p, pp), q0 = min(q, qq), q1 = max(q, qq);
    const double *rp = row_ptr(p), *rpp = row_ptr(pp), *rq = row_ptr(q), *rqq = row_ptr(qq);
    const double x0 = rd(rp + p0), x1 = rd(rp + p1), y0 = rd(rpp + p0), y1 = rd(rpp + p1);   // row p, its partner row: columns of p's pair
    const double u0 = rd(rp + q0), u1 = rd(rp + q1), v0 = rd(rpp + q0), v1 = rd(rpp + q1);   // the same rows: columns of q's pair
    const double z0 = rd(rq + q0), z1 = rd(rq + q1), w0 = rd(rqq + q0), w1 = rd(rqq + q1);   // row q, its partner row: columns of q's pair
    const bool p_low = p < kp.y, q_low = q < kq.y;
    auto rows2 = [](double2 cs, bool low, double x, double y) {   // the row rotation of one entry
      const double t = low ? rot_p(cs, x, y) : rot_q(cs, y, x);
      return cs.y == 0.0 ? x : t;
    };
    auto cols2 = [](double2 cs, bool low, double a0, double a1) {   // the column rotation of two
      const double t = low ? rot_p(cs, a0, a1) : rot_q(cs, a0, a1);
      return cs.y == 0.0 ? (low ? a0 : a1) : t;
    };
    app = cols2(cp, p_low, rows2(cp, p_low, x0, y0), rows2(cp, p_low, x1, y1));
    aqq = cols2(cq, q_low, rows2(cq, q_low, z0, w0), rows2(cq, q_low, z1, w1));
    apq = cols2(cq, q_low, rows2(cp, p_low, u0, v0), rows2(cp, p_low, u1, v1));
    if (kp.x == kq.x && cq.y != 0.0) apq = 0.0;   // p and q were a pair of round r: annihilated
  };
  // The rotation that annihilates apq, (1, 0) and false where it is at or below the tolerance.
  auto rotation = [&](double app, double aqq, double apq, double2 &cs2) {
    if (!(fabs(apq) > s_tol)) return false;
    const double th = (aqq - app) / (2.0 * apq);
    const double t = (th >= 0.0 ? 1.0 : -1.0) / (fabs(th) + sqrt(__fma_rn(th, th, 1.0)));
    cs2.x = 1.0 / sqrt(__fma_rn(t, t, 1.0));
    cs2.y = t * cs2.x;
    return true;
  };
  // AHEAD: the rotations of round r, from A after round r - 1 (r = 0: from A as it is), to every CTA: a
  // thread per pair of the last CTA.
  auto rotations_ahead = [&](int r) {
    for (int k0 = tid & ~31; k0 < half; k0 += threads) {
      const int k = k0 + lane;
      const int2 pq = rr_pair(m, r, min(k, half - 1));
      double2 cs2 = make_double2(1.0, 0.0);
      bool turns = false;
      if (k < half && pq.y < n) {
        double app, aqq, apq;
        entries(r - 1, pq.x, pq.y, app, aqq, apq);
        turns = rotation(app, aqq, apq, cs2);
      }
      if (k < half)
        for (int c = 0; c < cs; ++c) cluster.map_shared_rank(rot[r & 1], c)[k] = cs2;
      if (__any_sync(0xffffffffu, turns)) {
        if (lane < cs) *cluster.map_shared_rank(&s_any[r % 3], lane) = 1;
        if (lane == 0) *cluster.map_shared_rank(&s_rot, 0) = 1;
      }
    }
  };
  // Not AHEAD: the rotations of round r from the current A, by every CTA for itself; true if any turns.
  auto rotations_now = [&](int r) -> bool {
    bool turns = false;
    for (int k = tid; k < half; k += threads) {
      const int o = pair_pq[r & 1][k];
      const int2 pq = make_int2(o & 0xffff, o >> 16);
      double2 cs2 = make_double2(1.0, 0.0);
      if (pq.y < n) {
        const double *rp = row_ptr(pq.x);
        if (rotation(rd(rp + pq.x), rd(row_ptr(pq.y) + pq.y), rd(rp + pq.y), cs2)) turns = true;
      }
      rot[r & 1][k] = cs2;
    }
    return __syncthreads_or(turns) != 0;
  };
  if (tid == 0) s_rot = 1;
  cluster.sync();
  int sweep = 0;
  for (; sweep < max_sweeps; ++sweep) {
    const double *A = mine + cur * slab;
    double off = 0.0, tot = 0.0;
    if (tid < kThreads)
      for (int64_t e = tid; e < (int64_t)nloc * n; e += kThreads) {
        const double a = A[e];
        tot += a * a;
        if (r0 + e / n != e % n) off += a * a;
      }
    off = sum(off);
    tot = sum(tot);
    if (tid == 0) {
      double *p0 = cluster.map_shared_rank(s_part, 0);
      p0[2 * rank] = off;
      p0[2 * rank + 1] = tot;
      s_any[0] = s_any[1] = s_any[2] = 0;
    }
    cluster.sync();
    if (rank == 0 && tid == 0) {
      double o = 0.0, t = 0.0;
      for (int c = 0; c < cs; ++c) {
        o += s_part[2 * c];
        t += s_part[2 * c + 1];
      }
      // done when the off-diagonal part is negligible, or when the last sweep found nothing to
      // rotate (every |A[p][q]| at or below 1e-18 of the norm)
      const int done = o <= 1e-32 * t || !s_rot;
      const double tol = 1e-18 * sqrt(t);
      for (int c = 0; c < cs; ++c) {
        *cluster.map_shared_rank(&s_done, c) = done;
        *cluster.map_shared_rank(&s_tol, c) = tol;
      }
      s_rot = 0;   // set by the CTAs that find a rotation
    }
    cluster.sync();
    if (s_done) break;
    tables(0, cur);
    if (ahead) {
      if (rank == cs - 1) rotations_ahead(0);
      cluster.sync();
    } else {
      __syncthreads();
    }
    for (int r = 0; r < m - 1; ++r) {
      bool any;   // the round turns something: the same in every CTA
      if (ahead) {
        any = s_any[r % 3] != 0;
        if (tid == 0) s_any[(r + 2) % 3] = 0;   // read last round, written next round
        if (rank == cs - 1 && r + 1 < m - 1) rotations_ahead(r + 1);
      } else {
        any = rotations_now(r);
        if (any && rank == 0 && tid == 0) s_rot = 1;
      }
      if (r + 1 < m - 1) tables(r + 1, any ? cur ^ 1 : cur);
      if (!any && !ahead) {   // nobody writes: the next round's tables are all there is to wait for
        __syncthreads();
        continue;
      }
      if (any) {
        // this CTA's rows of A' = J^T A J into the next copy; its rows of V rotated in place
        const double *Acur = mine + cur * slab;
        double *Anext = mine + (cur ^ 1) * slab;
        const double2 *const rt = rot[r & 1];
        const int step_li = threads / half, step_l = threads - step_li * half;
        int li = tid / half, l = tid - li * half;
        for (int idx = tid; idx < nloc * half; idx += threads) {
          const int i = r0 + li;
          const int oi = of_index[r & 1][i], ki = oi & 0xffff, pq = pair_pq[r & 1][l];
          const double2 ri = rt[ki], rl = rt[l];
          const bool i_is_p = i < (oi >> 16);
          const double *ai = Acur + (int64_t)li * n;
          const double *ap = partner_row[r & 1][li];
          const int pl = pq & 0xffff, ql = pq >> 16;
          // row rotation of row i at columns pl (and ql)
          auto rowrot = [&](int j) {
            if (ri.y == 0.0) return ai[j];
            const double y = rd(ap + j);
            return i_is_p ? rot_p(ri, ai[j], y) : rot_q(ri, y, ai[j]);
          };
          double *out = Anext + (int64_t)li * n;
          const double xp = rowrot(pl);
          if (ql >= n) {
            out[pl] = xp;
          } else {
            const double xq = rowrot(ql);
            if (rl.y == 0.0) {
              out[pl] = xp;
              out[ql] = xq;
            } else {
              out[pl] = rot_p(rl, xp, xq);
              out[ql] = rot_q(rl, xp, xq);
              if (ki == l) out[i_is_p ? ql : pl] = 0.0;   // the entry this rotation annihilates
              double *v = V + (int64_t)li * n;
              const double u = v[pl], w = v[ql];
              v[pl] = rot_p(rl, u, w);
              v[ql] = rot_q(rl, u, w);
            }
          }
          li += step_li;
          l += step_l;
          if (l >= half) {
            l -= half;
            ++li;
          }
        }
      }
      cluster.sync();   // every CTA has written its next rows and rotations and read the current ones
      if (any) cur ^= 1;
    }
  }
  // The last rounds of the last sweep may have been idle ones, without a barrier: no CTA leaves while
  // another still reads its rows.
  cluster.sync();
  const double *A = mine + cur * slab;
  for (int i = tid; i < nloc; i += threads) Wg[b.woff + r0 + i] = A[(int64_t)i * n + r0 + i];
  for (int64_t e = tid; e < (int64_t)nloc * n; e += threads) Vg[b.off + (int64_t)r0 * n + e] = V[e];
  if (rank == 0 && tid == 0) sweeps[blockIdx.x / cs] = sweep;
}

[[noreturn]] void fatal(const char *who, const char *msg) {
  printf("Error in %s\n%s\n", who, msg);
  fflush(stdout);
  exit(1);
}

template <class T>
T *c_array(size_t n) {   // zero-filled, released with free() as the reference's GET_ARRAY_* arrays are
  T *p = static_cast<T *>(std::calloc(std::max<size_t>(n, 1), sizeof(T)));
  if (!p) fatal("DMRG_GET_SYSTEM_INFO", "host allocation failed");
  return p;
}

double wall_s() {
  return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

// The reference's DMRG_GET_SYSTEM_INFO_Q<nq>: qn[0..nq) are the LLLR pairs' quantum numbers.
DMRG_SYSTEM_INFO *system_info(int nq, const int *const *qn, DMRG_BASIS *B, const double *Vec, int max_dim, DMRG_TIME *T) {
  const double t0 = wall_s();
  char who_info[64], who_tm[64], msg[400];
  snprintf(who_info, sizeof(who_info), "DMRG_GET_DENSITY_MATRIX_INFO_Q%d", nq);
  snprintf(who_tm, sizeof(who_tm), "DMRG_MAKE_TRANSFORMATION_MATRIX_Q%d at Check Point", nq);
  const int dim_LLLR = B->dim_LLLR;
  if (dim_LLLR <= 0) {
    snprintf(msg, sizeof(msg), "dim_LLLR = %d", dim_LLLR);
    fatal(who_info, msg);
  }
  // blocks: runs of equal quantum numbers, which must ascend lexicographically
  auto key_less = [&](int a, int b) {
    for (int k = 0; k < nq; ++k)
      if (qn[k][a] != qn[k][b]) return qn[k][a] < qn[k][b];
    return false;
  };
  std::vector<int> blk_start{0};
  for (int i = 0; i + 1 < dim_LLLR; ++i) {
    if (key_less(i + 1, i)) {
      snprintf(msg, sizeof(msg), "Q_Number_LLLR[%d] > Q_Number_LLLR[%d]", i, i + 1);
      fatal(who_info, msg);
    }
    if (key_less(i, i + 1)) blk_start.push_back(i + 1);
  }
  blk_start.push_back(dim_LLLR);
  const int nb = (int)blk_start.size() - 1;
  // superblock states of each pair (DMRG_GET_DENSITY_MATRIX's checks)
  std::vector<long> base((size_t)dim_LLLR + 1, 0);
  for (int i = 0; i < dim_LLLR; ++i) base[i + 1] = base[i] + B->Sum_LLLR[i];
  if (base[dim_LLLR] != B->dim_LLLRRRRL) {
    snprintf(msg, sizeof(msg), "Base_LLLR[%d] (%ld) != dim_LLLRRRRL (%d)", dim_LLLR, base[dim_LLLR], B->dim_LLLRRRRL);
    fatal("DMRG_GET_DENSITY_MATRIX", msg);
  }
  const int d = B->dim_onsite, dim_RR = B->dim_RR;
  std::vector<GramBlk> gb(nb);
  std::vector<EigBlk> eb(nb);
  std::vector<int64_t> a_pre(nb + 1, 0);
  int64_t xs = 0, woff = 0;
  int max_n = 0;
  for (int g = 0; g < nb; ++g) {
    const int P = blk_start[g + 1] - blk_start[g], Q = B->Sum_LLLR[blk_start[g]];
    gb[g] = GramBlk{xs, a_pre[g], P, Q};
    eb[g] = EigBlk{a_pre[g], woff, P};
    a_pre[g + 1] = a_pre[g] + (int64_t)P * P;
    xs += (int64_t)P * Q;
    woff += P;
    max_n = std::max(max_n, P);
  }
  if (max_n > kJacobiMaxN) {
    snprintf(msg, sizeof(msg), "a density-matrix block of %d pairs exceeds %d", max_n, kJacobiMaxN);
    fatal("DMRG_GET_SYSTEM_INFO", msg);
  }
  std::vector<double> X((size_t)std::max<int64_t>(xs, 1));
  for (int g = 0; g < nb; ++g) {
    const int r0 = blk_start[g], P = gb[g].P, Q = gb[g].Q;
    for (int r = 0; r < P; ++r) {
      const int rb = r0 + r;
      if (B->Sum_LLLR[rb] != Q) {
        snprintf(msg, sizeof(msg), "Sum_LLLR[%d] (%d) != Sum_LLLR[%d] (%d)", r0, Q, rb, B->Sum_LLLR[rb]);
        fatal("DMRG_GET_DENSITY_MATRIX", msg);
      }
      const int ll = B->LL_LLLR[rb], lr = B->LR_LLLR[rb];
      for (int t = 0; t < Q; ++t) {
        const long sr = base[rb] + t, s0 = base[r0] + t;
        const int rr = B->RR_LLLRRRRL[sr], rl = B->RL_LLLRRRRL[sr];
        if (rr != B->RR_LLLRRRRL[s0] || rl != B->RL_LLLRRRRL[s0]) {
          snprintf(msg, sizeof(msg), "RR_row (%d) != RR_col (%d) || RL_row (%d) != RL_col (%d)", B->RR_LLLRRRRL[s0], rr,
                   B->RL_LLLRRRRL[s0], rl);
          fatal("DMRG_GET_DENSITY_MATRIX", msg);
        }
        const int inv = B->Inv_LLLRRRRL[(long)ll * d * dim_RR * d + (long)lr * dim_RR * d + (long)rr * d + rl];
        if (inv < 0) {
          snprintf(msg, sizeof(msg), "inv_row (%d) < 0", inv);
          fatal("DMRG_GET_DENSITY_MATRIX", msg);
        }
        X[gb[g].x_off + (int64_t)r * Q + t] = Vec[inv];
      }
    }
  }
  const double t_gather = wall_s();
  // device: density matrices and their eigen-decompositions
  std::vector<double> W((size_t)std::max<int64_t>(woff, 1)), Vh((size_t)std::max<int64_t>(a_pre[nb], 1));
  std::vector<int> sweeps(nb);
  int cs_used = 0;
  const int rc = guarded([&] {
    require_device();
    cudaStream_t st = stream();
    DevBuf<double> dX(X.size()), dA(Vh.size()), dV(Vh.size()), dW(W.size());
    DevBuf<GramBlk> dgb(nb);
    DevBuf<EigBlk> deb(nb);
    DevBuf<int64_t> dpre(nb + 1);
    DevBuf<int> dsw(nb);
    DG_CUDA(cudaMemcpyAsync(dX.get(), X.data(), sizeof(double) * X.size(), cudaMemcpyHostToDevice, st));
    DG_CUDA(cudaMemcpyAsync(dgb.get(), gb.data(), sizeof(GramBlk) * nb, cudaMemcpyHostToDevice, st));
    DG_CUDA(cudaMemcpyAsync(dpre.get(), a_pre.data(), sizeof(int64_t) * (nb + 1), cudaMemcpyHostToDevice, st));
    const int64_t total = a_pre[nb];
    if (total > 0) {
      const long grid = std::max(1L, std::min<long>((total + kThreads - 1) / kThreads, (long)sm_count() * 8));
      k_gram_batched<<<(int)grid, kThreads, 0, st>>>(dX.get(), dgb.get(), dpre.get(), nb, dA.get());
      count_launch();
      DG_CUDA(cudaGetLastError());
    }
    // one cluster a block, the largest blocks first
    // shared memory of a CTA whose cluster spreads a block of mn pairs over w CTAs
    auto smem_for = [&](int w, int mn) { return 3 * sizeof(double) * (size_t)((mn + w - 1) / w) * mn; };
    std::vector<int> by_size(nb);
    std::iota(by_size.begin(), by_size.end(), 0);
    std::stable_sort(by_size.begin(), by_size.end(), [&](int a, int b) { return eb[a].n > eb[b].n; });
    std::vector<EigBlk> eb_sorted(nb);
    for (int i = 0; i < nb; ++i) eb_sorted[i] = eb[by_size[i]];
    DG_CUDA(cudaMemcpyAsync(deb.get(), eb_sorted.data(), sizeof(EigBlk) * nb, cudaMemcpyHostToDevice, st));
    DG_CUDA(cudaMemsetAsync(dsw.get(), 0, sizeof(int) * nb, st));
    // Blocks whose rows do not fit 16 CTAs' shared memory (a prefix of the sorted list) keep them in
    // a global workspace sized for them alone; the others run from shared memory in a second launch,
    // so one large block does not send every block to global memory.
    int n_gmem = 0;
    while (n_gmem < nb && smem_for(16, eb_sorted[n_gmem].n) > kJacobiSmem) ++n_gmem;
    DevBuf<double> gwork;
    auto launch_part = [&](int first, int count, bool gmem) {
      if (count <= 0) return;
      const int mn = eb_sorted[first].n;
      // 16 CTAs a cluster (a non-portable size) when the part's largest block has 64 pairs or
      // more and the device runs such clusters, else 8
      int cs = 8;
      // A few large blocks bound the part's time, or many of the same size do (a block costs n^3).  In
      // the first case (the density blocks of a DMRG step: 30-46 blocks worth 4-5 times the largest)
      // every cluster takes whole SMs, so that the largest waits for nobody's FP64 instructions; about
      // six clusters of 16 CTAs then run at once.  In the second the CTAs share the SMs.  Eight blocks
      // of 128 pairs: 2.1 ms alone and in two waves 4.2, shared 3.0; Hubbard m=512 (largest 199):
      // 30.5 ms shared, 27.1 alone (with the rotations on a warp of each CTA).
      double cubes = 0.0;
      for (int i = first; i < first + count; ++i) cubes += std::pow((double)eb_sorted[i].n, 3.0);
      const bool alone = mn >= 64 && cubes <= sm_count() / 24 * std::pow((double)mn, 3.0);
      auto kernel = gmem ? (alone ? k_jacobi_cluster<true, kJacThreads> : k_jacobi_cluster<true, kThreads>)
                         : (alone ? k_jacobi_cluster<false, kJacThreads> : k_jacobi_cluster<false, kThreads>);
      DG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(gmem ? kJacobiAlone : kJacobiSmem)));
      if (mn >= 64 && cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) cs = 16;
      cudaGetLastError();
      if (!gmem && smem_for(8, mn) > kJacobiSmem) cs = 16;
      for (;;) {
        cudaLaunchConfig_t cfg;
        std::memset(&cfg, 0, sizeof(cfg));
        cfg.gridDim = dim3((unsigned)(count * cs));
        cfg.blockDim = dim3(alone ? kJacThreads : kThreads);
        // Alone and from 112 pairs on the last CTA forms the rotations ahead of the round and keeps no
        // rows (unless the largest block fits only 16 CTAs' shared memory): a round is then bound by
        // the update's FP64 issue.  Below, the update is shorter than a rotation's chain and each CTA
        // forms all rotations itself.  Measured, ahead against now, 16 CTAs: largest block 199 25.7 /
        // 31.7 ms, 122 9.7 / 10.1, 96 7.6 / 7.2, 65 4.1 / 3.7; 8 CTAs: 40 1.50 / 1.34, 14 0.49 / 0.44.
        const int workers = alone && mn >= kJacobiAhead && (gmem || smem_for(cs - 1, mn) <= kJacobiSmem) ? cs - 1 : cs;
        const size_t need = gmem ? 0 : smem_for(workers, mn);
        cfg.dynamicSmemBytes = alone && mn >= kJacobiAhead ? std::max(need, kJacobiAlone) : need;   // (one CTA a SM)
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)cs;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess || clusters < 1) {
          cudaGetLastError();
          DG_REQUIRE(cs == 16 && (gmem || smem_for(8, mn) <= kJacobiSmem), DG_ERR_CUDA, "the device runs no cluster of %d CTAs",
                     cs);
          cs = 8;   // try the portable size
          continue;
        }
        const int64_t gstride = 3 * (int64_t)((mn + workers - 1) / workers) * mn;
        if (gmem) gwork.alloc((size_t)count * cs * gstride);
        DG_CUDA(cudaLaunchKernelEx(&cfg, kernel, (const EigBlk *)(deb.get() + first), (const double *)dA.get(), dV.get(), dW.get(),
                                   workers, kJacobiSweeps, dsw.get() + first, gmem ? gwork.get() : (double *)nullptr, gstride));
        count_launch();
        cs_used = std::max(cs_used, cs);
        break;
      }
    };
    launch_part(0, n_gmem, true);
    launch_part(n_gmem, nb - n_gmem, false);
    DG_CUDA(cudaGetLastError());
    DG_CUDA(cudaMemcpyAsync(W.data(), dW.get(), sizeof(double) * W.size(), cudaMemcpyDeviceToHost, st));
    DG_CUDA(cudaMemcpyAsync(Vh.data(), dV.get(), sizeof(double) * Vh.size(), cudaMemcpyDeviceToHost, st));
    DG_CUDA(cudaMemcpyAsync(sweeps.data(), dsw.get(), sizeof(int) * nb, cudaMemcpyDeviceToHost, st));
    DG_CUDA(cudaStreamSynchronize(st));
    for (int i = 0; i < nb; ++i)
      DG_REQUIRE(sweeps[i] < kJacobiSweeps, DG_ERR_CUDA, "the Jacobi eigensolver did not converge on block %d", by_size[i]);
  });
  if (rc != DG_OK) {
    snprintf(msg, sizeof(msg), "GPU path failed (status %d): %s", rc, dg_last_error());
    fatal("DMRG_GET_SYSTEM_INFO", msg);
  }
  const double t_device = wall_s();
  // per block: eigenpairs in ascending order (LAPACK's), as (value, column of V_g)
  std::vector<int> order_in_blk((size_t)std::max<int64_t>(woff, 1));
  for (int g = 0; g < nb; ++g) {
    int *o = order_in_blk.data() + eb[g].woff;
    const double *w = W.data() + eb[g].woff;
    std::iota(o, o + eb[g].n, 0);
    std::stable_sort(o, o + eb[g].n, [&](int a, int b) { return w[a] < w[b]; });
  }
  auto value = [&](int g, int i) { return W[eb[g].woff + order_in_blk[eb[g].woff + i]]; };
  // every (block, index) in block order, then the stable descending sort (the reference's bubble sort)
  std::vector<int> sb, sbas;
  for (int g = 0; g < nb; ++g)
    for (int i = 0; i < eb[g].n; ++i) {
      sb.push_back(g);
      sbas.push_back(i);
    }
  if ((int)sb.size() != dim_LLLR) fatal(who_tm, "1");
  std::vector<int> perm(dim_LLLR);
  std::iota(perm.begin(), perm.end(), 0);
  std::stable_sort(perm.begin(), perm.end(), [&](int a, int b) { return value(sb[a], sbas[a]) > value(sb[b], sbas[b]); });
  DMRG_SYSTEM_INFO *S = static_cast<DMRG_SYSTEM_INFO *>(std::malloc(sizeof(DMRG_SYSTEM_INFO)));
  if (!S) fatal("DMRG_GET_SYSTEM_INFO", "host allocation failed");
  S->Val_DM_Dist = c_array<double>(dim_LLLR);
  S->sum_val_dm = 0;
  std::vector<double> val(dim_LLLR);
  for (int i = 0; i < dim_LLLR; ++i) {
    val[i] = value(sb[perm[i]], sbas[perm[i]]);
    S->Val_DM_Dist[i] = val[i];
    S->sum_val_dm = S->sum_val_dm + val[i];
  }
  const double zero = 1e-15;
  int dim_renorm = 0;
  if (dim_LLLR <= max_dim) {
    for (int i = dim_LLLR; i >= 1; --i)
      if (val[i - 1] > zero) {
        dim_renorm = i;
        break;
      }
  } else {
    for (int i = max_dim; i >= 1; --i)
      if (std::fabs(val[i - 1] - val[i]) > zero && val[i - 1] > zero) {
        dim_renorm = i;
        break;
      }
  }
  if (dim_renorm <= 0) fatal(who_tm, "2");
  S->tr_error = 0;
  for (int i = 0; i < dim_renorm; ++i) S->tr_error = S->tr_error + val[i];
  S->tr_error = S->sum_val_dm - S->tr_error;
  // the kept states, stably sorted by their quantum numbers (lexicographic, qn[0] first)
  std::vector<int> kept(perm.begin(), perm.begin() + dim_renorm);
  auto qn_of = [&](int k, int e) { return qn[k][blk_start[sb[e]]]; };
  std::stable_sort(kept.begin(), kept.end(), [&](int a, int b) {
    for (int k = 0; k < nq; ++k)
      if (qn_of(k, a) != qn_of(k, b)) return qn_of(k, a) < qn_of(k, b);
    return false;
  });
  long elem = 0;
  for (int e : kept) elem += eb[sb[e]].n;
  CCS1 *TM = static_cast<CCS1 *>(std::malloc(sizeof(CCS1)));
  CRS1 *TD = static_cast<CRS1 *>(std::malloc(sizeof(CRS1)));
  if (!TM || !TD) fatal("DMRG_GET_SYSTEM_INFO", "host allocation failed");
  TM->max_val = elem;
  TM->max_col = dim_renorm + 1;
  TM->Val = c_array<double>(elem);
  TM->Col = c_array<long>(dim_renorm + 1);
  TM->Row = c_array<int>(elem);
  TD->max_val = elem;
  TD->max_row = dim_renorm + 1;
  TD->Val = c_array<double>(elem);
  TD->Col = c_array<int>(elem);
  TD->Row = c_array<long>(dim_renorm + 1);
  S->Q_Number1 = c_array<int>(dim_renorm);
  S->Q_Number2 = c_array<int>(nq >= 2 ? dim_renorm : 1);
  S->Q_Number3 = c_array<int>(nq >= 3 ? dim_renorm : 1);
  if (nq < 2) S->Q_Number2[0] = INT_MIN;
  if (nq < 3) S->Q_Number3[0] = INT_MIN;
  long c = 0;
  for (int j = 0; j < dim_renorm; ++j) {
    const int e = kept[j], g = sb[e], n = eb[g].n;
    S->Q_Number1[j] = qn_of(0, e);
    if (nq >= 2) S->Q_Number2[j] = qn_of(1, e);
    if (nq >= 3) S->Q_Number3[j] = qn_of(2, e);
    const int colv = order_in_blk[eb[g].woff + sbas[e]];
    const double *V = Vh.data() + eb[g].off;
    for (int i = 0; i < n; ++i) {
      const double x = V[(int64_t)i * n + colv];
      TM->Val[c] = x;
      TM->Row[c] = blk_start[g] + i;
      TD->Val[c] = x;
      TD->Col[c] = blk_start[g] + i;
      ++c;
    }
    TM->Col[j + 1] = c;
    TD->Row[j + 1] = c;
  }
  if (c != TM->max_val) fatal(who_tm, "3");
  TM->row_dim = dim_LLLR;
  TM->col_dim = dim_renorm;
  TD->row_dim = dim_renorm;
  TD->col_dim = dim_LLLR;
  S->Trans_Matrix = TM;
  S->Trans_Matrix_Dagger = TD;
  S->dim_renorm = dim_renorm;
  S->dim_LLLR = dim_LLLR;
  const double t_end = wall_s();
  if (T) T->make_dens_mat = t_end - t0;
  if (const char *e = std::getenv("DG_SB_TRUNC_TIMES")) {   // phase report for profiling
    if (e[0] == '1') {
      int mx = 0;
      for (int sw : sweeps) mx = std::max(mx, sw);
      fprintf(stderr, "truncation: gather %.2f ms, device %.2f ms (clusters of %d CTAs, at most %d sweeps), host %.2f ms\n",
              (t_gather - t0) * 1e3, (t_device - t_gather) * 1e3, cs_used, mx, (t_end - t_device) * 1e3);
    }
  }
  return S;
}

}  // namespace
}  // namespace dg

extern "C" {

// include/dmrg.h:390-392
DMRG_SYSTEM_INFO *DMRG_GET_SYSTEM_INFO_Q1(int *Q_Number, DMRG_BASIS *Dmrg_Basis, double *Vec, int max_dim, int, DMRG_TIME *Dmrg_Time) {
  const int *q[1] = {Q_Number};
  return dg::system_info(1, q, Dmrg_Basis, Vec, max_dim, Dmrg_Time);
}

DMRG_SYSTEM_INFO *DMRG_GET_SYSTEM_INFO_Q2(int *Q_Number1, int *Q_Number2, DMRG_BASIS *Dmrg_Basis, double *Vec, int max_dim, int,
                                          DMRG_TIME *Dmrg_Time) {
  const int *q[2] = {Q_Number1, Q_Number2};
  return dg::system_info(2, q, Dmrg_Basis, Vec, max_dim, Dmrg_Time);
}

DMRG_SYSTEM_INFO *DMRG_GET_SYSTEM_INFO_Q3(int *Q_Number1, int *Q_Number2, int *Q_Number3, DMRG_BASIS *Dmrg_Basis, double *Vec,
                                          int max_dim, int, DMRG_TIME *Dmrg_Time) {
  const int *q[3] = {Q_Number1, Q_Number2, Q_Number3};
  return dg::system_info(3, q, Dmrg_Basis, Vec, max_dim, Dmrg_Time);
}

}  // extern "C"
