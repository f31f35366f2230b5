// rf_factor.cu — block ILU0 and pressure ILU0 of the reduced matrix (factorize_block_ilu0,
// factorize_pressure_ilu0: gmres_block_jacobi.rs:808-885, 284-353) from a plan built once per pattern.
//
// The factors follow the natural-order elimination, so rows form levels that run one after another.
// What has to be inside that chain is little: of a row of the plain 7-point shape ("simple": at most
// three lower blocks, each updating the diagonal alone) only the inverse of its diagonal block and
// its pressure pivot.  So
//   k_factor_prep    copies the present blocks and the pressure values, over the whole chip;
//   k_factor_levels  walks the levels on one thread-block cluster per matrix: four lanes per simple
//                    row form D = A_ii - sum (A_ik Dinv_k) U_ki and invert it;
//   k_factor_post    writes the simple rows' L = A_ik Dinv_k and pressure quotients, over the whole chip.
// Rows with a well's fill ("listed") hold up to as many blocks as the well has perforations, and each
// lower entry changes the ones after it.  They are eliminated right-looking: as soon as a lower
// entry's column is final, a warp applies that entry to the whole row (a lane per updated
// block), so that a level of the walk holds one step for every listed row instead of one
// row's whole chain.  An entry is applied after the entries before it, so every element takes the
// operations of the row-by-row elimination in their order, and the factors are equal bit for bit.
// What bounds it: the chain of levels, each a round of L2 loads of what the level before wrote, some
// 200 FP64 operations in sequence and the cluster barrier.  Everything that does not depend on the
// level before (records, matrix blocks, the listed steps' indices) is loaded before that barrier.
// ms per factorisation, against the form it replaces (a thread per short row, a warp per row with
// fill that walked the whole row in its own level; one CTA, or a cluster for large decks):
// 45x61x7 2.85 -> 0.55, 60x60x20 black oil 7.0 -> 0.86, 127x101x40 44.2 -> 4.0, the 16-variant
// ensemble's launches 2.48 -> 0.68, 10x10x3 0.23 -> 0.09, a chain of 200 one-row levels 0.70 -> 0.65.
#include <algorithm>
#include <cstring>

#include "rf_fiber.hpp"
#include "rf_mat3.cuh"
#include "rf_ops.hpp"

namespace rf {

namespace {

constexpr double kEpsF = kF64Eps;
constexpr int kFacThreads = 256;     // 255 registers: a row's operands are held at once
constexpr int kFacRowLanes = 4;      // lanes of a simple row: the three block rows, the pressure pivot
constexpr int kFacLower = 3;         // lower blocks of a simple row
constexpr int kFacSmemLevels = 4096; // level tables kept in shared memory up to this many levels

struct FacLevelArgs {
  int n_levels;
  const int* row_ptr;   // [n_levels + 1] simple rows
  const int* step_ptr;  // [n_levels + 1] listed steps
  const int4* rec;      // simple rows by level, 3 each: {row, dp, lower entries, -} {columns} {U entries, -1: none}
  const int4* step;     // {first entry, end, row or -1 when it is not finished by this step, dp}
  const int4* entry;    // {kp, column, first pair, end}
  const int2* pair;     // {U entry, updated entry}
  const double* val;
  const unsigned char* mask;
  const double* pval;
  double* lu;
  double* dinv;
  double* plu;
  double* pdiag;
};

__device__ __forceinline__ unsigned fac_ranks() {
  unsigned v;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(v));
  return v;
}
__device__ __forceinline__ unsigned fac_rank() {
  unsigned v;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(v));
  return v;
}

struct FacRec {
  int row, dp, nl, ck[kFacLower], up[kFacLower];  // row < 0: none
};
// A lane's part of what a simple row needs that no row of this launch writes: lane h < 3 of the four
// holds row h of the blocks, lane 3 the pressure values.
struct FacRow {
  FacRec r;
  unsigned char mk[kFacLower], mu[kFacLower], md;  // masks of the entries, their U blocks, the diagonal
  double A[kFacLower][3], D[3];                    // lane 3: A[j][0] pressure value, D[0] the diagonal's
};

__device__ __forceinline__ FacRec fac_rec(const FacLevelArgs& a, int q, int end) {
  FacRec r;
  r.row = -1;
  r.dp = r.nl = 0;
#pragma unroll
  for (int j = 0; j < kFacLower; ++j) r.ck[j] = 0, r.up[j] = -1;
  if (q < end) {
    const int4 h = __ldg(a.rec + 3 * size_t(q)), c = __ldg(a.rec + 3 * size_t(q) + 1),
               u = __ldg(a.rec + 3 * size_t(q) + 2);
    r.row = h.x, r.dp = h.y, r.nl = h.z;
    r.ck[0] = c.x, r.ck[1] = c.y, r.ck[2] = c.z;
    r.up[0] = u.x, r.up[1] = u.y, r.up[2] = u.z;
  }
  return r;
}

// Loads only: a value that were looked at here would be waited for before the level's barrier.
__device__ __forceinline__ FacRow fac_load(const FacLevelArgs& a, const FacRec& r) {
  FacRow w;
  w.r = r;
  const int h = threadIdx.x & 3, b0 = r.dp - r.nl;
  w.md = 0;
  w.D[0] = w.D[1] = w.D[2] = 0.0;
#pragma unroll
  for (int j = 0; j < kFacLower; ++j) {
    w.mk[j] = w.mu[j] = 0;
    w.A[j][0] = w.A[j][1] = w.A[j][2] = 0.0;
  }
  if (r.row < 0) return w;
  w.md = __ldg(a.mask + r.dp);
#pragma unroll
  for (int j = 0; j < kFacLower; ++j) {
    if (j >= r.nl || r.up[j] < 0) continue;
    w.mk[j] = __ldg(a.mask + b0 + j);
    w.mu[j] = __ldg(a.mask + r.up[j]);
    if (h == 3) {
      w.A[j][0] = __ldg(a.pval + b0 + j);
    } else {
#pragma unroll
      for (int e = 0; e < 3; ++e) w.A[j][e] = __ldg(a.val + size_t(b0 + j) * 9 + 3 * h + e);
    }
  }
  if (h == 3) {
    w.D[0] = __ldg(a.pval + r.dp);
  } else {
#pragma unroll
    for (int e = 0; e < 3; ++e) w.D[e] = __ldg(a.val + size_t(r.dp) * 9 + 3 * h + e);
  }
  return w;
}

// The diagonal block, its inverse and the pressure pivot of a simple row by four lanes (all lanes of
// the warp call): the lower entries in order, each L = A Dinv and D -= L U; absent blocks are
// skipped.  The loads of both kinds of lane come before either's arithmetic, and the three divisions
// of each (a row of cofactors by the determinant; the pressure quotients) are the same instructions.
__device__ __forceinline__ void fac_finish(const FacLevelArgs& a, const FacRow& w) {
  const FacRec& r = w.r;
  const int h = threadIdx.x & 3;
  const bool md = w.md != 0;
  bool on[kFacLower];  // the entry updates the diagonal: blocks, or pressure value, present
#pragma unroll
  for (int j = 0; j < kFacLower; ++j)
    on[j] = r.row >= 0 && j < r.nl && r.up[j] >= 0 && (h == 3 ? w.A[j][0] != 0.0 : md && w.mk[j] != 0 && w.mu[j] != 0);
  const bool zero = h < 3 && !md;  // an absent diagonal block
  double D[3] = {zero ? 0.0 : w.D[0], zero ? 0.0 : w.D[1], zero ? 0.0 : w.D[2]};
  double dk[kFacLower][9], u[kFacLower][9];  // lane 3: the column's pivot and the U value, in element 0
  if (h < 3) {
#pragma unroll
    for (int j = 0; j < kFacLower; ++j) {
      const double* pd = a.dinv + size_t(r.ck[j]) * 9;
      const double* pu = a.lu + size_t(max(r.up[j], 0)) * 9;
#pragma unroll
      for (int e = 0; e < 9; ++e) {
        dk[j][e] = on[j] ? pd[e] : 0.0;
        u[j][e] = on[j] ? pu[e] : 0.0;
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < kFacLower; ++j) {
      dk[j][0] = on[j] ? a.pdiag[r.ck[j]] : 1.0;
      u[j][0] = on[j] ? a.plu[r.up[j]] : 0.0;
    }
  }
  if (h < 3) {
#pragma unroll
    for (int j = 0; j < kFacLower; ++j) {
      if (!on[j]) continue;
      const double* A = w.A[j];
      double l[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) l[k] = A[0] * dk[j][k] + A[1] * dk[j][3 + k] + A[2] * dk[j][6 + k];
#pragma unroll
      for (int k = 0; k < 3; ++k) D[k] -= l[0] * u[j][k] + l[1] * u[j][3 + k] + l[2] * u[j][6 + k];
    }
  }
  __syncwarp();
  // the inverse (mat3_inverse_or_diag): every lane gathers the block and takes its row of cofactors
  double m[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) m[k] = __shfl_sync(0xffffffffu, D[k % 3], k / 3, 4);
  const double c11 = m[4] * m[8] - m[7] * m[5], c21 = m[3] * m[8] - m[6] * m[5], c31 = m[3] * m[7] - m[6] * m[4];
  const double det = m[0] * c11 - m[1] * c21 + m[2] * c31;
  double x[3], y[3] = {det, det, det};
  x[0] = h == 0 ? c11 : h == 1 ? -c21 : c31;
  x[1] = h == 0 ? m[2] * m[7] - m[8] * m[1] : h == 1 ? m[0] * m[8] - m[6] * m[2] : m[1] * m[6] - m[7] * m[0];
  x[2] = h == 0 ? m[1] * m[5] - m[4] * m[2] : h == 1 ? m[2] * m[3] - m[5] * m[0] : m[0] * m[4] - m[3] * m[1];
  if (h == 3) {
#pragma unroll
    for (int j = 0; j < kFacLower; ++j) x[j] = w.A[j][0], y[j] = dk[j][0];
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) x[k] = x[k] / y[k];
  if (r.row < 0) return;
  if (h == 3) {
    double ud = w.D[0];
#pragma unroll
    for (int j = 0; j < kFacLower; ++j)
      if (on[j]) ud -= (fabs(y[j]) > kEpsF ? x[j] : 0.0) * u[j][0];
    if (fabs(ud) <= kEpsF) ud = fabs(w.D[0]) > kEpsF ? w.D[0] : 1.0;
    a.pdiag[r.row] = ud;
    return;
  }
  if (det == 0.0) {
    double inv[9];
    mat3_inverse_or_diag(m, inv);
#pragma unroll
    for (int k = 0; k < 3; ++k) x[k] = h == 0 ? inv[k] : h == 1 ? inv[3 + k] : inv[6 + k];
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    a.dinv[size_t(r.row) * 9 + 3 * h + k] = x[k];
    a.lu[size_t(r.dp) * 9 + 3 * h + k] = D[k];
  }
}

// A lane's pair of an entry (none: the first block with itself, which is not used).
__device__ __forceinline__ int2 fac_pair(const FacLevelArgs& a, int e, int end) {
  return e < end ? __ldg(a.pair + e) : make_int2(0, 0);
}

// The first entries of a step and the lane's pairs of them, which the last step of a vertical well's row
// has three of; loaded ahead of the step's level.
constexpr int kFacAhead = 3;
struct FacStep {
  int4 s;  // s.z == -2: none
  int4 e[kFacAhead];
  int2 p[kFacAhead];
};

// One step of a listed row by a warp: its lower entries [s.x, s.y) in order, each applied to the
// blocks and pressure values after it; the last step inverts the diagonal.  All of an entry's loads
// are issued together.
__device__ __forceinline__ void fac_step(const FacLevelArgs& a, FacStep& w) {
  const int lane = threadIdx.x & 31, dp = w.s.w;
#pragma unroll 1
  for (int k = w.s.x; k < w.s.y; ++k) {
    const int4 e = w.e[0];
    int2 p = w.p[0];
    const int kp = e.x;
    const size_t c = size_t(e.y);
    double lk[9], dk[9], l[9], u[9], t[9], pu, pt, pv;
    unsigned char mu, mt;
    auto operands = [&]() {
      mu = __ldg(a.mask + p.x), mt = __ldg(a.mask + p.y);
      pv = __ldg(a.pval + p.y);
#pragma unroll
      for (int q = 0; q < 9; ++q) {
        u[q] = a.lu[size_t(p.x) * 9 + q];
        t[q] = a.lu[size_t(p.y) * 9 + q];
      }
      pu = a.plu[p.x], pt = a.plu[p.y];
    };
    const unsigned char mk = __ldg(a.mask + kp);
    const double pk = __ldg(a.pval + kp), acc = a.plu[kp], d = a.pdiag[c];
#pragma unroll
    for (int q = 0; q < 9; ++q) {
      lk[q] = a.lu[size_t(kp) * 9 + q];
      dk[q] = a.dinv[c * 9 + q];
    }
    operands();
    // the entries after this one move up
#pragma unroll
    for (int h = 0; h + 1 < kFacAhead; ++h) w.e[h] = w.e[h + 1], w.p[h] = w.p[h + 1];
    if (k + kFacAhead < w.s.y) {
      w.e[kFacAhead - 1] = __ldg(a.entry + k + kFacAhead);
      w.p[kFacAhead - 1] = fac_pair(a, w.e[kFacAhead - 1].z + lane, w.e[kFacAhead - 1].w);
    }
    const bool m = mk != 0, pm = pk != 0.0;
    mat3_mul(lk, dk, l);
    const double pl = pm && fabs(d) > kEpsF ? acc / d : 0.0;
    __syncwarp();  // all lanes have read the entry
#pragma unroll 1
    for (int f = e.z + lane; f < e.w;) {
      if (m && mu != 0 && mt != 0) {
        double prod[9];
        mat3_mul(l, u, prod);
#pragma unroll
        for (int q = 0; q < 9; ++q) a.lu[size_t(p.y) * 9 + q] = t[q] - prod[q];
      }
      if (pm && (pv != 0.0 || p.y == dp)) a.plu[p.y] = pt - pl * pu;
      f += 32;
      if (f >= e.w) break;
      p = fac_pair(a, f, e.w);
      operands();
    }
    if (lane < 9 && m) {
      double v = l[0];
#pragma unroll
      for (int q = 1; q < 9; ++q)
        if (lane == q) v = l[q];
      a.lu[size_t(kp) * 9 + lane] = v;
    }
    if (lane == 9 && pm) a.plu[kp] = pl;
    __syncwarp();
  }
  if (w.s.z >= 0) {
    if (lane == 0) {
      double D[9], inv[9];
#pragma unroll
      for (int q = 0; q < 9; ++q) D[q] = a.lu[size_t(dp) * 9 + q];
      mat3_inverse_or_diag(D, inv);
#pragma unroll
      for (int q = 0; q < 9; ++q) a.dinv[size_t(w.s.z) * 9 + q] = inv[q];
    } else if (lane == 1) {
      const double de = __ldg(a.pval + dp);
      double ud = a.plu[dp];
      if (fabs(ud) <= kEpsF) ud = fabs(de) > kEpsF ? de : 1.0;
      a.pdiag[w.s.z] = ud;
      a.plu[dp] = 0.0;
    }
    __syncwarp();
  }
}

// Cluster b of the grid factors item b.
struct FacLevelBatch {
  int count;
  FacLevelArgs item[kBatchItems];
};

__device__ void fac_levels_body(const FacLevelArgs& a) {
  __shared__ int s_row[kFacSmemLevels], s_step[kFacSmemLevels];
  const int L = a.n_levels;
  const bool staged = L + 1 <= kFacSmemLevels;
  if (staged) {
    for (int i = threadIdx.x; i <= L; i += kFacThreads) {
      s_row[i] = a.row_ptr[i];
      s_step[i] = a.step_ptr[i];
    }
    __syncthreads();
  }
  auto row_at = [&](int l) { return staged ? s_row[min(l, L)] : __ldg(a.row_ptr + min(l, L)); };
  auto step_at = [&](int l) { return staged ? s_step[min(l, L)] : __ldg(a.step_ptr + min(l, L)); };
  const int cs = int(fac_ranks()), rank = int(fac_rank());
  // warp w takes the rows 8 w.. of a level; the steps start from the warps the rows reach last
  const int nw = cs * (kFacThreads / 32), at = rank + cs * int(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int warp = nw - 1 - at, row0 = at * (32 / kFacRowLanes), row = row0 + lane / kFacRowLanes;
  const int rows = nw * (32 / kFacRowLanes);
  auto step_of = [&](int l) {
    const int q = step_at(l) + warp;
    return q < step_at(l + 1) ? __ldg(a.step + q) : make_int4(0, 0, -2, 0);
  };
  auto entries_of = [&](FacStep& w) {
#pragma unroll
    for (int h = 0; h < kFacAhead; ++h)
      w.e[h] = w.s.x + h < w.s.y ? __ldg(a.entry + w.s.x + h) : make_int4(0, 0, 0, 0);
  };
  auto pairs_of = [&](FacStep& w) {
#pragma unroll
    for (int h = 0; h < kFacAhead; ++h) w.p[h] = fac_pair(a, w.e[h].z + lane, w.e[h].w);
  };
  const bool any_steps = step_at(L) > 0;
  // a level's operands are loaded in the barriers before it: records, steps and entries levels ahead
  FacRow cur = fac_load(a, fac_rec(a, row_at(0) + row, row_at(1)));
  FacRec next = fac_rec(a, row_at(1) + row, row_at(2));
  FacStep w0, w1;
  w0.s = step_of(0), w1.s = step_of(1);
  int4 s2 = step_of(2);
  entries_of(w0), entries_of(w1);
  pairs_of(w0);
#pragma unroll 1
  for (int l = 0; l < L; ++l) {
    const int end = row_at(l + 1);
    // listed rows first: their chains are longer
    if (w0.s.z != -2) {
      fac_step(a, w0);
      const int send = step_at(l + 1);
#pragma unroll 1
      for (int q = step_at(l) + warp + nw; q < send; q += nw) {
        w0.s = __ldg(a.step + q);
        entries_of(w0);
        pairs_of(w0);
        fac_step(a, w0);
      }
    }
    __syncwarp();
#pragma unroll 1
    for (int q = row_at(l) + row0; q < end;) {  // the same for all lanes
      fac_finish(a, cur);
      q += rows;
      if (q < end) cur = fac_load(a, fac_rec(a, q + lane / kFacRowLanes, end));
    }
    __syncwarp();
    if (l + 1 == L) break;
    if (cs > 1)
      asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    cur = fac_load(a, next);
    next = fac_rec(a, row_at(l + 2) + row, row_at(l + 3));
    if (any_steps) {
      w0 = w1;
      pairs_of(w0);
      w1.s = s2;
      entries_of(w1);
      s2 = step_of(l + 3);
    }
    if (cs > 1)
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    else
      __syncthreads();
  }
}

__global__ void __launch_bounds__(kFacThreads, 1) k_factor_levels(const __grid_constant__ FacLevelArgs a) {
  fac_levels_body(a);
}
__global__ void __launch_bounds__(kFacThreads, 1) k_factor_levels_batch(const __grid_constant__ FacLevelBatch b) {
  const unsigned item = blockIdx.x / fac_ranks();
  if (item < unsigned(b.count)) fac_levels_body(b.item[item]);
}

// Present blocks and pressure values of the matrix; 2 x the matrix's bytes at the copy's rate.
__global__ void __launch_bounds__(kBlock) k_factor_prep(long long nnzb, const double* __restrict__ val,
                                                        const unsigned char* __restrict__ mask,
                                                        const double* __restrict__ pval, double* __restrict__ lu,
                                                        double* __restrict__ plu) {
  const long long stride = (long long)gridDim.x * blockDim.x, t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  for (long long t = t0; t < 9 * nnzb; t += stride) lu[t] = mask[t / 9] ? val[t] : 0.0;
  for (long long t = t0; t < nnzb; t += stride) plu[t] = pval[t];
}

// The simple rows' lower blocks and pressure quotients; a thread per row.
__global__ void __launch_bounds__(kBlock) k_factor_post(int n, const unsigned char* __restrict__ simple,
                                                        const int* __restrict__ rp, const int* __restrict__ col,
                                                        const int* __restrict__ diag, const double* __restrict__ val,
                                                        const unsigned char* __restrict__ mask,
                                                        const double* __restrict__ pval,
                                                        const double* __restrict__ dinv,
                                                        const double* __restrict__ pdiag, double* __restrict__ lu,
                                                        double* __restrict__ plu) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || !simple[i]) return;
  const int dp = diag[i];
  for (int k = rp[i]; k < dp; ++k) {
    const int c = col[k];
    if (mask[k]) {
      double A[9], dk[9], l[9];
#pragma unroll
      for (int e = 0; e < 9; ++e) {
        A[e] = val[size_t(k) * 9 + e];
        dk[e] = dinv[size_t(c) * 9 + e];
      }
      mat3_mul(A, dk, l);
#pragma unroll
      for (int e = 0; e < 9; ++e) lu[size_t(k) * 9 + e] = l[e];
    }
    const double pv = pval[k];
    if (pv != 0.0) {
      const double d = pdiag[c];
      plu[k] = fabs(d) > kEpsF ? pv / d : 0.0;
    }
  }
  plu[dp] = 0.0;
}

cudaError_t fac_launch(const void* fn, int clusters, int cs, void** args, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(clusters * cs);
  cfg.blockDim = dim3(kFacThreads);
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cs;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelExC(&cfg, fn, args);
}

// Whether a cluster of 16 can run (it needs the non-portable attribute).
bool fac_sixteen() {
  const void* fn = (const void*)k_factor_levels;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(16);
  cfg.blockDim = dim3(kFacThreads);
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 16;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int clusters = 0;
  const bool ok = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                  cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg) == cudaSuccess && clusters >= 1;
  cudaGetLastError();
  return ok;
}

// CTAs per matrix of an ensemble, whose variants share the chip and one launch.
constexpr int kFacBatchCtas = 4;

template <class V, class H>
void upload_plan(V& b, const H& h) {
  b.free();
  b.alloc(std::max<size_t>(h.size(), 1));
  if (!h.empty()) RF_CUDA(cudaMemcpy(b.p, h.data(), sizeof(h[0]) * h.size(), cudaMemcpyHostToDevice));
}

}  // namespace

void free_factor_plan(Ctx& c) {
  FactorPlan& P = c.fac;
  for (auto* b : {&P.d_row_ptr, &P.d_step_ptr}) b->free();
  for (auto* b : {&P.d_rec, &P.d_step, &P.d_entry}) b->free();
  P.d_pair.free();
  P.d_simple.free();
  P.built = 0;
}

void build_factor_plan(Ctx& c) {
  FactorPlan& P = c.fac;
  const int n = c.n, nl = c.levels.n_levels;
  const std::vector<int>&rp = c.h_row_ptr, &col = c.h_col, &diag = c.h_diag, &lp = c.levels.h_ptr;
  std::vector<int> lvl(n);
  for (int l = 0; l < nl; ++l)
    for (int q = lp[l]; q < lp[l + 1]; ++q) lvl[c.levels.h_rows[q]] = l;
  std::vector<unsigned char> simple(n, 0);
  std::vector<int> row_ptr(nl + 1, 0), step_ptr(nl + 1, 0);
  std::vector<int4> rec, step, entry;
  std::vector<int2> pair, own;
  std::vector<std::vector<int4>> steps(nl);
  rec.reserve(3 * size_t(n));
  for (int l = 0; l < nl; ++l) {
    for (int q = lp[l]; q < lp[l + 1]; ++q) {
      const int i = c.levels.h_rows[q], b0 = rp[i], dp = diag[i], b1 = rp[i + 1];
      // each lower entry's pairs: the U-row of its column against row i's later entries
      own.clear();
      int first[kFacLower + 1] = {0, 0, 0, 0};
      bool plain = dp - b0 <= kFacLower;
      auto merge = [&](int kp) {
        const int kr = col[kp];
        int ip = kp + 1;
        for (int up = diag[kr] + 1; up < rp[kr + 1]; ++up) {
          while (ip < b1 && col[ip] < col[up]) ++ip;
          if (ip >= b1) break;
          if (col[ip] == col[up]) own.push_back(make_int2(up, ip));
        }
      };
      for (int kp = b0; plain && kp < dp; ++kp) {
        merge(kp);
        const int at = first[kp - b0], cnt = int(own.size()) - at;
        first[kp - b0 + 1] = int(own.size());
        plain = cnt == 0 || (cnt == 1 && own[at].y == dp);
      }
      if (plain) {
        simple[i] = 1;
        int ck[kFacLower] = {0, 0, 0}, up[kFacLower] = {-1, -1, -1};
        for (int j = 0; j < dp - b0; ++j) {
          ck[j] = col[b0 + j];
          if (first[j + 1] > first[j]) up[j] = own[first[j]].x;
        }
        rec.push_back(make_int4(i, dp, dp - b0, 0));
        rec.push_back(make_int4(ck[0], ck[1], ck[2], 0));
        rec.push_back(make_int4(up[0], up[1], up[2], 0));
        continue;
      }
      // listed: an entry is applied in the first level after its column's, and after the
      // entry before it
      int at = 0, s0 = int(entry.size());
      for (int kp = b0; kp < dp; ++kp) {
        const int when = std::max(at, lvl[col[kp]] + 1);
        if (when > at && int(entry.size()) > s0) {
          steps[at].push_back(make_int4(s0, int(entry.size()), -1, dp));
          s0 = int(entry.size());
        }
        at = when;
        own.clear();
        merge(kp);
        entry.push_back(make_int4(kp, col[kp], int(pair.size()), int(pair.size() + own.size())));
        pair.insert(pair.end(), own.begin(), own.end());
      }
      steps[l].push_back(make_int4(s0, int(entry.size()), i, dp));
    }
    row_ptr[l + 1] = int(rec.size() / 3);
  }
  int work = 1;  // threads that the busiest level can use
  for (int l = 0; l < nl; ++l) {
    step.insert(step.end(), steps[l].begin(), steps[l].end());
    step_ptr[l + 1] = int(step.size());
    work = std::max(work, kFacRowLanes * (row_ptr[l + 1] - row_ptr[l]) + 32 * int(steps[l].size()));
  }
  // CTAs of a single deck's factorisation: half a CTA's threads each, since a level's loads are then
  // spread over more SMs, up to 16
  P.cs = 1;
  while (P.cs < 16 && P.cs * (kFacThreads / 2) < work) P.cs *= 2;
  if (P.cs == 16 && !fac_sixteen()) P.cs = 8;
  upload_plan(P.d_row_ptr, row_ptr);
  upload_plan(P.d_step_ptr, step_ptr);
  upload_plan(P.d_rec, rec);
  upload_plan(P.d_step, step);
  upload_plan(P.d_entry, entry);
  upload_plan(P.d_pair, pair);
  upload_plan(P.d_simple, simple);
  P.built = 1;
}

int factor_ctas(const Ctx& c) {
  if (!c.fac.built) return c.cluster_size;
  return c.batched ? kFacBatchCtas : c.fac.fixed ? c.fac.fixed : c.fac.cs;
}

void factor_fix(Ctx& c) { c.fac.fixed = c.cluster_fixed == 16 && !fac_sixteen() ? 8 : c.cluster_fixed; }

void factor_levels(Ctx& c) {
  FactorPlan& P = c.fac;
  const long long nnzb = c.nnzb;
  k_factor_prep<<<int(std::min<long long>((9 * nnzb + kBlock - 1) / kBlock, 16ll * c.num_sms)), kBlock, 0, c.stream>>>(
      nnzb, c.d_val.p, c.d_bmask.p, c.d_pval.p, c.d_lu.p, c.d_plu.p);
  FacLevelArgs a;
  a.n_levels = c.levels.n_levels;
  a.row_ptr = P.d_row_ptr.p;
  a.step_ptr = P.d_step_ptr.p;
  a.rec = P.d_rec.p;
  a.step = P.d_step.p;
  a.entry = P.d_entry.p;
  a.pair = P.d_pair.p;
  a.val = c.d_val.p;
  a.mask = c.d_bmask.p;
  a.pval = c.d_pval.p;
  a.lu = c.d_lu.p;
  a.dinv = c.d_dinv.p;
  a.plu = c.d_plu.p;
  a.pdiag = c.d_pdiag.p;
  if (!(c.batched && fiber_file(kBatchFactor, 0, &a, sizeof(a), kFacThreads, 0))) {
    void* args[] = {&a};
    RF_CUDA(fac_launch((const void*)k_factor_levels, 1, P.fixed ? P.fixed : P.cs, args, c.stream));
    c.launches++;
  }
  k_factor_post<<<(c.n + kBlock - 1) / kBlock, kBlock, 0, c.stream>>>(
      c.n, P.d_simple.p, c.d_row_ptr.p, c.d_col.p, c.d_diag.p, c.d_val.p, c.d_bmask.p, c.d_pval.p, c.d_dinv.p,
      c.d_pdiag.p, c.d_lu.p, c.d_plu.p);
  c.launches += 2;
}

static_assert(sizeof(FacLevelArgs) <= kBatchArgBytes, "factorisation arguments must fit a batch item");
bool launch_factor_batch(const BatchItem* const* items, int count, cudaStream_t stream) {
  FacLevelBatch b;
  b.count = count;
  for (int i = 0; i < count; ++i) std::memcpy(&b.item[i], items[i]->args, sizeof(FacLevelArgs));
  void* args[] = {&b};
  return fac_launch((const void*)k_factor_levels_batch, count, kFacBatchCtas, args, stream) == cudaSuccess;
}

}  // namespace rf
