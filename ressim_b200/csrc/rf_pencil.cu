// rf_pencil.cu — the pressure stage's BiCGStab (solve_pressure_with_bicgstab,
// gmres_block_jacobi.rs:622-729) with the ILU0 sweeps run along grid lines ("pencils") by one
// thread-block cluster.
//
// An ILU0 sweep over the natural-order 7-point grid is a wavefront: cell (i, j, k) needs its
// lower neighbours of level i+j+k-1, so nx+ny+nz-2 steps must run one after another and a sweep
// costs steps x (one dependent step).  The solves that walk the levels as row lists
// (rf_level.cu, rf_linear.cu) spend 1,400 cycles and more per step on staging, index decoding and
// the division.  Here a thread owns a line of cells (., j, k) and moves along x one cell per step:
//   - a step is three shared-memory reads (the x, y and z neighbours' results of the step before),
//     the row's products and subtractions, a shared-memory store and a barrier of the line warps;
//   - every array is stored in step order, [step][line] with the steps a line has not started or
//     has left filled with zeros: the rows of consecutive steps are contiguous, and no lane needs a
//     condition.  One warp copies eight (four, two) steps' rows at a time into shared memory, one bulk
//     copy per array, and the results back.  (Loads by the line threads themselves, in registers
//     several steps ahead, cost 100-150 cycles per step whatever their distance, branches in the
//     step another 40 each, and bulk copies of single steps 1,100 cycles a step to issue.)
//   - the division by the pivot is a multiplication by its reciprocal corrected to the correctly
//     rounded quotient (pen_div);
//   - the columns j are split over the cluster's CTAs.  One warp of each CTA sends the values of its
//     last column (backward: first) to the next CTA with st.async, whose completion counts on an
//     mbarrier per step there, another one receives them ahead of the line warps' barrier.
//     Waits are bounded (kPenWaitCycles); one that gives up sets a status the host turns into an error,
//     and the cluster ends the solve after the sweep it is in;
//   - rows with a well's fill (more entries, reaching far up the column) are solved by the sending
//     warp between two barriers, their products formed by one lane each.
// What bounds it: the chain of steps.  Cycles per step (B200, FP64): 203 forward and 242 backward
// with five line warps, 154 and 187 with one, 300-400 with the hand-over between CTAs, against some
// 1,430 before.  Report steps with the kernel it replaces and with its first form, the other kernels
// as they were then: 45x61x7 waterflood 175 -> 102 ms, 60x60x20 black oil
// 125 -> 66, 127x101x40 waterflood 1,617 -> 363 (mixed 1,581 -> 364), a 16-variant ensemble's 1,489
// -> 878; one linear solve on 40x31x5 25.5 -> 12.8 ms.  Factors and vectors come from L2.
// Every row takes the operations of the reference's sequential sweep in its order.  Dot products
// keep the order of the kernels this one stands in for (DotOrder): the sums do not depend on the
// cluster size or the thread count here, so results equal those kernels' bit for bit.
//
// Used when every cell's level is i+j+k (no well fill deepens the levels), each well's fill stays
// within one CTA's columns, the padding of the step order stays small and the wells' rows do not crowd
// the chain of steps (pen_crowded); other decks, and callers that name a kernel family, keep the
// level-list kernels.
#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "rf_fiber.hpp"
#include "rf_ops.hpp"
#include "rf_pencil_layout.hpp"
#include "rf_quotient.hpp"

namespace rf {

namespace {

constexpr double kEpsP = kF64Eps;
constexpr int kPenThreads = 512;
constexpr int kPenLineWarps = 13;  // warps 0..12 own lines
constexpr int kPenLoadWarp = 13;   // copies rows in and results out
constexpr int kPenRecvWarp = 14, kPenSendWarp = 15;  // neighbours' values in; out, and the wells' rows
constexpr int kPenLineThreads = 32 * kPenLineWarps;
constexpr long long kPenWaitCycles = 2000000000;  // a second; a whole sweep takes some milliseconds
constexpr unsigned kPenSpecial = 0x7ff80001u;            // high word of the reciprocal of a listed row

// Order of a dot product: virtual threads (vblocks blocks of vwpb warps) each sum the elements
// start, start + stride, ... < end of their own, a warp's 32 sums are added by a shuffle tree, a
// block's warps by a second one, the blocks one after another.
//   level kernels:          one block of NT threads over positions (rows numbered level by level),
//                           stride NT; in the matrix products the rows of more than 7 entries
//                           come after all others; the norm of s runs level by level (element t of
//                           every level, then t + NT, ...)
//   cluster, in slices:     block b over the natural rows [b S, b S + S), stride 256
//   cluster, grid-strided:  all blocks' threads over the natural rows
struct DotOrder {
  int vblocks, vwpb;
};

template <class T>
struct PenArgs {
  int n, nx, ny, nz, slots, chunk;  // slots: of all CTAs, guards included; steps copied at a time
  DotOrder dot;
  const int* cta;      // [cs + 1] first slot of each CTA's region
  const int* nat;      // [n] slot of each natural row
  // the dot products' orders: plain, after a product with the matrix, of the norm of s; list_ptr holds
  // the virtual warps' first chunks of the three one after another
  const int* list_ptr;
  const int* list[3];
  // matrix rows with entries outside the stencil
  int nspec;
  const int* spec_slot;
  const int* spec_ptr;
  const int* spec_col;  // slots
  const T* spec_val;
  // the same rows in the sweeps: first one of each CTA, step and line, slot, entry ranges per
  // direction, entry codes (window index, or 0x8000 + listed row of the CTA) and values
  const int* well_cta;   // [cs + 1]
  const int2* well_at;   // [nspec] {step, line}
  const int* well_slot;  // [nspec]
  const int* well_ptr;   // [2][nspec + 1]
  const unsigned short* well_code;
  const T* well_val;
  const T* well_piv;     // [nspec]
  // factor records, four values per row; FP64: a step's first halves, then its second halves
  const T* lrec;       // L values of the z-, y-, x- neighbours, tag
  const T* brec;       // U values of the x+, y+, z+ neighbours, pivot
  const double* rd;    // [slots] reciprocal of the pivot
  const T* arec;       // [slots][8]: matrix row z-, y-, x-, diagonal, x+, y+, z+, tag
  const double* rhs;   // natural order
  double* x;           // natural order
  unsigned char* work; // slots doubles (iterate), then 9 vectors of `slots` T
  long long* iter_counter;
  int* status;
  long long wait_limit;  // cycles
  int max_iters;
  int lost;              // >= 0: the forward sweeps' message that never arrives complete (tests), else -1
};

// ---- small device helpers ----
__device__ __forceinline__ unsigned pen_smem(const void* p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ unsigned pen_map(unsigned addr, unsigned rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ unsigned pen_rank() {
  unsigned v;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(v));
  return v;
}
__device__ __forceinline__ unsigned pen_ranks() {
  unsigned v;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(v));
  return v;
}
// all threads of the cluster; memory written before is visible after
__device__ __forceinline__ void pen_sync(int cs) {
  if (cs > 1)
    asm volatile(
        "barrier.cluster.arrive.release.aligned;\n\t"
        "barrier.cluster.wait.acquire.aligned;" ::: "memory");
  else
    __syncthreads();
}
__device__ __forceinline__ void pen_bar(int threads) {
  asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
}
__device__ __forceinline__ double lds(unsigned a, double) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float lds(unsigned a, float) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ int lds_i(unsigned a) {
  int v;
  asm volatile("ld.shared.s32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ int2 lds_i2(unsigned a) {
  int2 v;
  asm volatile("ld.shared.v2.s32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void sts(unsigned a, double v) {
  asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void sts(unsigned a, float v) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void sts(unsigned a, int v) {
  asm volatile("st.shared.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
// a store under a condition without a branch
__device__ __forceinline__ void sts_if(int on, unsigned a, double v) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %0, 0;\n\t@q st.shared.f64 [%1], %2;\n\t}" ::"r"(on), "r"(a), "d"(v)
               : "memory");
}
__device__ __forceinline__ void sts_if(int on, unsigned a, float v) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %0, 0;\n\t@q st.shared.f32 [%1], %2;\n\t}" ::"r"(on), "r"(a), "f"(v)
               : "memory");
}
__device__ __forceinline__ void lds4(unsigned a, unsigned half, double& w, double& x, double& y, double& z) {
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(w), "=d"(x) : "r"(a) : "memory");
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(y), "=d"(z) : "r"(a + half) : "memory");
}
__device__ __forceinline__ void lds4(unsigned a, unsigned, float& w, float& x, float& y, float& z) {
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(w), "=f"(x), "=f"(y), "=f"(z) : "r"(a) : "memory");
}
// Bulk copies: 16-byte aligned addresses and sizes (pen_stride).
__device__ __forceinline__ void bulk_in(unsigned dst, const void* src, unsigned bytes, unsigned bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void bulk_out(void* dst, unsigned src, unsigned bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes)
               : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
// between accesses by threads and by bulk copies, of shared memory alone or of all memory
__device__ __forceinline__ void proxy_fence_shared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async;" ::: "memory"); }
__device__ __forceinline__ void st_async(unsigned addr, double v, unsigned mbar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr),
               "l"(__double_as_longlong(v)), "r"(mbar)
               : "memory");
}
__device__ __forceinline__ void st_async(unsigned addr, float v, unsigned mbar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr),
               "r"(__float_as_int(v)), "r"(mbar)
               : "memory");
}
__device__ __forceinline__ bool mbar_try(unsigned bar, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n\t.reg .pred q;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 q, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}
// bounded wait for the phase of parity `parity`, a lane's own; false when it gave up
__device__ __forceinline__ bool mbar_wait_cluster(unsigned bar, unsigned parity, const long long& limit) {
  if (mbar_try(bar, parity)) return true;
  const long long t0 = clock64(), most = limit;
  do {
    if (mbar_try(bar, parity)) return true;
  } while (clock64() - t0 < most);
  return false;
}
// four values of a constant array with one 32-byte (FP64) or 16-byte load; a 32-byte sector holds two
// of the FP32 ones, so those stay in L1 for the second (without: 127x101x40, 77 -> 71 ms per solve)
__device__ __forceinline__ void ld4(const double* p, double& a, double& b, double& c, double& d) {
  asm volatile("ld.global.nc.L1::no_allocate.v4.f64 {%0, %1, %2, %3}, [%4];"
               : "=d"(a), "=d"(b), "=d"(c), "=d"(d)
               : "l"(p));
}
__device__ __forceinline__ void ld4(const float* p, float& a, float& b, float& c, float& d) {
  asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(a), "=f"(b), "=f"(c), "=f"(d)
               : "l"(p));
}
__device__ __forceinline__ int tag_of(double v) { return __double2loint(v); }
__device__ __forceinline__ int tag_of(float v) { return __float_as_int(v); }

// One direction's sweeps of one CTA; kept in shared memory.
template <class T>
struct PenSweep {
  const T* rec;        // factor records of the CTA's first step
  const double* rd;    // reciprocals (backward)
  int* status;
  long long first;     // its slot
  long long limit;     // cycles a wait may take
  int lost;            // as in PenArgs
  int nx, nz, jc, steps, rounded, chunk, stride, ct, nbar, c, cs;
  int nwell;           // listed rows
  unsigned rows, ghost;                                                 // result rows, the neighbour's column
  unsigned place, full;                                                 // copied rows, their mbarriers
  unsigned nbr, mbar;                                                   // neighbour's values and mbarriers
  unsigned bad, gave;  // flags: a quotient needs the division; a wait gave up
  unsigned well_in, well_y, well_x, piv, at, slot, ptr, code, val;
};
// What the passes by slot and the reductions need of the CTA.
struct PenCta {
  int c, cs, j0, jc, stride, lo, hi;  // rank, CTAs, columns, row stride, slots [lo, hi)
};

// The line warps of a sweep.  FWD: y = in - L y; else out = U^-1 y.  R lines per thread.  GENERAL:
// the IEEE division in every row (after a quotient outside pen_div's range).  Row m's copied values
// and its result lie at place m modulo two chunks; threads past the last line repeat it.
template <class T, bool FWD, int R, bool GENERAL>
__device__ __noinline__ void pen_line(const PenSweep<T>& w) {
  constexpr unsigned B = sizeof(T);
  const int nz = w.nz, jc = w.jc, P = jc * nz, stride = w.stride, nbar = w.nbar, CT = w.ct, rounded = w.rounded,
            ring = 2 * w.chunk;
  const unsigned RB = B * unsigned(stride);
  // copied rows: a place's records, inputs and reciprocals are three arrays over the ring, so that
  // a chunk of each is one copy
  const unsigned recs = w.place, ins = recs + unsigned(ring) * 4u * RB, rds = ins + unsigned(ring) * RB;
  const unsigned half = 16u * unsigned(stride);
  unsigned ax[R], ay[R], az[R], ym[R], yg[R], zm[R], pl[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int p = min(int(threadIdx.x) + r * CT, stride - 1), k = p / jc, j = p - k * jc;
    const bool real = p < P, zs = real && (FWD ? k > 0 : k < nz - 1), ys = real && (FWD ? j > 0 : j < jc - 1),
               recv = real && (FWD ? w.c > 0 : w.c + 1 < w.cs);
    const int d = FWD ? -1 : 1;
    const unsigned zero = w.ghost + B * unsigned(2 * nz);
    az[r] = zs ? w.rows + B * unsigned(p + d * jc) : zero;
    ay[r] = ys ? w.rows + B * unsigned(p + d) : recv ? w.ghost + B * unsigned(k) : zero;
    ax[r] = w.rows + B * unsigned(p);
    zm[r] = zs ? ~0u : 0u;             // offset of the step before's row
    ym[r] = ys ? ~0u : 0u;
    yg[r] = !ys && recv ? ~0u : 0u;    // which of the neighbour's columns
    pl[r] = unsigned(p);
  }
  const int m0 = FWD ? 0 : rounded - 1;
  int at = m0 % ring;  // place of the row read next
  unsigned cur = unsigned(at) * RB, prev = unsigned((at + (FWD ? ring - 1 : 1)) % ring) * RB, par = 0;
  const unsigned last = unsigned(ring - 1) * RB, gb = B * unsigned(nz);
  T f0[R], f1[R], f2[R], f3[R], in[R];
  double rd[R];
  // a step's copied row, read before the step's barrier
  auto read = [&]() {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      lds4(recs + unsigned(at) * 4u * RB + 16u * pl[r], half, f0[r], f1[r], f2[r], f3[r]);
      in[r] = lds(ins + unsigned(at) * RB + B * pl[r], T(0));
      if (!FWD) rd[r] = lds(rds + 8u * (unsigned(at) * unsigned(stride) + pl[r]), 0.0);
    }
    at = FWD ? (at + 1 == ring ? 0 : at + 1) : (at == 0 ? ring - 1 : at - 1);
  };
  int bad = 0;
  pen_bar(nbar);
  read();
#pragma unroll 1
  for (int b = 0; b < rounded; ++b) {
    unsigned yo[R], zo[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      yo[r] = ay[r] + (prev & ym[r]) + (par & yg[r]);
      zo[r] = az[r] + (prev & zm[r]);
    }
    pen_bar(nbar);
    T dx[R], dy[R], dz[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      dz[r] = lds(zo[r], T(0));
      dy[r] = lds(yo[r], T(0));
      dx[r] = lds(ax[r] + prev, T(0));
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      T s = in[r];
      int keep;
      if (FWD) {
        s -= f0[r] * dz[r];
        s -= f1[r] * dy[r];
        s -= f2[r] * dx[r];
        keep = tag_of(f3[r]) == 0 ? 1 : 0;
      } else {
        s -= f0[r] * dx[r];
        s -= f1[r] * dy[r];
        s -= f2[r] * dz[r];
        keep = unsigned(__double2hiint(rd[r])) != kPenSpecial ? 1 : 0;
        if (GENERAL) {
          s = f3[r] != T(0) ? s / f3[r] : s;  // 0: outside the line
        } else {
          bool ok;
          s = pen_div(s, f3[r], rd[r], ok);
          bad |= ok ? 0 : keep;
        }
      }
      sts_if(keep, ax[r] + cur, s);
    }
    read();
    prev = cur;
    cur = FWD ? (cur == last ? 0u : cur + RB) : (cur == 0 ? last : cur - RB);
    par ^= gb;
  }
  pen_bar(nbar);
  if (!FWD && !GENERAL && bad) sts(w.bad, 1);
}

// All lanes of a warp of which a wait gave up.
template <class T>
__device__ __forceinline__ void pen_gave_up(const PenSweep<T>& w) {
  if ((threadIdx.x & 31) != 0) return;
  sts(w.gave, 1);
  if (w.status) atomicExch(w.status, 3);
}

// The copying warp.  At the start of a chunk it writes the chunk before's results to `out` and
// starts the copies of the next one in their places; before a chunk's last step it waits for the
// next chunk (whose first row the line warps read then), and for the results' places to be free.
// Once a wait has given up, here or in a sweep before, it starts no copies and waits for none, so that
// no mbarrier is armed again before its phase has ended, and it ends after those in flight.
template <class T, bool FWD>
__device__ __noinline__ void pen_load(const PenSweep<T>& w, unsigned phase0, const T* in_, T* out_) {
  constexpr unsigned B = sizeof(T);
  const int stride = w.stride, rounded = w.rounded, nbar = w.nbar, G = w.chunk, chunks = rounded / G,
            lane = threadIdx.x & 31;
  const unsigned full = w.full, RB = B * unsigned(stride);
  const unsigned recs = w.place, ins = recs + unsigned(2 * G) * 4u * RB, rds = ins + unsigned(2 * G) * RB;
  const unsigned cb = unsigned(G) * RB, db = 8u * unsigned(G) * unsigned(stride);
  // chunk number c of the sweep covers the rows [G k, G k + G), k = c or, backward, from the end
  // the same for all lanes; no forward sweep starts after a wait gave up
  bool ok = FWD || lds_i(w.gave) == 0;
  unsigned open = 0;             // the halves whose copies have not been waited for
  auto issue = [&](int c) {
    if (!ok || c >= chunks) return;
    const int k = FWD ? c : chunks - 1 - c;
    const unsigned h = unsigned(k & 1), bar = full + 8u * h;
    open |= 1u << h;
    if (lane != 0) return;
    const long long row = (long long)k * G * stride;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(5u * cb + (FWD ? 0u : db))
                 : "memory");
    bulk_in(recs + h * 4u * cb, w.rec + 4 * row, 4u * cb, bar);
    bulk_in(ins + h * cb, in_ + w.first + row, cb, bar);
    if (!FWD) bulk_in(rds + h * db, w.rd + row, db, bar);
  };
  auto write = [&](int c) {
    const int k = FWD ? c : chunks - 1 - c;
    bulk_out(out_ + w.first + (long long)k * G * stride, w.rows + unsigned(k & 1) * cb, cb);
  };
  // phases of the two mbarriers: phase0 holds their parities at the start of the sweep
  unsigned par = phase0;
  auto wait = [&](int c) {
    if (!ok) return;
    const unsigned h = unsigned((FWD ? c : chunks - 1 - c) & 1);
    const bool got = mbar_wait_cluster(full + 8u * h, (par >> h) & 1u, w.limit);
    ok = __all_sync(0xffffffffu, got);
    if (!ok) return;
    par ^= 1u << h;
    open &= ~(1u << h);
  };
  issue(0);
  issue(1);
  wait(0);
  pen_bar(nbar);  // the line warps read the first row
#pragma unroll 1
  for (int c = 0; c < chunks; ++c) {
#pragma unroll 1
    for (int t = 0; t < G; ++t) {
      if (t == G - 1 && c + 1 < chunks) wait(c + 1);
      // chunk c's results take the place of chunk c - 2's
      if (t == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
      pen_bar(nbar);
      if (t == 0 && c > 0) {
        if (lane == 0) {
          proxy_fence_shared();
          write(c - 1);
        }
        issue(c + 1);
      }
    }
  }
  pen_bar(nbar);
  if (lane == 0) {
    proxy_fence_shared();
    write(chunks - 1);
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  if (ok) return;
  pen_gave_up(w);
  for (unsigned h = 0; h < 2; ++h)
    if ((open >> h) & 1u) mbar_wait_cluster(full + 8u * h, (par >> h) & 1u, w.limit);
  __syncwarp();
}

// The receiving warp: before each step's barrier it waits for the neighbouring CTA's values of the
// step before and puts them into the result row.  Lane k takes layer k (and k + 32, ...).  A lane whose
// wait gave up waits no more in this sweep; all lanes take the same steps and barriers all the same.
template <class T, bool FWD>
__device__ __noinline__ void pen_recv(const PenSweep<T>& w, unsigned phase) {
  constexpr unsigned B = sizeof(T);
  const int lane = threadIdx.x & 31, nx = w.nx, nz = w.nz, NM = nx + nz - 1, rounded = w.rounded, nbar = w.nbar;
  for (int u = lane; u < NM; u += 32) {
    const int cnt = min(nz - 1, u) - max(0, u - nx + 1) + 1;  // lines k with 0 <= u - k < nx
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(w.mbar + 8u * unsigned(u)),
                 "r"(unsigned((FWD && u == w.lost ? cnt + 1 : cnt) * sizeof(T)))
                 : "memory");
  }
  __syncwarp();
  bool ok = true;  // a lane's own
  // step b reads the values sent as number u: b, or backward b less the rounding to whole chunks
  const int skip = FWD ? 0 : rounded - w.steps;
  const int kk = FWD ? lane : nz - 1 - lane;  // place in the message
  unsigned mb = w.mbar, to = w.ghost + B * unsigned(lane), from = w.nbr + B * unsigned(kk);
  const unsigned gb = B * unsigned(nz), to_sum = 2 * to + gb;  // the two columns alternate
  if (skip & 1) to = to_sum - to;
  pen_bar(nbar);
#pragma unroll 1
  for (int b = 0; b < skip; ++b) pen_bar(nbar);
  const int steps = rounded - skip;
#pragma unroll 1
  for (int u = 0; u < steps; ++u) {
    if (u < NM) {
      if (ok) ok = mbar_wait_cluster(mb, phase, w.limit);
      if (lane < nz && unsigned(u - kk) < unsigned(nx)) sts(to, lds(from, T(0)));
      for (int k = lane + 32; k < nz; k += 32) {
        const int q = FWD ? k : nz - 1 - k;
        if (unsigned(u - q) < unsigned(nx))
          sts(to + B * unsigned(k - lane), lds(w.nbr + B * unsigned(u * nz + q), T(0)));
      }
      __syncwarp();
      mb += 8;
      from += gb;
    }
    to = to_sum - to;
    pen_bar(nbar);
  }
  pen_bar(nbar);
  if (!__all_sync(0xffffffffu, ok)) pen_gave_up(w);
}

// The sending warp (of a CTA with listed rows, or a neighbour to send to): after each step's
// barrier it solves the step's listed rows, then sends the step before's values of the CTA's last
// (backward: first) column on, lane k layer k.  A listed row's entries (the first 32) are in
// registers before its step, an entry per lane: what a step takes is one read, a product per lane
// and the sum in entry order.
template <class T, bool FWD>
__device__ __noinline__ void pen_send(const PenSweep<T>& w, const T* in) {
  constexpr unsigned B = sizeof(T);
  const int lane = threadIdx.x & 31, nx = w.nx, nz = w.nz, jc = w.jc, NM = nx + nz - 1, rounded = w.rounded,
            nbar = w.nbar, nwell = w.nwell, ring = 2 * w.chunk, stride = w.stride;
  const unsigned RB = B * unsigned(stride), last = w.rows + unsigned(ring - 1) * RB, rows = w.rows;
  const bool sends = FWD ? w.c + 1 < w.cs : w.c > 0;
  const unsigned wy = FWD ? w.well_y : w.well_x, gb = B * unsigned(nz);
  unsigned rring = 0, rmbar = 0;
  if (sends) {
    const unsigned to = unsigned(FWD ? w.c + 1 : w.c - 1);
    rring = pen_map(w.nbr, to);
    rmbar = pen_map(w.mbar, to);
  }
  // the listed rows' right-hand sides: forward from `in`, backward the forward sweep's values
  if (FWD)
    for (int e = lane; e < nwell; e += 32)
      sts(w.well_in + B * unsigned(e), in[lds_i(w.slot + 4u * unsigned(e))]);
  __syncwarp();
  // the next listed row: step, line's offset, right-hand side, this lane's entry (address, of the row
  // before or of the neighbour's column of the step's parity, or fixed)
  int e = FWD ? 0 : nwell - 1, at = -1, e0 = 0, cnt = 0;
  unsigned line = 0, ea = 0, em = 0, eg = 0;
  T ev = T(0), es = T(0), piv = T(1);
  auto entry = [&](int k, unsigned& ad, unsigned& rm, unsigned& gm, T& v) {
    unsigned short c;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(c) : "r"(w.code + 2u * unsigned(k)) : "memory");
    v = lds(w.val + B * unsigned(k), T(0));
    const bool far = (c & 0x8000u) != 0, col = !far && int(c) >= stride;
    ad = far ? wy + B * unsigned(c & 0x7fffu) : col ? w.ghost + B * unsigned(int(c) - stride) : B * unsigned(c);
    rm = far || col ? 0u : ~0u;
    gm = col ? ~0u : 0u;
  };
  auto next_row = [&]() {
    at = -1;
    if (e < 0 || e >= nwell) return;
    at = lds_i(w.at + 8u * unsigned(e));
    line = B * unsigned(lds_i(w.at + 8u * unsigned(e) + 4u));
    const unsigned ptr = w.ptr + 4u * unsigned(FWD ? e : nwell + 1 + e);
    e0 = lds_i(ptr);
    cnt = lds_i(ptr + 4) - e0;
    es = lds((FWD ? w.well_in : w.well_y) + B * unsigned(e), T(0));
    if (!FWD) piv = lds(w.piv + B * unsigned(e), T(0));
    ev = T(0);
    ea = em = eg = 0;
    if (lane < cnt) entry(e0 + lane, ea, em, eg, ev);
    if (lane >= cnt) ea = w.ghost + 2 * gb;  // the zero
  };
  next_row();
  int m = FWD ? 0 : rounded - 1;
  unsigned cur = rows + unsigned(m & (ring - 1)) * RB,
           prev = rows + unsigned((m + (FWD ? ring - 1 : 1)) & (ring - 1)) * RB, par = 0;
  // the values sent after the barrier of step b are number u = b - u0 of the receiver's
  const int kk = lane, k0 = FWD ? kk : nz - 1 - kk;
  int u = FWD ? -jc : nx + nz - 2 - rounded;
  const unsigned edge = B * unsigned(k0 * jc + (FWD ? jc - 1 : 0));
  pen_bar(nbar);
#pragma unroll 1
  for (int b = 0; b <= rounded; ++b) {
    pen_bar(nbar);
    while (at == m && b < rounded) {  // several listed rows may share a step
      T pr = ev * lds(ea + (prev & em) + (par & eg), T(0));
      T s = es;
#pragma unroll 1
      for (int k = 0; k < cnt; k += 32) {
        const int n = min(32, cnt - k);
        if (k > 0) {
          pr = T(0);
          if (lane < n) {
            unsigned ad, rm, gm;
            T v;
            entry(e0 + k + lane, ad, rm, gm, v);
            pr = v * lds(ad + (prev & rm) + (par & gm), T(0));
          }
        }
#pragma unroll 1
        for (int t = 0; t < n; t += 4) {  // lanes past the last entry hold zero: s - 0 is s
          const T p0 = __shfl_sync(0xffffffffu, pr, t), p1 = __shfl_sync(0xffffffffu, pr, t + 1),
                  p2 = __shfl_sync(0xffffffffu, pr, t + 2), p3 = __shfl_sync(0xffffffffu, pr, t + 3);
          s -= p0;
          s -= p1;
          s -= p2;
          s -= p3;
        }
      }
      if (!FWD) s = s / piv;
      if (lane == 0) {
        sts(cur + line, s);
        sts(wy + B * unsigned(e), s);
      }
      __syncwarp();
      e += FWD ? 1 : -1;
      next_row();
    }
    if (sends) {
      if (unsigned(u) < unsigned(NM)) {
        if (kk < nz && unsigned(u - kk) < unsigned(nx))
          st_async(rring + B * unsigned(u * nz + kk), lds(prev + edge, T(0)), rmbar + 8u * unsigned(u));
        for (int q = lane + 32; q < nz; q += 32)
          if (unsigned(u - q) < unsigned(nx))
            st_async(rring + B * unsigned(u * nz + q),
                     lds(prev + B * unsigned((FWD ? q : nz - 1 - q) * jc + (FWD ? jc - 1 : 0)), T(0)),
                     rmbar + 8u * unsigned(u));
      }
      __syncwarp();
      ++u;
    }
    prev = cur;
    cur = FWD ? (cur == last ? rows : cur + RB) : (cur == rows ? last : cur - RB);
    par ^= gb;
    m += FWD ? 1 : -1;
  }
}

// One sweep; called by all threads, the caller synchronises the CTA afterwards.  phase0: parities of
// the copies' mbarriers, phase: of the neighbour's.
template <class T, bool FWD>
__device__ __forceinline__ void pen_sweep(const PenSweep<T>& w, unsigned phase0, const T* in, T* out, unsigned phase,
                                          bool general) {
  const int warp = int(threadIdx.x) >> 5;
  if (warp == kPenLoadWarp) {
    pen_load<T, FWD>(w, phase0, in, out);
  } else if (warp == kPenSendWarp) {
    if (w.nwell > 0 || (FWD ? w.c + 1 < w.cs : w.c > 0)) pen_send<T, FWD>(w, in);
  } else if (warp == kPenRecvWarp) {
    if (FWD ? w.c > 0 : w.c + 1 < w.cs) pen_recv<T, FWD>(w, phase);
  } else if (int(threadIdx.x) < w.ct) {
    if (w.stride <= kPenLineThreads) {
      if (FWD || !general)
        pen_line<T, FWD, 1, false>(w);
      else
        pen_line<T, false, 1, true>(w);
    } else {
      if (FWD || !general)
        pen_line<T, FWD, 2, false>(w);
      else
        pen_line<T, false, 2, true>(w);
    }
  }
}

// Zeros in the result rows and the neighbour's columns, which lines outside their cells read times zero.
template <class T>
__device__ __noinline__ void pen_clear(const PenSweep<T>& w) {
  constexpr unsigned B = sizeof(T);
  for (int e = threadIdx.x; e < 2 * w.chunk * w.stride; e += kPenThreads) sts(w.rows + B * unsigned(e), T(0));
  for (int e = threadIdx.x; e < 2 * w.nz; e += kPenThreads) sts(w.ghost + B * unsigned(e), T(0));
}

// out = A in on the CTA's cells.  A thread takes part of a line: the x neighbours come from its own
// loads, the y and z ones at constant distances (in a neighbouring CTA's region with its own).  Rows
// with entries outside the stencil take a warp each.
template <class T>
__device__ __noinline__ void pen_spmv(const PenArgs<T>& a, const PenCta& g, const T* in, T* out) {
  const int nx = a.nx, nz = a.nz, jc = g.jc, lines = jc * nz, P = g.stride;
  const int segs = max(1, kPenThreads / lines);
  for (int t = threadIdx.x; t < lines * segs; t += kPenThreads) {
    const int line = t % lines, sg = t / lines, k = line / jc, j = line - k * jc;
    const int i0 = nx * sg / segs, i1 = nx * (sg + 1) / segs;
    const long long row = (long long)g.lo + (long long)(kPenGuard + i0 + j + k) * P + line;
    // y neighbours: same region, or the neighbouring CTA's last / first column
    long long ym = row - P - 1, yp = row + P + 1;
    int dym = P, dyp = P;
    if (j == 0 && g.c > 0) {
      const int jn = pen_first_col(g.c, g.cs, a.ny) - pen_first_col(g.c - 1, g.cs, a.ny);
      dym = pen_stride(jn * nz);
      ym = (long long)a.cta[g.c - 1] + (long long)(kPenGuard + i0 + jn - 1 + k) * dym + k * jn + jn - 1;
    }
    if (j == jc - 1 && g.c + 1 < g.cs) {
      const int jn = pen_first_col(g.c + 2, g.cs, a.ny) - pen_first_col(g.c + 1, g.cs, a.ny);
      dyp = pen_stride(jn * nz);
      yp = (long long)a.cta[g.c + 1] + (long long)(kPenGuard + i0 + k) * dyp + k * jn;
    }
    const T* ar = a.arec + 8 * row;
    const T* c = in + row;
    const T* cym = in + ym;
    const T* cyp = in + yp;
    T* o = out + row;
    const int up = P + jc;  // z neighbours: one step and one layer of lines away
    T xm = c[-P], x0 = c[0];
    constexpr int U = 2;
#pragma unroll 1
    for (int i = i0; i < i1; i += U) {
      T m[U][8], vx[U], vym[U], vyp[U], vzm[U], vzp[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {  // past the line's end: guard rows
        ld4(ar + 8 * u * P, m[u][0], m[u][1], m[u][2], m[u][3]);
        ld4(ar + 8 * u * P + 4, m[u][4], m[u][5], m[u][6], m[u][7]);
        vx[u] = c[(u + 1) * P];
        vzm[u] = c[u * P - up];
        vzp[u] = c[u * P + up];
        vym[u] = cym[u * dym];
        vyp[u] = cyp[u * dyp];
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        T s = T(0);
        s += m[u][0] * vzm[u];
        s += m[u][1] * vym[u];
        s += m[u][2] * xm;
        s += m[u][3] * x0;
        s += m[u][4] * vx[u];
        s += m[u][5] * vyp[u];
        s += m[u][6] * vzp[u];
        if (i + u < i1 && tag_of(m[u][7]) == 0) o[u * P] = s;
        xm = x0;
        x0 = vx[u];
      }
      ar += 8 * U * P;
      c += U * P;
      cym += U * dym;
      cyp += U * dyp;
      o += U * P;
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = kPenThreads / 32, nspec = a.nspec;
  for (int e = g.c + g.cs * warp; e < nspec; e += g.cs * nw) {
    const int k0 = __ldg(a.spec_ptr + e), k1 = __ldg(a.spec_ptr + e + 1);
    T s = T(0);
    for (int k = k0; k < k1; k += 32) {
      const T pr = k + lane < k1 ? a.spec_val[k + lane] * in[__ldg(a.spec_col + k + lane)] : T(0);
      const int cnt = min(32, k1 - k);
      for (int u = 0; u < cnt; ++u) s += __shfl_sync(0xffffffffu, pr, u);
    }
    if (lane == 0) out[__ldg(a.spec_slot + e)] = s;
  }
}

// A virtual warp's two sums to every CTA's `red`.
__device__ __forceinline__ void pen_publish(double s0, double s1, double* red, int v, int nvw, int cs) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int h = 16; h > 0; h >>= 1) {
    s0 += __shfl_down_sync(0xffffffffu, s0, h);
    s1 += __shfl_down_sync(0xffffffffu, s1, h);
  }
  s0 = __shfl_sync(0xffffffffu, s0, 0);
  s1 = __shfl_sync(0xffffffffu, s1, 0);
  if (lane < cs) {
    const unsigned at = pen_smem(red + v);
    const unsigned r0 = pen_map(at, unsigned(lane)), r1 = pen_map(at + 8u * unsigned(nvw), unsigned(lane));
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(r0), "d"(s0) : "memory");
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(r1), "d"(s1) : "memory");
  }
}
// After all virtual warps' sums: cluster barrier, each block's warps by a shuffle tree, the blocks
// in order; every thread gets both totals.
__device__ __forceinline__ double2 pen_totals(const DotOrder& o, const double* red, int nvw, int cs) {
  pen_sync(cs);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, vwpb = o.vwpb, vblocks = o.vblocks;
  __shared__ double tot[2][16];
  double x0 = 0.0, x1 = 0.0;
  if (warp < vblocks || vblocks == 1) {
    const int b = vblocks == 1 ? 0 : warp;
    if (lane < vwpb) {
      x0 = red[b * vwpb + lane];
      x1 = red[nvw + b * vwpb + lane];
    }
#pragma unroll
    for (int h = 16; h > 0; h >>= 1) {
      x0 += __shfl_down_sync(0xffffffffu, x0, h);
      x1 += __shfl_down_sync(0xffffffffu, x1, h);
    }
    x0 = __shfl_sync(0xffffffffu, x0, 0);
    x1 = __shfl_sync(0xffffffffu, x1, 0);
  }
  if (vblocks == 1) return make_double2(x0, x1);
  if (warp < vblocks && lane == 0) {
    tot[0][warp] = x0;
    tot[1][warp] = x1;
  }
  __syncthreads();
  x0 = x1 = 0.0;
  for (int b = 0; b < vblocks; ++b) {
    x0 += tot[0][b];
    x1 += tot[1][b];
  }
  __syncthreads();
  return make_double2(x0, x1);
}

// The dot products x0 . y0 and x1 . y1 (TWO) in the order of DotOrder: `list` holds, for each
// virtual warp (first chunk at ptr[v]), chunks of 32 slots, lane by lane, in the order of its
// sums (-1: none).  S_PASS: x0 = r, y0 = v, and s = r - alpha v is formed, stored to x1 and squared.
// The loads of U chunks are unconditional and issued together: one at a time, each chunk would
// cost a round trip.
template <class T, bool TWO, bool S_PASS>
__device__ __noinline__ double2 pen_dots(const DotOrder& o, const PenCta& g, double* red, const int* ptr,
                                         const int* list, const T* x0, const T* y0, T* x1, const T* y1, double alpha) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = kPenThreads / 32, cs = g.cs;
  const int nvw = o.vblocks * o.vwpb;
  for (int v = g.c + cs * warp; v < nvw; v += cs * nw) {
    const int end = 32 * ptr[v + 1] + lane;
    double s0 = 0.0, s1 = 0.0;
    constexpr int U = 8;
    int q[U], next[U];
#pragma unroll
    for (int h = 0; h < U; ++h) next[h] = __ldg(list + 32 * (ptr[v] + h) + lane);
#pragma unroll 1
    for (int e = 32 * ptr[v] + lane; e < end; e += 32 * U) {
      T u0[U], w0[U], u1[U], w1[U];
#pragma unroll
      for (int h = 0; h < U; ++h) {
        q[h] = next[h];
        next[h] = __ldg(list + e + 32 * (U + h));  // 2 U chunks of -1 end the list
      }
#pragma unroll
      for (int h = 0; h < U; ++h) {
        const int at = max(q[h], 0);
        u0[h] = x0[at];
        w0[h] = y0[at];
        if (TWO) {
          u1[h] = x1[at];
          w1[h] = y1[at];
        }
      }
#pragma unroll
      for (int h = 0; h < U; ++h) {
        // a lane without an element adds zero (the sums start at +0 and so are never -0)
        const bool on = q[h] >= 0 && e + 32 * h < end;
        double p0;
        if (S_PASS) {
          const T si = T(double(u0[h]) - alpha * double(w0[h]));
          if (on) x1[q[h]] = si;
          p0 = double(si) * double(si);
        } else {
          p0 = double(u0[h]) * double(w0[h]);
        }
        s0 += on ? p0 : 0.0;
        if (TWO) s1 += on ? double(u1[h]) * double(w1[h]) : 0.0;
      }
    }
    pen_publish(s0, s1, red, v, nvw, cs);
  }
  return pen_totals(o, red, nvw, cs);
}

// After a wait gave up, when no CTA sends any more: waits, bounded, for the values still on their way
// into this CTA.  phase_f, phase_b: parities of the last forward and backward sweep's mbarriers.
template <class T>
__device__ __noinline__ void pen_drain(const PenSweep<T>* w, unsigned phase_f, unsigned phase_b) {
  const int NM = w[0].nx + w[0].nz - 1;
  for (int m = threadIdx.x; m < NM; m += kPenThreads) {
    if (w[0].c > 0) mbar_wait_cluster(w[0].mbar + 8u * unsigned(m), phase_f, w[0].limit);
    if (w[0].c + 1 < w[0].cs) mbar_wait_cluster(w[1].mbar + 8u * unsigned(m), phase_b, w[0].limit);
  }
  __syncwarp();
}

template <class T>
__device__ void pen_body(const PenArgs<T>& a, unsigned char* raw) {
  // a solve that gave up has left its mark, which the host reads after the linear solve
  if (a.status && *(const volatile int*)a.status != 0) return;
  __shared__ PenSweep<T> sweep[2];
  __shared__ PenCta shared_cta;
  PenCta g;
  g.cs = int(pen_ranks());
  g.c = int(pen_rank());
  g.j0 = pen_first_col(g.c, g.cs, a.ny);
  g.jc = pen_first_col(g.c + 1, g.cs, a.ny) - g.j0;
  g.lo = a.cta[g.c];
  g.hi = a.cta[g.c + 1];
  const int tid = threadIdx.x, nt = kPenThreads, lo = g.lo, hi = g.hi;
  const int n = a.n, nx = a.nx, nz = a.nz, P = g.stride = pen_stride(g.jc * nz);
  const int nvw = a.dot.vblocks * a.dot.vwpb;
  const int cols = (a.ny + g.cs - 1) / g.cs;  // the widest CTA's columns
  const int w0 = a.well_cta[g.c], nwell = a.well_cta[g.c + 1] - w0;
  const int wells = a.well_cta[g.cs];  // the entry ranges' second half starts at wells + 1
  const int f0 = a.well_ptr[w0], f1 = a.well_ptr[w0 + nwell];
  const int b0 = a.well_ptr[wells + 1 + w0], b1 = a.well_ptr[wells + 1 + w0 + nwell];
  const PenLayout o = pen_layout<T>(nx, nz, cols, g.cs, a.chunk, nvw, nwell, f1 - f0 + b1 - b0);
  double* const red_base = reinterpret_cast<double*>(raw + o.red);
  const unsigned bad_at = pen_smem(raw + o.bad), gave_at = bad_at + 4u;
  for (int e = tid; e < 2 * a.chunk * P; e += nt) reinterpret_cast<T*>(raw + o.rows)[e] = T(0);
  for (int e = tid; e <= 2 * nz; e += nt) reinterpret_cast<T*>(raw + o.ghost)[e] = T(0);
  for (int e = tid; e < nwell; e += nt) {
    reinterpret_cast<int2*>(raw + o.at)[e] = a.well_at[w0 + e];
    reinterpret_cast<int*>(raw + o.slot)[e] = a.well_slot[w0 + e];
    reinterpret_cast<T*>(raw + o.piv)[e] = a.well_piv[w0 + e];
  }
  for (int e = tid; e <= nwell; e += nt) {
    reinterpret_cast<int*>(raw + o.ptr)[e] = a.well_ptr[w0 + e] - f0;
    reinterpret_cast<int*>(raw + o.ptr)[nwell + 1 + e] = a.well_ptr[wells + 1 + w0 + e] - b0 + (f1 - f0);
  }
  for (int e = tid; e < f1 - f0 + b1 - b0; e += nt) {
    const int from = e < f1 - f0 ? f0 + e : b0 + e - (f1 - f0);
    reinterpret_cast<unsigned short*>(raw + o.code)[e] = a.well_code[from];
    reinterpret_cast<T*>(raw + o.val)[e] = a.well_val[from];
  }
  if (g.cs > 1)
    for (int m = tid; m < 2 * (nx + nz - 1); m += nt)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(pen_smem(raw + o.mbar) + 8u * unsigned(m)) : "memory");
  if (tid < 2)
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(pen_smem(raw + o.full) + 8u * unsigned(tid)) : "memory");
  if (tid == 0) {
    sts(bad_at, 0);
    sts(gave_at, 0);
    shared_cta = g;
  }
  if (tid < 2) {
    PenSweep<T> w;
    const long long first = (long long)lo + (long long)kPenGuard * P;
    w.rec = (tid == 0 ? a.lrec : a.brec) + 4 * first;
    w.rd = a.rd + first;
    w.status = a.status;
    w.first = first;
    w.nx = nx, w.nz = nz, w.jc = g.jc, w.c = g.c, w.cs = g.cs, w.nwell = nwell, w.chunk = a.chunk;
    w.steps = pen_steps(nx, g.jc, nz), w.rounded = pen_rounded(w.steps, a.chunk);
    w.stride = P;
    w.ct = ((P <= kPenLineThreads ? P : (P + 1) / 2) + 31) / 32 * 32;
    // line warps, the copying warp, where there are any the receiving and the sending warp
    const bool below = g.c > 0, above = g.c + 1 < g.cs;
    w.nbar = w.ct + 32 + ((tid == 0 ? below : above) ? 32 : 0) + (nwell > 0 || (tid == 0 ? above : below) ? 32 : 0);
    w.rows = pen_smem(raw + o.rows), w.ghost = pen_smem(raw + o.ghost);
    w.place = pen_smem(raw + o.place), w.full = pen_smem(raw + o.full);
    w.nbr = pen_smem(raw + o.nbr), w.bad = bad_at, w.gave = gave_at;
    w.limit = a.wait_limit, w.lost = a.lost;
    w.mbar = pen_smem(raw + o.mbar) + (tid == 0 ? 0u : 8u * unsigned(nx + nz - 1));
    w.well_in = pen_smem(raw + o.well_in), w.well_y = pen_smem(raw + o.well_y), w.well_x = pen_smem(raw + o.well_x);
    w.piv = pen_smem(raw + o.piv), w.at = pen_smem(raw + o.at), w.slot = pen_smem(raw + o.slot);
    w.ptr = pen_smem(raw + o.ptr), w.code = pen_smem(raw + o.code), w.val = pen_smem(raw + o.val);
    sweep[tid] = w;
  }
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  const size_t ns = size_t(a.slots);
  double* xq = reinterpret_cast<double*>(a.work);
  T* r = reinterpret_cast<T*>(a.work + sizeof(double) * ns);
  T *rh = r + ns, *p = r + 2 * ns, *v = r + 3 * ns, *s = r + 4 * ns, *t = r + 5 * ns, *ph = r + 6 * ns,
    *sh = r + 7 * ns, *y = r + 8 * ns;
  // natural rows: scattered into step order, gathered at the end; r is zero in the slots outside the
  // lines, and so are the vectors formed from it
  const int na = int(unsigned(n) * unsigned(g.c) / unsigned(g.cs)),
            nb = int(unsigned(n) * unsigned(g.c + 1) / unsigned(g.cs));
  for (int q = lo + tid; q < hi; q += nt) r[q] = T(0);
  pen_sync(g.cs);
  for (int i = na + tid; i < nb; i += nt) {
    const int q = a.nat[i];
    const double ri = a.rhs[i] - 0.0;
    const T rt = T(ri);
    xq[q] = 0.0;
    r[q] = rt;
    rh[q] = rt;
    v[q] = T(0);
    p[q] = T(0);
  }
  pen_sync(g.cs);
  int parity = 0;
  auto red = [&]() {  // the sums of one reduction stay while the next one is gathered
    parity ^= 1;
    return red_base + size_t(parity) * 2 * nvw;
  };
  // the orders' first chunks: plain, product, norm of s
  const int* const lp0 = a.list_ptr;
  const int* const lp1 = lp0 + nvw + 1;
  const int* const lp2 = lp1 + nvw + 1;
  const PenCta& gs = shared_cta;
  double2 d = pen_dots<T, false, false>(a.dot, gs, red(), lp0, a.list[0], r, r, nullptr, nullptr, 0.0);
  const double rnorm0 = sqrt(d.x);
  const double tol = fmax(rnorm0, kEpsP) * 1e-6;
  const int max_iters = rnorm0 <= tol ? 0 : a.max_iters;
  double rho = d.x, rho_prev = 1.0, alpha = 1.0, omega = 1.0;
  int started = 0;
  unsigned ph_f = 0, ph_b = 0, ph_c = 0;
  // a sweep completes the copies' two mbarriers once per chunk of theirs
  const int chunks = pen_rounded(pen_steps(nx, g.jc, nz), a.chunk) / a.chunk;
  const unsigned flip = unsigned((chunks + 1) / 2 & 1) | unsigned(chunks / 2 & 1) << 1;
  bool general = false;  // a backward sweep met a quotient outside pen_div's range
  // Two halves per iteration: p, v = A M^-1 p and alpha; s, t = A M^-1 s and omega.
#pragma unroll 1
  for (int it = 0; it < max_iters; ++it) {
    started = it + 1;
    if (!isfinite(rho) || fabs(rho) < kEpsP) break;
    const double beta = it == 0 ? 0.0 : (rho / rho_prev) * (alpha / omega);
    bool stop = false;
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      T* const mp = half == 0 ? ph : sh;
      T* const ap = half == 0 ? v : t;
      if (half == 0) {
        if (it == 0) {
          for (int q = lo + tid; q < hi; q += nt) p[q] = r[q];
        } else {
          for (int q0 = lo + tid; q0 < hi; q0 += 4 * nt) {
            T r4[4], p4[4], v4[4];
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              const int q = min(q0 + h * nt, hi - 1);
              r4[h] = r[q], p4[h] = p[q], v4[h] = v[q];
            }
#pragma unroll
            for (int h = 0; h < 4; ++h)
              if (q0 + h * nt < hi) p[q0 + h * nt] = T(double(r4[h]) + beta * (double(p4[h]) - omega * double(v4[h])));
          }
        }
        proxy_fence();
        __syncthreads();
      } else {
        d = pen_dots<T, false, true>(a.dot, gs, red(), lp2, a.list[2], r, v, s, nullptr, alpha);
        proxy_fence();
        if (sqrt(d.x) <= tol) {
          for (int q = lo + tid; q < hi; q += nt) xq[q] += alpha * double(ph[q]);
          stop = true;
          break;
        }
      }
      pen_sweep<T, true>(sweep[0], ph_c, half == 0 ? p : s, y, ph_f, false);
      ph_f ^= 1u;
      ph_c ^= flip;
      __syncthreads();
#pragma unroll 1
      for (;;) {
        pen_sweep<T, false>(sweep[1], ph_c, y, mp, ph_b, general);
        ph_b ^= 1u;
        ph_c ^= flip;
        __syncthreads();
        // any CTA's flags reach all of them.  `bad`: the sweep is repeated, and the solve goes on, in
        // the general form; `gave`: the solve ends
        const int2 own = lds_i2(bad_at);
        if ((own.x | own.y) != 0 && tid < g.cs) {
          if (!general && own.x != 0)
            asm volatile("st.shared::cluster.s32 [%0], 1;" ::"r"(pen_map(bad_at, unsigned(tid))) : "memory");
          if (own.y != 0)
            asm volatile("st.shared::cluster.s32 [%0], 1;" ::"r"(pen_map(gave_at, unsigned(tid))) : "memory");
        }
        pen_sync(g.cs);
        const int2 any = lds_i2(bad_at);
        if (any.y != 0) {
          stop = true;
          break;
        }
        if (general || any.x == 0) break;
        general = true;
        pen_clear(sweep[1]);  // the attempt may have left NaNs: pen_div of a pivot that pen_recip refuses
        __syncthreads();
      }
      if (stop) break;
      pen_spmv<T>(a, gs, mp, ap);
      pen_sync(g.cs);
      if (half == 0) {
        d = pen_dots<T, false, false>(a.dot, gs, red(), lp1, a.list[1], rh, v, nullptr, nullptr, 0.0);
        if (!isfinite(d.x) || fabs(d.x) < kEpsP) {
          stop = true;
          break;
        }
        alpha = rho / d.x;
      } else {
        d = pen_dots<T, true, false>(a.dot, gs, red(), lp1, a.list[1], t, t, t, s, 0.0);
      }
    }
    if (stop || !isfinite(d.x) || d.x <= kEpsP) break;
    omega = d.y / d.x;
    if (!isfinite(omega) || fabs(omega) < kEpsP) break;
    // four slots' loads in flight (with those of p above; two at a time: 45x61x7 9.8 -> 8.7 ms per
    // solve, 21x20x5 3.44 -> 3.11, 127x101x40 FP32 71 -> 66)
    for (int q0 = lo + tid; q0 < hi; q0 += 4 * nt) {
      T p4[4], s4[4], r4[4], t4[4];
      double x4[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const int q = min(q0 + h * nt, hi - 1);
        x4[h] = xq[q], p4[h] = ph[q], s4[h] = sh[q], r4[h] = s[q], t4[h] = t[q];
      }
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const int q = q0 + h * nt;
        if (q < hi) {
          xq[q] = x4[h] + (alpha * double(p4[h]) + omega * double(s4[h]));
          r[q] = T(double(r4[h]) - omega * double(t4[h]));
        }
      }
    }
    pen_sync(g.cs);
    d = pen_dots<T, true, false>(a.dot, gs, red(), lp0, a.list[0], r, r, rh, r, 0.0);
    if (sqrt(d.x) <= tol) break;
    rho_prev = rho;
    rho = d.y;
  }
  if (lds_i(gave_at) != 0) pen_drain(sweep, ph_f ^ 1u, ph_b ^ 1u);
  pen_sync(g.cs);
  for (int i = na + tid; i < nb; i += nt) a.x[i] = xq[a.nat[i]];
  if (g.c == 0 && tid == 0 && a.iter_counter)
    atomicAdd((unsigned long long*)a.iter_counter, (unsigned long long)started);
  pen_sync(g.cs);  // no CTA leaves while another may still reach its shared memory
}

// One solve, and many solves in one launch: cluster b solves item b.
template <class T>
struct PenBatch {
  int count;
  PenArgs<T> item[kBatchItems];
};
template <class T>
__global__ void __launch_bounds__(kPenThreads, 1) k_bicgstab_pencil(const __grid_constant__ PenArgs<T> a) {
  extern __shared__ __align__(16) unsigned char pen_raw[];
  pen_body(a, pen_raw);
}
template <class T>
__global__ void __launch_bounds__(kPenThreads, 1) k_bicgstab_pencil_batch(const __grid_constant__ PenBatch<T> b) {
  extern __shared__ __align__(16) unsigned char pen_raw[];
  const unsigned item = blockIdx.x / pen_ranks();
  if (item < unsigned(b.count)) pen_body(b.item[item], pen_raw);
}

// The records from the factors and the pressure matrix (after each factorisation), one thread per
// natural row.
template <class T>
struct PenPack {
  int n, nspec, nwe, nse;
  const int* nat;
  const int* rec_at;   // [n] index of the record's first half (FP64: of 2-value halves), or of the record
  const int* rec_half; // [n] distance to the second half
  const int* stencil;  // n x 7
  const unsigned char* special;  // [n]
  const double* plu;
  const double* pdiag;
  const double* pval;
  const int* well_map;  // well entries -> factor entries
  const int* well_row;  // listed rows -> natural rows
  const int* spec_map;
  T* lrec;
  T* brec;
  T* arec;
  double* rd;
  T* well_val;
  T* well_piv;
  T* spec_val;
};
__device__ __forceinline__ void put_tag(double& v, int tag) { v = __longlong_as_double((long long)tag); }
__device__ __forceinline__ void put_tag(float& v, int tag) { v = __int_as_float(tag); }

template <class T>
__global__ void __launch_bounds__(kBlock) k_pencil_pack(const __grid_constant__ PenPack<T> a) {
  const int stride = gridDim.x * blockDim.x, t0 = blockIdx.x * blockDim.x + threadIdx.x;
  for (int row = t0; row < a.n; row += stride) {
    const size_t q = size_t(a.nat[row]);
    const int* st = a.stencil + 7 * size_t(row);
    const bool special = a.special[row] != 0;
    T l[4], b[4], m[8];
    int e[7];
#pragma unroll
    for (int k = 0; k < 7; ++k) e[k] = special ? -1 : st[k];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      l[k] = e[k] >= 0 ? T(a.plu[e[k]]) : T(0);
      b[k] = e[4 + k] >= 0 ? T(a.plu[e[4 + k]]) : T(0);
    }
#pragma unroll
    for (int k = 0; k < 7; ++k) m[k] = e[k] >= 0 ? T(a.pval[e[k]]) : T(0);
    put_tag(l[3], special ? 1 : 0);
    put_tag(m[7], special ? 1 : 0);
    const T piv = T(a.pdiag[row]);
    const T d = fabs(double(piv)) > kEpsP ? piv : T(1);
    b[3] = d;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const size_t at = sizeof(T) == 8 ? size_t(a.rec_at[row]) + (k < 2 ? k : a.rec_half[row] + k - 2) : 4 * q + k;
      a.lrec[at] = l[k];
      a.brec[at] = b[k];
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) a.arec[8 * q + k] = m[k];
    a.rd[q] = special ? __hiloint2double(int(kPenSpecial), 0) : pen_recip(d);
  }
  for (int e = t0; e < a.nwe; e += stride) a.well_val[e] = T(a.plu[a.well_map[e]]);
  for (int e = t0; e < a.nse; e += stride) a.spec_val[e] = T(a.pval[a.spec_map[e]]);
  for (int e = t0; e < a.nspec; e += stride) {
    const T piv = T(a.pdiag[a.well_row[e]]);
    a.well_piv[e] = fabs(double(piv)) > kEpsP ? piv : T(1);
  }
}

int log2_of(int v) {
  int k = 0;
  while ((1 << (k + 1)) <= v) ++k;
  return k;
}

template <class T>
const void* pen_fn(bool batch) {
  return batch ? (const void*)k_bicgstab_pencil_batch<T> : (const void*)k_bicgstab_pencil<T>;
}

cudaLaunchConfig_t pen_config(int cs, int clusters, size_t smem, cudaStream_t stream, cudaLaunchAttribute* at) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cs * clusters);
  cfg.blockDim = dim3(kPenThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cs;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

int column_owner(int j, int cs, int ny) {
  int b = 0;
  while (pen_first_col(b + 1, cs, ny) <= j) ++b;
  return b;
}

// Shared memory of a solve on cs CTAs (the largest CTA's).
template <class T>
size_t pen_smem_bytes(const Ctx& c, int cs, int chunk, int nvw) {
  size_t most = 0;
  const int cols = (c.ny + cs - 1) / cs;
  std::vector<int> wells(cs, 0), entries(cs, 0);
  for (const PencilPlan::Listed& r : c.pen.listed) {
    const int b = column_owner(r.j, cs, c.ny);
    wells[b]++;
    entries[b] += r.entries;
  }
  for (int b = 0; b < cs; ++b)
    most = std::max(most, pen_layout<T>(c.nx, c.nz, cols, cs, chunk, nvw, wells[b], entries[b]).total);
  return most;
}

// Rows of the step-order layout, in slots.
int pen_cta_slots(const Ctx& c, int cols) {
  // whole chunks of any size
  return (pen_rounded(pen_steps(c.nx, cols, c.nz), kPenChunk) + 2 * kPenGuard) * pen_stride(cols * c.nz);
}
long long pen_slots(const Ctx& c, int cs) {
  long long m = 0;
  for (int b = 0; b < cs; ++b)
    m += pen_cta_slots(c, pen_first_col(b + 1, cs, c.ny) - pen_first_col(b, cs, c.ny));
  return m;
}

// Whether the solve can run on cs CTAs: lines per CTA, fill within a CTA's columns, shared memory, a
// launchable cluster.  Raises the kernels' limits as a side effect.
template <class T>
bool pen_cs_fits(Ctx& c, int cs) {
  if (cs > c.ny) return false;
  const int cols = (c.ny + cs - 1) / cs;
  if ((long long)cols * c.nz > 2 * kPenLineThreads || (long long)(cols + 1) * c.nz >= 0x7ff0) return false;
  for (const auto& pr : c.pen.fill_cols)  // columns that must share a CTA
    if (column_owner(pr.first, cs, c.ny) != column_owner(pr.second, cs, c.ny)) return false;
  int optin = 0;
  RF_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c.device));
  // step order's padding: a deck much shorter along x than across would hold mostly zeros
  if (pen_slots(c, cs) > 4 * (long long)c.n + 16384) return false;
  // 512: the longest DotOrder (16 blocks of 32 warps)
  int chunk = kPenChunk;
  while (chunk > 2 && pen_smem_bytes<T>(c, cs, chunk, 512) + 2048 > size_t(optin)) chunk /= 2;
  const size_t bytes = pen_smem_bytes<T>(c, cs, chunk, 512);
  if (bytes + 2048 > size_t(optin)) return false;
  c.pen.chunk[sizeof(T) == 4 ? 1 : 0][log2_of(cs)] = chunk;
  for (int batch = 0; batch < 2; ++batch) {
    const void* fn = pen_fn<T>(batch != 0);
    raise_dynamic_smem(fn, bytes);
    if (cs > 8) RF_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = pen_config(cs, 1, bytes, nullptr, at);
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg) != cudaSuccess || clusters < 1) {
      cudaGetLastError();
      return false;
    }
  }
  return true;
}

// The most listed rows on one chain of a forward sweep's steps, through the CTAs: a step comes after the
// CTA's step before and the step that sends it the neighbour's column.
int pen_listed_path(const Ctx& c, int cs) {
  std::vector<int> before, path;
  int cols_before = 0;
  for (int b = 0; b < cs; ++b) {
    const int first = pen_first_col(b, cs, c.ny), cols = pen_first_col(b + 1, cs, c.ny) - first;
    path.assign(pen_steps(c.nx, cols, c.nz), 0);
    for (const PencilPlan::Listed& r : c.pen.listed)
      if (r.j >= first && r.j < first + cols) path[r.ik + r.j - first]++;
    for (int m = 0; m < int(path.size()); ++m) {
      int at = m > 0 ? path[m - 1] : 0;
      if (b > 0) at = std::max(at, before[std::min(m + cols_before, int(before.size()) - 1)]);
      path[m] += at;
    }
    before.swap(path);
    cols_before = cols;
  }
  return before.back();
}

// Whether the level-order kernel is the faster one for the deck's wells.  A step's listed rows are solved
// one after another, 1.6 us each per iteration where they lie on one chain of steps; the level-order
// kernel spreads a level's rows over its threads and takes 2.6-4.3 us per level and iteration, the solve
// along lines 1.0-1.8 us besides the listed rows.  us per iteration along lines / in level order, wells through
// all layers (FP64; FP32 alike): 10x10x5 with 2 / 8 / 23 wells (10 / 38 / 97 rows on a chain, 23 levels)
// 54 / 64, 94 / 76, 179 / 87; 20x20x5 with 8 / 23 / 58 (30 / 65 / 162, 43) 98 / 143, 149 / 154, 293 / 167;
// 16x64x16 with 8 / 16 / 24 (90 / 163 / 229, 94) 261 / 367, 385 / 383, 494 / 399; 64x64x8 with 112 (223, 134)
// 476 / 579.  The cluster kernels are slower than it throughout (36,000 to 80,000 cells, chains of up to
// 3.4 rows per level: 1.9-3.8 times).
bool pen_crowded(const Ctx& c, int cs) {
  if (!level_automatic(c)) return false;
  return 10 * pen_listed_path(c, cs) > 17 * c.levels.n_levels - 130;
}

// CTAs per solve: the fewest whose columns are one warp's lines (a warp's barrier is 15 cycles, 13
// warps' 45, and a step's rows come from L2 over more SMs; each hand-over to the next CTA costs some
// 100 cycles of a step).  Thousand cycles per iteration on 1 / 4 / 8 / 16 CTAs: 21x20x5 211 / 173 /
// 181 / 202, 40x31x5 267 / 203 / 197 / 221, 45x61x7 789 / 429 / 388 / 381, 60x60x20 - / 1067 / 764 /
// 618.  An ensemble's variants share the chip: at most 8 CTAs each for up to 32 variants, 4 beyond
// (a report step of 16 variants on 4 / 8 / 16 CTAs: 407 / 374 / 493 ms, of 32: 1006 / 962 / 1260, of
// 64: 1361 / 1479 / 2204; fewer CTAs, and more variants, were not timed).  A size that
// rf_set_cluster_size asked for is taken where the deck fits it.
int pencil_want(Ctx& c) {
  PencilPlan& P = c.pen;
  const int f = c.precision == 1 ? 1 : 0;
  const int most = c.ensemble == 0 ? 16 : c.ensemble <= 32 ? 8 : 4;
  int want = 1;
  while (want < most && c.nz * ((c.ny + want - 1) / want) > 32) want *= 2;
  if (c.cluster_fixed > 0) want = c.cluster_fixed;
  auto fits = [&](int k) {
    int& v = P.fits[f][k];
    if (v < 0) v = (f == 1 ? pen_cs_fits<float>(c, 1 << k) : pen_cs_fits<double>(c, 1 << k)) ? 1 : 0;
    return v > 0;
  };
  const int k0 = log2_of(want);
  int k = k0;
  while (k >= 0 && !fits(k)) --k;
  if (k < 0) {
    k = k0 + 1;
    while (k < 5 && !fits(k)) ++k;
  }
  return k < 5 && !pen_crowded(c, 1 << k) ? 1 << k : 0;
}

template <class V, class H>
void upload_to(V& b, const H& h) {
  b.free();
  b.alloc(h.size());
  if (!h.empty()) RF_CUDA(cudaMemcpy(b.p, h.data(), sizeof(h[0]) * h.size(), cudaMemcpyHostToDevice));
}

// The step-order layout for P.cs CTAs.
void layout_for(Ctx& c, int cs) {
  PencilPlan& P = c.pen;
  const int n = c.n, nx = c.nx, ny = c.ny, nz = c.nz;
  std::vector<int> cta(cs + 1, 0), first(cs), cols(cs);
  for (int b = 0; b < cs; ++b) {
    first[b] = pen_first_col(b, cs, ny);
    cols[b] = pen_first_col(b + 1, cs, ny) - first[b];
    cta[b + 1] = cta[b] + pen_cta_slots(c, cols[b]);  // n < 2^26: offsets of four values per slot stay below 2^31
  }
  std::vector<int> owner(ny);
  for (int j = 0; j < ny; ++j) owner[j] = column_owner(j, cs, ny);
  std::vector<int> nat(n), rec_at(n), rec_half(n);
  auto line_of = [&](int r) { return (r / (nx * ny)) * cols[owner[(r / nx) % ny]] + (r / nx) % ny - first[owner[(r / nx) % ny]]; };
  auto step_of = [&](int r) { return r % nx + (r / nx) % ny - first[owner[(r / nx) % ny]] + r / (nx * ny); };
  for (int r = 0; r < n; ++r) {
    const int b = owner[(r / nx) % ny];
    const int stride = pen_stride(cols[b] * nz), row = cta[b] + (kPenGuard + step_of(r)) * stride;
    nat[r] = row + line_of(r);
    rec_at[r] = 4 * row + 2 * line_of(r);
    rec_half[r] = 2 * stride;
  }
  std::vector<int> spec_slot, spec_col;
  for (int r : P.h_spec_row) spec_slot.push_back(nat[r]);
  for (int r : P.h_spec_col_row) spec_col.push_back(nat[r]);
  // the listed rows by CTA and step
  std::vector<int> ord(P.h_spec_row);
  std::stable_sort(ord.begin(), ord.end(), [&](int x, int y) {
    const int bx = owner[(x / nx) % ny], by = owner[(y / nx) % ny];
    return bx != by ? bx < by : step_of(x) < step_of(y);
  });
  const int ns = int(ord.size());
  std::vector<int> well_cta(cs + 1, 0), slot(ns), ptr(2 * (size_t(ns) + 1)), map, number(n, -1);
  std::vector<int2> at(ns);
  std::vector<unsigned short> code;
  for (int e = 0; e < ns; ++e) {
    const int b = owner[(ord[e] / nx) % ny];
    well_cta[b + 1]++;
    at[e] = make_int2(step_of(ord[e]), line_of(ord[e]));
    slot[e] = nat[ord[e]];
  }
  for (int b = 0; b < cs; ++b) well_cta[b + 1] += well_cta[b];
  for (int e = 0; e < ns; ++e) number[ord[e]] = e - well_cta[owner[(ord[e] / nx) % ny]];
  for (int d = 0; d < 2; ++d) {
    ptr[d * (ns + 1)] = int(map.size());
    for (int e = 0; e < ns; ++e) {
      const int r = ord[e], b = owner[(r / nx) % ny], jc = cols[b], line = line_of(r), k = r / (nx * ny);
      const int* st = &c.h_stencil[7 * size_t(r)];
      const int e0 = d == 0 ? c.h_row_ptr[r] : c.h_diag[r] + 1, e1 = d == 0 ? c.h_diag[r] : c.h_row_ptr[r + 1];
      const int sg = d == 0 ? -1 : 1, j = (r / nx) % ny - first[b];
      for (int q = e0; q < e1; ++q) {
        int cd;
        if (q == st[d == 0 ? kZm : kZp])
          cd = line + sg * jc;
        else if (q == st[d == 0 ? kYm : kYp])
          cd = (d == 0 ? j > 0 : j < jc - 1) ? line + sg : pen_stride(jc * nz) + k;
        else if (q == st[d == 0 ? kXm : kXp])
          cd = line;
        else
          cd = 0x8000 | number[c.h_col[q]];
        code.push_back(static_cast<unsigned short>(cd));
        map.push_back(q);
      }
      ptr[d * (ns + 1) + e + 1] = int(map.size());
    }
  }
  P.cs = cs;
  P.slots = cta[cs];
  P.n_well_entries = int(map.size());
  upload_to(P.d_cta, cta);
  upload_to(P.d_nat, nat);
  upload_to(P.d_rec_at, rec_at);
  upload_to(P.d_rec_half, rec_half);
  P.h_nat = nat;
  P.dots_key.clear();
  upload_to(P.d_spec_slot, spec_slot);
  upload_to(P.d_spec_col, spec_col);
  upload_to(P.d_well_cta, well_cta);
  upload_to(P.d_well_at, at);
  upload_to(P.d_well_slot, slot);
  upload_to(P.d_well_ptr, ptr);
  upload_to(P.d_well_row, ord);
  upload_to(P.d_well_map, map);
  upload_to(P.d_well_code, code);
  const size_t m = size_t(P.slots);
  auto zeros = [](auto& b, size_t count) {
    b.free();
    b.alloc(count);
    RF_CUDA(cudaMemset(b.p, 0, sizeof(*b.p) * count));
  };
  zeros(P.d_well_val, map.size() + 1);
  zeros(P.d_well_piv, size_t(ns) + 1);
  zeros(P.d_lrec, 4 * m);
  zeros(P.d_brec, 4 * m);
  zeros(P.d_arec, 8 * m);
  zeros(P.d_rd, m);
  zeros(P.d_work, 10 * sizeof(double) * m);
  RF_CUDA(cudaDeviceSynchronize());
  P.packed = P.typed = -1;
}

// The slots of the dot products' elements, virtual warp by virtual warp, for the order the solve's
// dot products take (rebuilt when the kernel it stands in for changes).
void dot_lists(Ctx& c, const PencilDots& d) {
  PencilPlan& P = c.pen;
  const std::vector<int> key{d.kind, d.threads, d.blocks, d.slice};  // empty after a new layout
  if (P.dots_key == key) return;
  const int n = c.n, vblocks = d.kind == 0 ? 1 : d.blocks, vwpb = d.threads / 32, nvw = vblocks * vwpb;
  std::vector<int> ptr;
  constexpr int kPad = 16;  // pen_dots reads up to 2 U chunks past a virtual warp's last
  auto finish = [&](int which, const std::vector<std::vector<int>>& lanes) {
    // lanes[v]: chunks of 32 slots
    std::vector<int> list;
    for (int v = 0; v < nvw; ++v) {
      ptr.push_back(int(list.size() / 32));
      list.insert(list.end(), lanes[v].begin(), lanes[v].end());
    }
    ptr.push_back(int(list.size() / 32));
    list.insert(list.end(), size_t(32) * kPad, -1);
    upload_to(P.d_list[which], list);
  };
  std::vector<std::vector<int>> lanes(nvw);
  if (d.kind != 0) {
    for (int v = 0; v < nvw; ++v) {
      const int b = v / vwpb, w = v % vwpb;
      const int first = (d.kind == 1 ? b * d.slice : b * d.threads) + 32 * w;
      const int end = d.kind == 1 ? std::min(n, (b + 1) * d.slice) : n;
      const int step = d.kind == 1 ? d.threads : d.blocks * d.threads;
      for (int e = first; e < end; e += step)
        for (int l = 0; l < 32; ++l) lanes[v].push_back(e + l < end ? P.h_nat[e + l] : -1);
    }
    finish(0, lanes);
    ptr.resize(3 * (size_t(nvw) + 1));
    for (int k = 1; k < 3; ++k) std::copy(ptr.begin(), ptr.begin() + nvw + 1, ptr.begin() + k * (nvw + 1));
  } else {
    const std::vector<int>& rows = c.levels.h_rows;
    const std::vector<int>& lp = c.levels.h_ptr;
    std::vector<char> is_long(n, 0);
    std::vector<int> longs;
    for (int q = 0; q < n; ++q)
      if (c.h_row_ptr[rows[q] + 1] - c.h_row_ptr[rows[q]] > 7) {
        is_long[q] = 1;
        longs.push_back(P.h_nat[rows[q]]);
      }
    for (int v = 0; v < nvw; ++v)
      for (int e = 32 * v; e < n; e += d.threads)
        for (int l = 0; l < 32; ++l) lanes[v].push_back(e + l < n ? P.h_nat[rows[e + l]] : -1);
    finish(0, lanes);
    for (int v = 0; v < nvw; ++v) {
      size_t at = 0;
      for (int e = 32 * v; e < n; e += d.threads)
        for (int l = 0; l < 32; ++l, ++at)
          if (e + l < n && is_long[e + l]) lanes[v][at] = -1;
      for (int e = 32 * v; e < int(longs.size()); e += d.threads)
        for (int l = 0; l < 32; ++l) lanes[v].push_back(e + l < int(longs.size()) ? longs[e + l] : -1);
    }
    finish(1, lanes);
    for (int v = 0; v < nvw; ++v) {
      lanes[v].clear();
      for (int l = 0; l < c.levels.n_levels; ++l)
        for (int e = 32 * v; e < lp[l + 1] - lp[l]; e += d.threads)
          for (int t = 0; t < 32; ++t) lanes[v].push_back(e + t < lp[l + 1] - lp[l] ? P.h_nat[rows[lp[l] + e + t]] : -1);
    }
    finish(2, lanes);
  }
  upload_to(P.d_list_ptr, ptr);
  P.dots_key = key;
}

// The rows outside the 7-point shape; false: the deck keeps the level-list kernels.
bool pencil_structure(Ctx& c) {
  PencilPlan& P = c.pen;
  const int n = c.n, nx = c.nx, ny = c.ny, nz = c.nz, L = c.levels.n_levels;
  // smaller decks take the dense inverse of the pressure matrix
  if (n <= kDenseCoarseCells || n >= (1 << 26) || L != nx + ny + nz - 2) return false;
  const std::vector<int>& lp = c.levels.h_ptr;
  const std::vector<int>& rows = c.levels.h_rows;
  for (int l = 0; l < L; ++l)
    for (int q = lp[l]; q < lp[l + 1]; ++q) {
      const int r = rows[q];
      if (r % nx + (r / nx) % ny + r / (nx * ny) != l) return false;
    }
  // rows with entries outside the stencil, or read by one (the pattern is symmetric)
  std::vector<unsigned char> special(n, 0);
  P.fill_cols.clear();
  for (int r = 0; r < n; ++r) {
    const int* st = &c.h_stencil[7 * size_t(r)];
    for (int e = c.h_row_ptr[r]; e < c.h_row_ptr[r + 1]; ++e) {
      bool in = false;
      for (int k = 0; k < 7; ++k) in = in || st[k] == e;
      if (in) continue;
      special[r] = special[c.h_col[e]] = 1;
      P.fill_cols.insert({(r / nx) % ny, (c.h_col[e] / nx) % ny});
    }
  }
  P.h_spec_row.clear();
  P.h_spec_col_row.clear();
  P.listed.clear();
  std::vector<int> spec_ptr{0}, spec_map;
  for (int r = 0; r < n; ++r) {
    if (!special[r]) continue;
    P.h_spec_row.push_back(r);
    P.listed.push_back({(r / nx) % ny, r % nx + r / (nx * ny), c.h_row_ptr[r + 1] - c.h_row_ptr[r] - 1});
    for (int e = c.h_row_ptr[r]; e < c.h_row_ptr[r + 1]; ++e) {
      P.h_spec_col_row.push_back(c.h_col[e]);
      spec_map.push_back(e);
    }
    spec_ptr.push_back(int(spec_map.size()));
  }
  if (P.h_spec_row.size() >= 0x7fff) return false;
  P.n_spec_entries = int(spec_map.size());
  upload_to(P.d_special, special);
  upload_to(P.d_spec_ptr, spec_ptr);
  upload_to(P.d_spec_map, spec_map);
  P.d_spec_val.free();
  P.d_spec_val.alloc(spec_map.size());
  for (int k = 0; k < 5; ++k) {
    P.fits[0][k] = P.fits[1][k] = -1;
  }
  return true;
}

}  // namespace

// Host or device memory that cannot be had, or any CUDA error, leaves the deck without the plan: the
// solves keep the level-list kernels, and what failed for good shows in the calls after it.
void build_pencil_plan(Ctx& c) noexcept {
  PencilPlan& P = c.pen;
  P.built = 0;
  P.cs = 0;
  // RESSIM_LOST_MESSAGE=m (read when a context is set up) makes every receiving CTA wait, in the forward
  // sweeps, for more than its m-th message holds, and shortens the limit: the tests' wait that runs out
  const char* lost = std::getenv("RESSIM_LOST_MESSAGE");
  P.lost_message = lost ? std::atoi(lost) : -1;
  try {
    P.built = pencil_structure(c) ? 1 : 0;
  } catch (const std::exception&) {
    cudaGetLastError();
    free_pencil_plan(c);
  }
  pencil_replan(c);
}

// The layout for the CTAs the context's solves run on now (its precision, or joining an ensemble,
// changes them).  Called from a destructor too.
void pencil_replan(Ctx& c) noexcept {
  if (!c.pen.built) return;
  try {
    const int cs = pencil_want(c);
    if (cs > 0 && cs != c.pen.cs) layout_for(c, cs);
    c.pen.cs = cs;
    if (cs > 0) dot_lists(c, pressure_dots(c));
  } catch (const std::exception&) {
    cudaGetLastError();
    free_pencil_plan(c);
  }
}

void free_pencil_plan(Ctx& c) {
  PencilPlan& P = c.pen;
  for (auto* b : {&P.d_cta, &P.d_nat, &P.d_rec_at, &P.d_rec_half, &P.d_spec_slot, &P.d_spec_ptr, &P.d_spec_col,
                  &P.d_spec_map, &P.d_well_cta, &P.d_well_slot, &P.d_well_ptr, &P.d_well_row, &P.d_well_map,
                  &P.d_list_ptr, &P.d_list[0], &P.d_list[1], &P.d_list[2]})
    b->free();
  P.d_well_at.free();
  P.d_well_code.free();
  for (auto* b : {&P.d_well_val, &P.d_well_piv, &P.d_spec_val, &P.d_lrec, &P.d_brec, &P.d_arec, &P.d_rd}) b->free();
  for (auto* b : {&P.d_special, &P.d_work}) b->free();
  P.built = 0;
  P.cs = 0;
}

bool pencil_active(const Ctx& c) {
  return c.pressure_solver == 0 && c.pen.built && c.pen.cs > 0;
}

void pencil_pack(Ctx& c) {
  PencilPlan& P = c.pen;
  const int f = c.precision == 1 ? 1 : 0;
  // The sweeps rely on zeros in the slots outside the lines, and the buffers hold either value type: what
  // the other one left there would be read as factors and vectors (halves of doubles, some of them
  // NaN).  The solves' vectors keep their zeros from one solve to the next.
  if (P.typed >= 0 && P.typed != f) {
    for (auto* b : {&P.d_lrec, &P.d_brec, &P.d_arec})
      RF_CUDA(cudaMemsetAsync(b->p, 0, sizeof(double) * b->n, c.stream));
    RF_CUDA(cudaMemsetAsync(P.d_work.p, 0, P.d_work.n, c.stream));
  }
  P.typed = f;
  auto go = [&](auto zero) {
    using T = decltype(zero);
    PenPack<T> a;
    a.n = c.n;
    a.nspec = int(P.h_spec_row.size());
    a.nwe = P.n_well_entries;
    a.nse = P.n_spec_entries;
    a.nat = P.d_nat.p;
    a.stencil = c.d_stencil.p;
    a.special = P.d_special.p;
    a.plu = c.d_plu.p;
    a.pdiag = c.d_pdiag.p;
    a.pval = c.d_pval.p;
    a.well_map = P.d_well_map.p;
    a.well_row = P.d_well_row.p;
    a.spec_map = P.d_spec_map.p;
    a.lrec = reinterpret_cast<T*>(P.d_lrec.p);
    a.brec = reinterpret_cast<T*>(P.d_brec.p);
    a.arec = reinterpret_cast<T*>(P.d_arec.p);
    a.rd = P.d_rd.p;
    a.rec_at = P.d_rec_at.p;
    a.rec_half = P.d_rec_half.p;
    a.well_val = reinterpret_cast<T*>(P.d_well_val.p);
    a.well_piv = reinterpret_cast<T*>(P.d_well_piv.p);
    a.spec_val = reinterpret_cast<T*>(P.d_spec_val.p);
    k_pencil_pack<T><<<std::min(blocks_for(c.n), 4 * c.num_sms), kBlock, 0, c.stream>>>(a);
  };
  if (c.precision == 1)
    go(0.0f);
  else
    go(0.0);
  c.launches++;
  P.packed = f;
}

static_assert(sizeof(PenArgs<double>) <= kBatchArgBytes, "batched launch arguments must fit a batch item");

bool launch_pencil_batch(int type, const BatchItem* const* items, int count, cudaStream_t stream) {
  const int cs = 1 << (type / 2 - 1);
  auto go = [&](auto zero) {
    using T = decltype(zero);
    PenBatch<T> b;
    b.count = count;
    size_t smem = 0;
    for (int i = 0; i < count; ++i) {
      std::memcpy(&b.item[i], items[i]->args, sizeof(PenArgs<T>));
      smem = std::max(smem, items[i]->smem);
    }
    void* args[] = {&b};
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = pen_config(cs, count, smem, stream, at);
    return cudaLaunchKernelExC(&cfg, pen_fn<T>(true), args) == cudaSuccess;
  };
  return type % 2 ? go(0.0f) : go(0.0);
}

void launch_bicgstab_pencil(Ctx& c, const double* rhs, double* x) {
  PencilPlan& P = c.pen;
  const PencilDots dots = pressure_dots(c);
  const int f = c.precision == 1 ? 1 : 0, cs = P.cs;
  if (P.packed != f) throw CudaError("pressure solve along lines: factors not packed for this precision");
  dot_lists(c, dots);
  auto go = [&](auto zero) {
    using T = decltype(zero);
    PenArgs<T> a;
    a.n = c.n;
    a.nx = c.nx;
    a.ny = c.ny;
    a.nz = c.nz;
    a.slots = P.slots;
    a.chunk = P.chunk[f][log2_of(cs)];
    a.dot.vblocks = dots.kind == 0 ? 1 : dots.blocks;
    a.dot.vwpb = dots.threads / 32;
    a.cta = P.d_cta.p;
    a.nat = P.d_nat.p;
    a.list_ptr = P.d_list_ptr.p;
    for (int k = 0; k < 3; ++k) a.list[k] = dots.kind == 0 ? P.d_list[k].p : P.d_list[0].p;
    a.nspec = int(P.h_spec_row.size());
    a.spec_slot = P.d_spec_slot.p;
    a.spec_ptr = P.d_spec_ptr.p;
    a.spec_col = P.d_spec_col.p;
    a.spec_val = reinterpret_cast<const T*>(P.d_spec_val.p);
    a.well_cta = P.d_well_cta.p;
    a.well_at = P.d_well_at.p;
    a.well_slot = P.d_well_slot.p;
    a.well_ptr = P.d_well_ptr.p;
    a.well_code = P.d_well_code.p;
    a.well_val = reinterpret_cast<const T*>(P.d_well_val.p);
    a.well_piv = reinterpret_cast<const T*>(P.d_well_piv.p);
    a.lrec = reinterpret_cast<const T*>(P.d_lrec.p);
    a.brec = reinterpret_cast<const T*>(P.d_brec.p);
    a.arec = reinterpret_cast<const T*>(P.d_arec.p);
    a.rd = P.d_rd.p;
    a.rhs = rhs;
    a.x = x;
    a.work = P.d_work.p;
    a.iter_counter = c.d_bicg_iters;
    a.status = c.d_pipe_status.p;
    a.lost = P.lost_message;
    a.wait_limit = P.lost_message >= 0 ? kPenWaitCycles / 50 : kPenWaitCycles;
    a.max_iters = 50;
    const size_t smem = pen_smem_bytes<T>(c, cs, a.chunk, a.dot.vblocks * a.dot.vwpb);
    if (c.batched && fiber_file(kBatchPressure, f + 2 * (1 + log2_of(cs)), &a, sizeof(a), kPenThreads, smem)) return;
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = pen_config(cs, 1, smem, c.stream, at);
    void* args[] = {&a};
    RF_CUDA(cudaLaunchKernelExC(&cfg, pen_fn<T>(false), args));
    c.launches++;
  };
  if (f == 1)
    go(0.0f);
  else
    go(0.0);
}

}  // namespace rf
