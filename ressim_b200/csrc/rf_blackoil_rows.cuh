// rf_blackoil_rows.cuh — one cell's, one perforation's and one well's residual and Jacobian rows
// in the three-phase black-oil mode, as __host__ __device__ functions: the kernels k_terms3,
// k_rows3, k_perfs3 and k_wells3 run them, and a host build runs the same code on the CPU
// against the oracle's assembly.  cell_row3 is the host build's whole row;
// the device evaluates the terms it is made of in one kernel and adds them up in a second one.
// Contributions follow the reference's triplet order
// (fim/assembly_ad.rs:782-983): accumulation, then faces z-, y-, x-, x+, y+, z+, then wells;
// Jacobian entries with |v| <= 1e-14 are dropped before they are added.
#pragma once

#include "rf_blackoil.cuh"

namespace rf {

RF_HD double filt3(double v) { return fabs(v) > 1e-14 ? v : 0.0; }

// The terms a cell's row is made of.  A face's are evaluated once, for both of its cells: the three
// component fluxes (kFaceValues) and their derivatives by the lower-index cell's [p, sw, hc], then
// the higher's (kFaceDerivs); the cell's own are the inventory change and the inventory's
// derivatives.  Device code keeps them in arrays of n cells, [term][cell].
constexpr int kFaceValues = 3, kFaceDerivs = 18, kFaceTerms = kFaceValues + kFaceDerivs;
constexpr int kCellValues = 3, kCellDerivs = 9, kCellTerms = kCellValues + kCellDerivs;

// What the row functions read of the deck and its state.
struct CellFields3 {
  int nx, ny, nz;
  const double *pv, *tx, *ty, *tz, *depth;
  const int* reg;
  const double *p, *sw, *hc, *pp, *psw, *phc, *base_rs;
};
// the DRSDT0 Rs cap of a cell: the simulator's Rs at the substep start
RF_HD double base3(const Fluid& f, const CellFields3& c, int i) { return f.drsdt0 ? c.base_rs[i] : 0.0; }

// The face from cell i to its next one along `dir` (0 x, 1 y, 2 z): transmissibility (0: none), other cell.
RF_HD double face3(const CellFields3& c, int i, int dir, int& hi) {
  const int nxy = c.nx * c.ny, at = dir == 0 ? i % c.nx : dir == 1 ? (i / c.nx) % c.ny : i / nxy;
  hi = i + (dir == 0 ? 1 : dir == 1 ? c.nx : nxy);
  if (at + 1 >= (dir == 0 ? c.nx : dir == 1 ? c.ny : c.nz)) return 0.0;
  return (dir == 0 ? c.tx : dir == 1 ? c.ty : c.tz)[i];
}
RF_HD void face_values3(const Fluid& f, const CellFields3& c, int i, int hi, double trans, double fv[3]) {
  const int nxy = c.nx * c.ny;
  face_flux3<double>(f, trans, c.depth[i / nxy], c.depth[hi / nxy], c.reg[i], c.p[i], c.sw[i], c.hc[i], c.reg[hi],
                     c.p[hi], c.sw[hi], c.hc[hi], fv, base3(f, c, i), base3(f, c, hi));
}
RF_HD void face_derivs3(const Fluid& f, const CellFields3& c, int i, int hi, double trans, double d[kFaceDerivs]) {
  const int nxy = c.nx * c.ny;
  Dual<6> fd[3];
  face_flux3<Dual<6>>(f, trans, c.depth[i / nxy], c.depth[hi / nxy], c.reg[i], dvar<6>(c.p[i], 0), dvar<6>(c.sw[i], 1),
                      dvar<6>(c.hc[i], 2), c.reg[hi], dvar<6>(c.p[hi], 3), dvar<6>(c.sw[hi], 4), dvar<6>(c.hc[hi], 5),
                      fd, base3(f, c, i), base3(f, c, hi));
#pragma unroll
  for (int e = 0; e < 3; ++e)
#pragma unroll
    for (int v = 0; v < 6; ++v) d[6 * e + v] = fd[e].d[v];
}
// accumulation; the previous inventory uses the same (frozen) regime, as the substep's previous
// state and first iterate are the same classified state
RF_HD void cell_values3(const Fluid& f, const CellFields3& c, int i, double r[3]) {
  const double bi = base3(f, c, i);
  double cur[3], prev[3];
  inventory3<double>(f, c.pv[i], c.reg[i], c.p[i], c.sw[i], c.hc[i], bi, cur);
  inventory3<double>(f, c.pv[i], c.reg[i], c.pp[i], c.psw[i], c.phc[i], bi, prev);
#pragma unroll
  for (int e = 0; e < 3; ++e) r[e] = 0.0 + (cur[e] - prev[e]);
}
RF_HD void cell_derivs3(const Fluid& f, const CellFields3& c, int i, double d[kCellDerivs]) {
  Dual<3> cd[3];
  inventory3<Dual<3>>(f, c.pv[i], c.reg[i], dvar<3>(c.p[i], 0), dvar<3>(c.sw[i], 1), dvar<3>(c.hc[i], 2),
                      base3(f, c, i), cd);
#pragma unroll
  for (int e = 0; e < 3; ++e)
#pragma unroll
    for (int v = 0; v < 3; ++v) d[3 * e + v] = filt3(cd[e].d[v]);
}
// A face's part of a cell's residual and diagonal block; UP: the cell is the face's lower one.
// Terms lie `stride` apart.
template <bool UP>
RF_HD void face_add3(const double* t, size_t stride, double dt, double r[3], double diag[9]) {
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    const double fv = t[e * stride];
    r[e] += (UP ? fv : -fv) * dt;
#pragma unroll
    for (int v = 0; v < 3; ++v) {
      const double d = t[(kFaceValues + 6 * e + (UP ? v : 3 + v)) * stride];
      diag[3 * e + v] += filt3((UP ? d : -d) * dt);
    }
  }
}
// Entry k of its block in the column of the face's other cell.
RF_HD double face_off3(const double* t, size_t stride, double dt, bool up, int k) {
  const double d = t[(kFaceValues + 6 * (k / 3) + (up ? 3 : 0) + k % 3) * stride];
  return filt3((up ? d : -d) * dt);
}

// Residual row and Jacobian block row of cell i (accumulation, then the six faces), written into
// res[3i..] and the row's blocks of val (stencil: 7 block positions per row, -1 absent).
RF_HD void cell_row3(const Fluid& f, int nx, int ny, int nz, int i, double dt,
                     const double* __restrict__ pv, const double* __restrict__ tx,
                     const double* __restrict__ ty, const double* __restrict__ tz,
                     const double* __restrict__ depth, const int* __restrict__ reg,
                     const double* __restrict__ p, const double* __restrict__ sw,
                     const double* __restrict__ hc, const double* __restrict__ pp,
                     const double* __restrict__ psw, const double* __restrict__ phc,
                     const int* __restrict__ row_ptr, const int* __restrict__ stencil,
                     double* __restrict__ res, double* __restrict__ val,
                     const double* __restrict__ base_rs) {
  const int nxy = nx * ny;
  for (int k = row_ptr[i]; k < row_ptr[i + 1]; ++k)
#pragma unroll
    for (int e = 0; e < 9; ++e) val[size_t(k) * 9 + e] = 0.0;
  const CellFields3 c{nx, ny, nz, pv, tx, ty, tz, depth, reg, p, sw, hc, pp, psw, phc, base_rs};
  double r[3], diag[9];
  cell_values3(f, c, i, r);
  cell_derivs3(f, c, i, diag);
  const int* st = stencil + size_t(i) * 7;
  const int at[3] = {i % nx, (i / nx) % ny, i / nxy}, step[3] = {1, nx, nxy};
  const int lower[3] = {kXm, kYm, kZm}, upper[3] = {kXp, kYp, kZp};
  auto face = [&](int lo, int dir, bool up) {
    int hi;
    const double t = face3(c, lo, dir, hi);
    if (!(t > 0.0)) return;
    double terms[kFaceTerms];
    face_values3(f, c, lo, hi, t, terms);
    face_derivs3(f, c, lo, hi, t, terms + kFaceValues);
    if (up)
      face_add3<true>(terms, 1, dt, r, diag);
    else
      face_add3<false>(terms, 1, dt, r, diag);
    for (int e = 0; e < 9; ++e) val[size_t(st[up ? upper[dir] : lower[dir]]) * 9 + e] = face_off3(terms, 1, dt, up, e);
  };
  for (int dir = 2; dir >= 0; --dir)
    if (at[dir] > 0) face(i - step[dir], dir, false);
  for (int dir = 0; dir < 3; ++dir) face(i, dir, true);
#pragma unroll
  for (int e = 0; e < 3; ++e) res[3 * i + e] = r[e];
#pragma unroll
  for (int e = 0; e < 9; ++e) val[size_t(st[kDiag]) * 9 + e] = diag[e];
}

// Perforation k: its source terms in the cell's rows and diagonal block, and its connection row.
// `part`: kPerfAll, or one of the four independent evaluations (the device gives each a warp).
constexpr int kPerfAll = -1, kPerfParts = 4;
RF_HD void perf_row3(const Fluid& f, int n_wells, int k, double dt, const int* __restrict__ perf_cell,
                     const int* __restrict__ perf_inj, const int* __restrict__ perf_well,
                     const int* __restrict__ perf_has_wi, const double* __restrict__ perf_wi,
                     const double* __restrict__ perf_head, const int* __restrict__ reg,
                     const double* __restrict__ p, const double* __restrict__ sw, const double* __restrict__ hc,
                     const double* __restrict__ bhp, const double* __restrict__ q, const int* __restrict__ diag_pos,
                     double* __restrict__ res, double* __restrict__ val, double* __restrict__ res_tail,
                     double* __restrict__ jrw, double* __restrict__ jwr_perf, double* __restrict__ jww_perf_bhp,
                     const double* __restrict__ base_rs, int part = kPerfAll) {
  const int c = perf_cell[k], w = perf_well[k], rg = reg[c];
  const double bc = f.drsdt0 ? base_rs[c] : 0.0;
  const bool inj = perf_inj[k] != 0;
  const double pc = p[c], swc = sw[c], hcc = hc[c], b = bhp[w], qk = q[k];
  if (part == kPerfAll || part == 0) {
    double coef[3];
    component_coefficients3<double>(f, inj, rg, pc, swc, hcc, coef, bc);
#pragma unroll
    for (int e = 0; e < 3; ++e) res[3 * c + e] += coef[e] * qk * dt;
  }
  if (part == kPerfAll || part == 1) {
    double* dblk = val + size_t(diag_pos[c]) * 9;
    Dual<4> P = dvar<4>(pc, 0), SW = dvar<4>(swc, 1), HC = dvar<4>(hcc, 2), Q = dvar<4>(qk, 3);
    Dual<4> ca[3];
    component_coefficients3<Dual<4>>(f, inj, rg, P, SW, HC, ca, bc);
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      Dual<4> row = ca[e] * Q;
#pragma unroll
      for (int v = 0; v < 3; ++v) dblk[3 * e + v] += filt3(row.d[v] * dt);
      jrw[3 * k + e] = filt3(row.d[3] * dt);
    }
  }
  const bool wi = perf_has_wi[k] != 0;
  if (part == kPerfAll || part == 2) {
    const double conn = wi ? connection_rate3<double>(f, perf_wi[k], perf_head[k], inj, rg, pc, swc, hcc, b, bc) : 0.0;
    res_tail[n_wells + k] = wi ? 0.0 + (qk - conn) : 0.0;
  }
  if (part == kPerfAll || part == 3) {
    if (wi) {
      Dual<4> ca = connection_rate3<Dual<4>>(f, perf_wi[k], perf_head[k], inj, rg, dvar<4>(pc, 0), dvar<4>(swc, 1),
                                             dvar<4>(hcc, 2), dvar<4>(b, 3), bc);
#pragma unroll
      for (int v = 0; v < 3; ++v) jwr_perf[3 * k + v] = filt3(-ca.d[v]);
      jww_perf_bhp[k] = filt3(-ca.d[3]);
    } else {
#pragma unroll
      for (int v = 0; v < 3; ++v) jwr_perf[3 * k + v] = 0.0;
      jww_perf_bhp[k] = 0.0;
    }
  }
}

// Control row of physical well w.
RF_HD void well_row3(const Fluid& f, int w, const WellControlH& c, const int* __restrict__ well_ptr,
                     const int* __restrict__ well_perfs, const int* __restrict__ perf_cell,
                     const int* __restrict__ reg, const double* __restrict__ p, const double* __restrict__ sw,
                     const double* __restrict__ hc, const double* __restrict__ bhp, const double* __restrict__ q,
                     double* __restrict__ res_tail, double* __restrict__ jwr_ctrl, double* __restrict__ jww_ctrl_q,
                     double* __restrict__ jww_ctrl_bhp, const double* __restrict__ base_rs) {
  const bool inj = c.injector != 0;
  auto base = [&](int cell) { return f.drsdt0 ? base_rs[cell] : 0.0; };
  const double b = bhp[w];
  for (int a = well_ptr[w]; a < well_ptr[w + 1]; ++a) {
    const int k = well_perfs[a];
#pragma unroll
    for (int v = 0; v < 3; ++v) jwr_ctrl[3 * k + v] = 0.0;
    jww_ctrl_q[k] = 0.0;
  }
  if (!c.enabled || !c.rate_controlled) {
    res_tail[w] = 0.0 + (b - c.bhp_target);
    jww_ctrl_bhp[w] = 1.0;
    return;
  }
  if (!c.has_target) {
    res_tail[w] = 0.0;
    jww_ctrl_bhp[w] = 0.0;
    return;
  }
  double actual = 0.0;
  for (int a = well_ptr[w]; a < well_ptr[w + 1]; ++a) {
    const int k = well_perfs[a], cell = perf_cell[k];
    actual = actual + (c.uses_surface_target
                           ? surface_rate3<double>(f, inj, reg[cell], p[cell], sw[cell], hc[cell], q[k], base(cell))
                           : reservoir_rate<double>(inj, q[k]));
  }
  const double bhp_slack = inj ? c.bhp_limit - b : b - c.bhp_limit;
  const double rate_slack = c.target_rate - actual;
  const double bs = fmax(fabs(c.bhp_limit), 1.0), rsc = fmax(fabs(c.target_rate), 1.0);
  res_tail[w] = 0.0 + fischer_burmeister(bhp_slack / bs, rate_slack / rsc);
  double da, db;
  fb_gradient(bhp_slack / bs, rate_slack / rsc, da, db);
  const double dslack = inj ? -1.0 : 1.0;
  jww_ctrl_bhp[w] = filt3(da * dslack / bs);
  const double factor = -db / rsc;
  for (int a = well_ptr[w]; a < well_ptr[w + 1]; ++a) {
    const int k = well_perfs[a], cell = perf_cell[k];
    Dual<4> P = dvar<4>(p[cell], 0), SW = dvar<4>(sw[cell], 1), HC = dvar<4>(hc[cell], 2), Q = dvar<4>(q[k], 3);
    Dual<4> rate = c.uses_surface_target ? surface_rate3<Dual<4>>(f, inj, reg[cell], P, SW, HC, Q, base(cell))
                                         : reservoir_rate<Dual<4>>(inj, Q);
#pragma unroll
    for (int v = 0; v < 3; ++v) jwr_ctrl[3 * k + v] = filt3(factor * rate.d[v]);
    jww_ctrl_q[k] = filt3(factor * rate.d[3]);
  }
}


}  // namespace rf
