"""The pressure solve along grid lines against the level-list kernels it stands in for (GPU tests).

Every row of its sweeps takes the same operations in the same order, its divisions are correctly
rounded, and its dot products are summed in the replaced kernel's order, so the results are equal
bit for bit: no tolerance.  The sizes cover one line, one warp of lines and a line more, lines of
two rows per thread, columns that split unevenly over the CTAs, steps short of a whole chunk, wells
whose fill fits a CTA's columns and wells whose fill does not (which keep the level-list kernels).
"""
import numpy as np
import pytest

from ressim_b200 import Deck, Ensemble, ReservoirSimulator, decks, linear_solve_bsr

pytestmark = pytest.mark.gpu


def _replaced(n):
    return "level" if n <= 32768 else "cluster"


def _seven_point(nx, ny, nz, seed):
    """A diagonally dominant, unsymmetric 7-point block system with a full right-hand side."""
    rng = np.random.default_rng(seed)
    n = nx * ny * nz
    ptr, col, val = [0], [], []
    for r in range(n):
        i, j, k = r % nx, (r // nx) % ny, r // (nx * ny)
        near = [(r - nx * ny, k > 0), (r - nx, j > 0), (r - 1, i > 0), (r, True), (r + 1, i < nx - 1),
                (r + nx, j < ny - 1), (r + nx * ny, k < nz - 1)]
        for c, there in near:
            if not there:
                continue
            b = rng.uniform(-1.0, 1.0, (3, 3)) * 0.1
            if c == r:
                b += np.diag(rng.uniform(4.0, 9.0, 3))
            else:
                b[0, 0] = -rng.uniform(0.1, 1.4)
            col.append(c)
            val.append(b)
        ptr.append(len(col))
    return np.array(ptr), np.array(col), np.concatenate([v.ravel() for v in val]), rng.standard_normal(3 * n)


def _deck(nx, ny, nz):
    d = Deck(nx, ny, nz, 0.2)
    d.set_initial_pressure(300.0)
    return d


@pytest.mark.parametrize("threads", [0, 96])
@pytest.mark.parametrize("dims", [(300, 1, 1), (10, 32, 1), (12, 33, 1), (31, 3, 11), (31, 17, 4), (40, 29, 15), (40, 5, 60),
                                  (33, 97, 11)])
def test_linear_solve_equals_replaced_kernel(dims, threads):
    n = int(np.prod(dims))
    ptr, col, val, rhs = _seven_point(*dims, seed=n)
    out = []
    for kind in ("auto", _replaced(n)):
        g = ReservoirSimulator.from_deck(_deck(*dims))
        g.set_pressure_solver(kind, threads)
        out.append(linear_solve_bsr(g, ptr, col, val, rhs))
        g.close()
    (x0, r0), (x1, r1) = out
    assert r0.iterations == r1.iterations and r0.converged == r1.converged
    assert np.array_equal(x0, x1)


@pytest.mark.parametrize("scale", [1e-300, 1e-160, 1e160, 1e300, np.inf])
def test_quotients_outside_the_corrected_range(scale):
    """Scaled systems drive the sweeps' quotients out of the corrected reciprocal's range (the rows are
    then divided), an infinite one through non-finite values."""
    dims = (13, 12, 5)
    ptr, col, val, rhs = _seven_point(*dims, seed=8)
    out = []
    for kind in ("auto", "level"):
        g = ReservoirSimulator.from_deck(_deck(*dims))
        g.set_pressure_solver(kind)
        r = rhs.copy()
        r[4] *= scale
        first = linear_solve_bsr(g, ptr, col, val, r)
        second = linear_solve_bsr(g, ptr, col, val * (scale if np.isfinite(scale) else 1.0), rhs)
        out.append((first, second))
        g.close()
    for (x0, r0), (x1, r1) in zip(*out):
        assert r0.iterations == r1.iterations and r0.converged == r1.converged
        assert np.array_equal(x0, x1, equal_nan=True)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("fluid,dims,dt", [("water", (20, 19, 14), 2.0), ("water", (11, 40, 5), 2.0),
                                           ("oil", (10, 10, 3), 2.0), ("water", (45, 61, 13), 0.5),
                                           ("water", (60, 112, 60), 0.05)])
def test_report_steps_with_wells_equal_replaced_kernel(fluid, dims, dt, precision):
    runs = []
    for kind in ("auto", _replaced(int(np.prod(dims)))):
        d = (decks.black_oil_3d(*dims, seed=4, rate_per_perf=5.0) if fluid == "oil"
             else decks.waterflood_3d(*dims, seed=4, rate_per_perf=20.0, gravity=True))
        g = ReservoirSimulator.from_deck(d)
        g.set_linear_precision(precision)
        g.set_pressure_solver(kind)
        newton = [g.step(dt)["newton_iterations"] for _ in range(2)]
        runs.append((newton, g.state(), g.get_well_bhp().copy()))
        g.close()
    (n0, s0, b0), (n1, s1, b1) = runs
    assert n0 == n1
    assert all(np.array_equal(s0[k], s1[k]) for k in s0) and np.array_equal(b0, b1)


def test_ensemble_equals_single_runs_of_replaced_kernel():
    """Variants in batched launches (fewer CTAs each) give the single decks' results."""
    members = [decks.ensemble_variant(i) for i in (3, 11)]
    e = Ensemble(members)
    e.step(0.5)
    for i, d in enumerate(members):
        g = ReservoirSimulator.from_deck(d)
        g.set_pressure_solver("level")
        g.step(0.5)
        s, t = g.state(), e.state(i)
        assert all(np.array_equal(s[k], t[k]) for k in s)
        g.close()
    e.close()
