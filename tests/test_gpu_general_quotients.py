"""Solves whose backward sweeps meet quotients outside the corrected reciprocal's range (GPU tests).

Such a sweep of the pressure solve along grid lines is repeated with IEEE divisions, and the solve goes
on with them, on every CTA of the cluster.  The systems below reach that with finite results: values
that decay below 1e-250 away from the one source, on one CTA and on several, without wells and with
wells in some of the CTAs only, and a pivot beyond 1e30 whose row the first attempt leaves as a NaN
in the repeated sweep's first rows.  Results equal the level-order kernel's bit for bit: no tolerance.
"""
import numpy as np
import pytest

from ressim_b200 import Deck, ReservoirSimulator, linear_solve_bsr

pytestmark = pytest.mark.gpu


def _pattern(nx, ny, nz):
    n = nx * ny * nz
    r = np.arange(n)
    i, j, k = r % nx, r // nx % ny, r // (nx * ny)
    near = ((k > 0, -nx * ny), (j > 0, -nx), (i > 0, -1), (i >= 0, 0), (i < nx - 1, 1), (j < ny - 1, nx),
            (k < nz - 1, nx * ny))
    ptr = np.concatenate(([0], np.cumsum(sum(there.astype(int) for there, _ in near))))
    row = np.repeat(r, np.diff(ptr))
    col = np.concatenate([[q + off for there, off in near if there[q]] for q in range(n)])
    return ptr, row, col


def _solve_both(dims, ptr, col, val, rhs, precision="fp64", wells=()):
    out = []
    for kind in ("auto", "level"):
        d = Deck(*dims, 0.2)
        d.set_initial_pressure(300.0)
        for n, (i, j) in enumerate(wells):
            for k in range(dims[2]):
                d.add_well_with_id(i, j, k, 250.0, 0.1, 0.0, False, f"PROD{n}")
        g = ReservoirSimulator.from_deck(d)
        g.set_linear_precision(precision)
        g.set_pressure_solver(kind)
        out.append(linear_solve_bsr(g, ptr, col, val.ravel(), rhs))
        g.close()
    (x0, r0), (x1, r1) = out
    assert np.all(np.isfinite(x1)) and np.any(x1 != 0.0)
    assert r0.iterations == r1.iterations and r0.converged == r1.converged
    assert np.array_equal(x0, x1)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("end", [0, -1])
@pytest.mark.parametrize("dims,wells", [((400, 1, 1), ()), ((170, 3, 2), ()), ((150, 20, 4), ()), ((60, 70, 2), ()),
                                        ((110, 4, 5), ((3, 1),)), ((150, 20, 4), ((3, 1),)),
                                        ((150, 20, 4), ((140, 19), (70, 18))), ((90, 33, 6), ((45, 16), (2, 30)))])
def test_values_that_decay_below_the_range(dims, wells, end, precision):
    rng = np.random.default_rng(3)
    ptr, row, col = _pattern(*dims)
    val = np.zeros((len(col), 3, 3))
    on = row == col
    val[on] = np.eye(3) * rng.uniform(4.0, 9.0, (int(on.sum()), 1, 1))
    val[~on, 0, 0] = -rng.uniform(1e-5, 1e-3, int((~on).sum()))
    rhs = np.zeros(3 * int(np.prod(dims)))
    rhs.reshape(-1, 3)[end] = 1.0
    _solve_both(dims, ptr, col, val, rhs, precision, wells)


@pytest.mark.parametrize("dims,cell", [((13, 12, 5), 400), ((13, 12, 5), 403), ((40, 31, 4), 2100), ((350, 1, 1), 200)])
def test_a_pivot_above_the_range(dims, cell):
    """Couplings of 1e18 in both directions between two neighbours along x make the second one's pivot
    about -1e35."""
    rng = np.random.default_rng(5)
    ptr, row, col = _pattern(*dims)
    val = rng.uniform(-0.1, 0.1, (len(col), 3, 3))
    on = row == col
    val[on] += np.eye(3) * rng.uniform(6.0, 9.0, (int(on.sum()), 1, 1))
    val[~on, 0, 0] = -rng.uniform(0.1, 0.9, int((~on).sum()))
    val[(row == cell) & (col == cell + 1), 0, 0] = 1e18
    val[(row == cell + 1) & (col == cell), 0, 0] = 1e18
    _solve_both(dims, ptr, col, val, rng.standard_normal(3 * int(np.prod(dims))))
