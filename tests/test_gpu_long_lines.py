"""Wells far along a long line of cells in the pressure solve along grid lines (GPU tests).

A well's fill rows are solved in the step of their cell; a line of more than 32,768 cells has steps
beyond the range of 16 bits.  Results equal the replaced kernel's bit for bit: no tolerance.
"""
import numpy as np
import pytest

from ressim_b200 import Deck, ReservoirSimulator, linear_solve_bsr

pytestmark = pytest.mark.gpu


def _system(deck, nx, nz, perforated):
    """A diagonally dominant, unsymmetric system on an nx x 1 x nz grid with the fill of one well."""
    rng = np.random.default_rng(nx)
    n = nx * nz
    rows = []
    for r in range(n):
        i, k = r % nx, r // nx
        near = {r}
        near.update(c for c, there in ((r - nx, k > 0), (r - 1, i > 0), (r + 1, i < nx - 1), (r + nx, k < nz - 1))
                    if there)
        if r in perforated:
            near.update(perforated)
        rows.append(sorted(near))
    ptr = np.concatenate(([0], np.cumsum([len(c) for c in rows])))
    col = np.concatenate(rows)
    row = np.repeat(np.arange(n), np.diff(ptr))
    val = rng.uniform(-0.1, 0.1, (len(col), 3, 3))
    on = row == col
    val[on] += np.einsum("ij,jk->ijk", rng.uniform(5.0, 9.0, (n, 3)), np.eye(3))
    val[~on, 0, 0] = -rng.uniform(0.1, 1.2, int((~on).sum()))
    return ptr, col, val.ravel(), rng.standard_normal(3 * n)


@pytest.mark.parametrize("nx,nz,cells", [(33000, 1, [(120, 0), (121, 0), (32767, 0), (32768, 0), (32900, 0), (32990, 0)]),
                                         (32768, 3, [(32767, 0), (32767, 1), (32767, 2)])])
def test_fill_rows_past_step_32767_equal_replaced_kernel(nx, nz, cells):
    d = Deck(nx, 1, nz, 0.2)
    d.set_initial_pressure(300.0)
    for i, k in cells:
        d.add_well_with_id(i, 0, k, 250.0, 0.1, 0.0, False, "PROD")
    perforated = {k * nx + i for i, k in cells}
    system, out = _system(d, nx, nz, perforated), []
    for kind in ("auto", "cluster"):
        g = ReservoirSimulator.from_deck(d)
        g.set_pressure_solver(kind)
        out.append(linear_solve_bsr(g, *system))
        g.close()
    (x0, r0), (x1, r1) = out
    assert np.all(np.isfinite(x1)) and np.any(x1 != 0.0)
    assert r0.iterations == r1.iterations and r0.converged == r1.converged
    assert np.array_equal(x0, x1)
