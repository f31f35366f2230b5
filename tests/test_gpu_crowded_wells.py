"""Decks whose wells crowd the pressure solve along grid lines (GPU tests).

The rows of a well's fill are solved one after another there, so that decks with many wells for their
size keep the level-order kernel.  The automatic choice is checked on both sides of its line, and
that its results equal both kernels' bit for bit: no tolerance.
"""
import numpy as np
import pytest

from ressim_b200 import ReservoirSimulator, decks

pytestmark = pytest.mark.gpu


def _deck(dims, columns):
    d = decks.waterflood_3d(*dims, seed=4, rate_per_perf=5.0)
    d.wells = []
    for w, (i, j) in enumerate(columns):
        for k in range(dims[2]):
            d.add_well_with_id(i, j, k, 500.0 if w % 2 else 250.0, 0.1, 0.0, bool(w % 2), f"W{w}")
    return d


def _columns(dims, count):
    at = np.random.default_rng(1).permutation(dims[0] * dims[1])[:count]
    return [(int(a) % dims[0], int(a) // dims[0]) for a in at]


@pytest.mark.parametrize("dims,count,kernel", [((10, 10, 5), 2, "lines"), ((10, 10, 5), 30, "level"), ((5, 7, 9), 35, "level"),
                                               ((20, 20, 5), 6, "lines"), ((20, 20, 5), 60, "level"),
                                               ((16, 64, 16), 4, "lines"), ((16, 64, 16), 56, "level"),
                                               ((40, 40, 3), 40, "lines"), ((60, 60, 10), 90, "lines")])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_choice_and_results(dims, count, kernel, precision):
    deck, runs = _deck(dims, _columns(dims, count)), []
    for kind in ("auto", "level" if deck.n_cells <= 32768 else "cluster"):
        g = ReservoirSimulator.from_deck(deck)
        g.set_linear_precision(precision)
        g.set_pressure_solver(kind)
        if kind == "auto":
            assert g.profile()["pressure_kernel"] == kernel
        newton = [g.step(0.25)["newton_iterations"] for _ in range(2)]
        runs.append((newton, g.state()))
        g.close()
    (n0, s0), (n1, s1) = runs
    assert n0 == n1 and all(np.array_equal(s0[k], s1[k]) for k in s0)
