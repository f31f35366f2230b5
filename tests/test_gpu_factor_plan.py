"""The factorisation from its plan against the searching form (GPU tests).

Every element takes the same operations in the same order, so states, well BHPs and Newton counts
are equal bit for bit: no tolerance.  The decks cover one row per level, levels of more rows than
one pass of the cluster, wells of up to 46 layers (more updated blocks than a warp has lanes),
wells along x and y (fill whose columns are not in level order), neighbouring wells, a well in every
cell of a small deck, the mixed form, and an ensemble's batched launch.
"""
import numpy as np
import pytest

from ressim_b200 import Ensemble, ReservoirSimulator, decks

pytestmark = pytest.mark.gpu


def _horizontal(nx, ny, nz):
    d = decks.waterflood_3d(nx, ny, nz, seed=4, rate_per_perf=5.0)
    d.wells = []
    for i in range(nx):
        d.add_well_with_id(i, 0, 0, 500.0, 0.1, 0.0, True, "INJ1")
    for j in range(ny):
        d.add_well_with_id(nx - 1, ny - 1 - j, nz - 1, 250.0, 0.1, 0.0, False, "PROD")
    for i, j, k in ((1, 2, 0), (2, 2, 1), (3, 3, 1), (3, 4, 0)):  # a well that bends
        d.add_well_with_id(i, j, k, 500.0, 0.1, 0.0, True, "INJ2")
    return d


def _crowded(nx, ny, nz):
    d = decks.waterflood_3d(nx, ny, nz, seed=6, rate_per_perf=2.0)
    d.wells = []
    for j in range(ny):
        for i in range(nx):
            for k in range(nz):
                d.add_well_with_id(i, j, k, 500.0 if (i + j) % 2 else 250.0, 0.1, 0.0, bool((i + j) % 2), f"W{i}-{j}")
    return d


DECKS = {
    "one row per level": lambda: decks.waterflood_1d(700)[0],
    "wells of 46 layers": lambda: decks.waterflood_3d(9, 11, 46, seed=2, rate_per_perf=5.0),
    "wide levels": lambda: decks.waterflood_3d(61, 64, 58, seed=3, rate_per_perf=5.0),
    "horizontal": lambda: _horizontal(23, 19, 3),
    "crowded": lambda: _crowded(5, 7, 9),
    "black oil": lambda: decks.black_oil_3d(11, 13, 8, seed=5, rate_per_perf=5.0),
}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("name", list(DECKS))
def test_plan_equals_searching_form(name, precision, monkeypatch):
    deck, runs = DECKS[name](), []
    for recipes in ("1", "0"):
        monkeypatch.setenv("RESSIM_FACTOR_RECIPES", recipes)
        g = ReservoirSimulator.from_deck(deck)
        g.set_linear_precision(precision)
        newton = g.step(0.25)["newton_iterations"]
        runs.append((g.state(), g.get_well_bhp().copy(), newton))
        g.close()
    (s1, b1, n1), (s0, b0, n0) = runs
    assert n1 == n0
    for k in ("pressure", "sat_water", "sat_gas"):
        assert np.array_equal(s1[k], s0[k]), k
    assert np.array_equal(b1, b0)


def test_batched_plan_equals_searching_form(monkeypatch):
    ds, runs = [decks.ensemble_variant(v) for v in (3, 7, 9)], []
    for recipes in ("1", "0"):
        monkeypatch.setenv("RESSIM_FACTOR_RECIPES", recipes)
        e = Ensemble(ds)
        e.step(1.0)
        runs.append([(e.state(v)["pressure"].copy(), e.state(v)["sat_water"].copy()) for v in range(len(ds))])
        e.close()
    for (p1, s1), (p0, s0) in zip(*runs):
        assert np.array_equal(p1, p0) and np.array_equal(s1, s0)
