"""rf_set_cluster_size reaches the factorisation and the pressure solve along grid lines (GPU tests).

The size changes where the work runs, not its results on a deck whose dot products have the level
order; on a larger deck it fixes their order, as it does for the cluster kernel of that size.  Results
are equal bit for bit: no tolerance.
"""
import numpy as np
import pytest

from ressim_b200 import ReservoirSimulator, decks

pytestmark = pytest.mark.gpu


def _run(deck, ctas, precision, kind="auto", dt=0.5):
    g = ReservoirSimulator.from_deck(deck)
    g.set_linear_precision(precision)
    g.set_pressure_solver(kind)
    used = g.set_cluster_size(ctas)
    p = g.profile()
    newton = g.step(dt)["newton_iterations"]
    out = used, p["pressure_ctas"], p["factor_ctas"], newton, g.state()
    g.close()
    return out


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_sizes_asked_for_are_the_ones_that_run(precision):
    deck = decks.waterflood_3d(45, 31, 7, seed=4, rate_per_perf=20.0)
    auto = _run(deck, 0, precision)
    for ctas in (1, 2, 4, 8, 16):
        used, pressure, factor, newton, state = _run(deck, ctas, precision)
        assert (used, pressure, factor) == (ctas, ctas, ctas)
        assert newton == auto[3] and all(np.array_equal(state[k], auto[4][k]) for k in state)


def test_zero_restores_the_automatic_sizes():
    deck = decks.waterflood_3d(45, 31, 7, seed=4, rate_per_perf=20.0)
    g = ReservoirSimulator.from_deck(deck)
    first = g.profile()
    g.set_cluster_size(2)
    assert g.profile()["pressure_ctas"] == g.profile()["factor_ctas"] == 2
    g.set_cluster_size(0)
    assert [g.profile()[k] for k in ("pressure_ctas", "factor_ctas")] == [first[k] for k in ("pressure_ctas", "factor_ctas")]
    g.close()


@pytest.mark.parametrize("ctas", [4, 16])
def test_larger_deck_equals_the_cluster_kernel_of_that_size(ctas):
    deck = decks.waterflood_3d(45, 61, 13, seed=4, rate_per_perf=20.0)
    lines, cluster = (_run(deck, ctas, "fp64", kind, 0.25) for kind in ("auto", "cluster"))
    assert lines[1] == lines[2] == ctas
    assert lines[3] == cluster[3] and all(np.array_equal(lines[4][k], cluster[4][k]) for k in lines[4])
