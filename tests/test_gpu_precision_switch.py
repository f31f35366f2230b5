"""Changing a live context's precision between report steps (GPU tests).

`rf_set_linear_precision` takes effect at the next linear solve, so a solver that has run in one
value type goes on in the other, in the same buffers.  The pressure solve along grid lines must still
give the results of the kernel it stands in for, bit for bit: no tolerance.  The decks run on one CTA
and on several, with wells, and as an ensemble's batched launches.
"""
import numpy as np
import pytest

from ressim_b200 import Ensemble, ReservoirSimulator, _abi, _lib, decks

pytestmark = pytest.mark.gpu

CODES = {"fp64": _abi.RF_PRECISION_FP64, "mixed": _abi.RF_PRECISION_MIXED}


def _deck(fluid, dims):
    if fluid == "oil":
        return decks.black_oil_3d(*dims, seed=4, rate_per_perf=5.0)
    return decks.waterflood_3d(*dims, seed=4, rate_per_perf=20.0, gravity=True)


@pytest.mark.parametrize("order", [("fp64", "mixed"), ("mixed", "fp64"), ("fp64", "mixed", "fp64", "mixed")])
@pytest.mark.parametrize("fluid,dims,dt", [("oil", (10, 10, 3), 2.0), ("water", (21, 5, 5), 2.0),
                                           ("water", (40, 8, 5), 1.0), ("water", (45, 31, 7), 0.5),
                                           ("water", (45, 61, 13), 0.25)])
def test_steps_after_a_switch_equal_replaced_kernel(fluid, dims, dt, order):
    deck, runs = _deck(fluid, dims), []
    for kind in ("auto", "level" if deck.n_cells <= 32768 else "cluster"):
        g = ReservoirSimulator.from_deck(deck)
        g.set_pressure_solver(kind)
        steps = []
        for mode in order:
            g.set_linear_precision(mode)
            newton = g.step(dt)["newton_iterations"]
            steps.append((newton, g.state(), g.get_well_bhp().copy()))
        runs.append(steps)
        g.close()
    for (n0, s0, b0), (n1, s1, b1) in zip(*runs):
        assert n0 == n1
        assert all(np.array_equal(s0[k], s1[k]) for k in s0) and np.array_equal(b0, b1)


def test_ensemble_switch_equals_single_runs_of_replaced_kernel():
    members = [decks.ensemble_variant(i) for i in (3, 11)]
    e = Ensemble(members)
    for mode in ("fp64", "mixed", "fp64"):
        for c in e._ctx:
            assert _lib.load().rf_set_linear_precision(c, CODES[mode]) == _abi.RF_OK
        e.step(0.5)
    for i, d in enumerate(members):
        g = ReservoirSimulator.from_deck(d)
        g.set_pressure_solver("level")
        for mode in ("fp64", "mixed", "fp64"):
            g.set_linear_precision(mode)
            g.step(0.5)
        s, t = g.state(), e.state(i)
        assert all(np.array_equal(s[k], t[k]) for k in s)
        g.close()
    e.close()
