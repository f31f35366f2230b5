"""Waits of the pressure solve along grid lines that run out (GPU tests).

RESSIM_LOST_MESSAGE=m (read when a context is set up) makes every CTA of a solve that receives a
neighbour's values wait for more than message m holds, with a limit of some 20 ms.  The wait gives up, the
kernel ends by itself with a status, the step returns an error, and the device goes on serving other
contexts.  The messages are the first, one in the middle and the last of a sweep, on two CTAs and on
more, in both value types, and in a batched launch.
"""
import time

import numpy as np
import pytest

from ressim_b200 import Ensemble, ReservoirSimulator, decks
from ressim_b200.simulator import DeviceError

pytestmark = pytest.mark.gpu


def _step(deck, kind, precision):
    g = ReservoirSimulator.from_deck(deck)
    g.set_linear_precision(precision)
    g.set_pressure_solver(kind)
    try:
        g.step(0.5)
        return g.state()
    finally:
        g.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("dims", [(40, 8, 5), (45, 31, 7)])
@pytest.mark.parametrize("where", [0.0, 0.5, 1.0])
def test_a_wait_that_runs_out_is_an_error(dims, where, precision, monkeypatch):
    deck = decks.waterflood_3d(*dims, seed=4, rate_per_perf=20.0)
    monkeypatch.setenv("RESSIM_LOST_MESSAGE", str(int(where * (dims[0] + dims[2] - 2))))
    t0 = time.perf_counter()
    with pytest.raises(DeviceError, match="gave up"):
        _step(deck, "auto", precision)
    assert time.perf_counter() - t0 < 30.0
    monkeypatch.delenv("RESSIM_LOST_MESSAGE")
    a, b = (_step(deck, kind, precision) for kind in ("auto", "level"))
    assert all(np.array_equal(a[k], b[k]) for k in a)


def test_in_a_batched_launch(monkeypatch):
    members = [decks.ensemble_variant(i) for i in (3, 11)]
    monkeypatch.setenv("RESSIM_LOST_MESSAGE", "5")
    e = Ensemble(members)
    with pytest.raises(DeviceError, match="gave up"):
        e.step(0.5)
    e.close()
    monkeypatch.delenv("RESSIM_LOST_MESSAGE")
    e = Ensemble(members)
    e.step(0.5)
    e.close()
