"""The profile names the kernels that serve the pressure stage (GPU tests)."""
import pytest

from ressim_b200 import Ensemble, ReservoirSimulator, decks

pytestmark = pytest.mark.gpu


def _backward_well():
    """A well from (9, 0) to (2, 1): the second cell comes after the first in natural order but lies on
    an earlier diagonal, so its level is not i + j + k and the solve along lines does not apply."""
    d = decks.waterflood_3d(23, 19, 3, seed=4, rate_per_perf=5.0)
    for i, j in ((9, 0), (2, 1)):
        d.add_well_with_id(i, j, 1, 250.0, 0.1, 0.0, False, "PROD2")
    return d


@pytest.mark.parametrize("deck,kind,kernel", [
    (lambda: decks.waterflood_3d(12, 10, 3, seed=11, rate_per_perf=20.0), "auto", "lines"),
    (lambda: decks.waterflood_3d(45, 31, 7, seed=11, rate_per_perf=20.0), "auto", "lines"),
    (lambda: decks.waterflood_3d(12, 10, 3, seed=11, rate_per_perf=20.0), "level", "level"),
    (lambda: decks.waterflood_3d(12, 10, 3, seed=11, rate_per_perf=20.0), "cluster", "cluster"),
    (_backward_well, "auto", "level"),
])
def test_kernel_named_is_the_one_that_runs(deck, kind, kernel):
    g = ReservoirSimulator.from_deck(deck())
    g.set_pressure_solver(kind)
    p = g.profile()
    assert p["pressure_kernel"] == kernel
    assert p["level_kernels"] == (kernel == "level")
    assert p["pressure_ctas"] in (1, 2, 4, 8, 16) and p["factor_ctas"] in (1, 2, 4, 8, 16)
    assert kernel != "level" or p["pressure_ctas"] == 1
    g.close()


def test_ensemble_variants_run_along_lines():
    e = Ensemble([decks.ensemble_variant(i) for i in (3, 11)])
    assert [e.profile(i)["pressure_kernel"] for i in range(2)] == ["lines", "lines"]
    e.close()
