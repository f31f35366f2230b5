"""The black-oil assembly from face terms on decks with partial warps, single layers and long columns
against the oracle (GPU tests), to the tolerances of test_gpu_blackoil."""
import pytest

from ressim_b200 import decks
from test_gpu_blackoil import check, run_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(16, 2, 1), (11, 3, 1), (3, 31, 1), (5, 2, 7), (3, 3, 11)])
def test_blackoil_shapes_match_oracle(dims):
    deck = decks.black_oil_3d(*dims, seed=3, rate_per_perf=3.0)
    _, _, rows = run_pair(deck, 1.0, 1)
    check(rows)
