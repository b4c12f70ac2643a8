"""The ensemble's measurement (every configuration in three launches through
the plane-generator pool) against the oracle, and the links FP64 ensembles pass
from step to step as their first two rows."""
import numpy as np
import pytest

from conftest import topc_tolerance

pytestmark = pytest.mark.gpu

SIZES = [(1, 2, 3, 4), (2, 2, 2, 2), (33, 1, 1, 2), (5, 4, 6, 11), (8, 8, 8, 8), (5, 4, 6, 11), (16, 8, 8, 9)]
MANY = [(2, 3, 2, 2 + c % 5) for c in range(131)]  # more than the launch parameter's list holds


@pytest.mark.parametrize("precision", ["fp64", "fp32_18", "fp32_12"])
@pytest.mark.parametrize("sizes", [SIZES, MANY], ids=["mixed", "many"])
def test_rows_match_oracle(oracle, sizes, precision):
    from latticeyangmills_b200 import Ensemble

    rel = 1e-12 if precision == "fp64" else 16 * 2.0**-24
    with Ensemble(sizes, precision) as ens:
        fields = [oracle.gen_expiah(n, 0.35, 23, c) for c, n in enumerate(sizes)]
        for c, U in enumerate(fields):
            ens.upload(c, U)
        rows = ens.flow(0.01, 0, 0)
    for c, (n, U) in enumerate(zip(sizes, fields)):
        plaq, topc, energy = oracle.superobs(U, n)
        scale = max(abs(energy), 18.0 * oracle.volume(n))
        assert abs(rows[0, c, 2] - plaq) <= rel
        assert abs(rows[0, c, 4] - energy) <= rel * scale
        assert abs(rows[0, c, 3] - topc) <= topc_tolerance(-scale, rel)


@pytest.mark.parametrize("precision", ["fp64", "fp32_12"])
@pytest.mark.parametrize("form", [1, 3])
@pytest.mark.parametrize("sizes", [SIZES, MANY], ids=["mixed", "many"])
def test_one_call_equals_single_steps(sizes, form, precision):
    """Measured or not, in one call (graphs in the middle) or step by step: the
    same links and rows, bit for bit."""
    from latticeyangmills_b200 import Ensemble

    out = []
    for calls, every in (([6], 1), ([6], 4), ([1] * 6, 1)):
        with Ensemble(sizes, precision) as ens:
            ens.set_tuning(form)
            for c in range(len(sizes)):
                ens.init_links(c, "expiah", 0.3, 40 + c)
            for k in calls:
                rows = ens.flow(0.02, k, every)
            out.append((rows[-1], [ens.download(c) for c in range(len(sizes))]))
    for rows, links in out[1:]:
        np.testing.assert_array_equal(rows, out[0][0])
        for a, b in zip(links, out[0][1]):
            np.testing.assert_array_equal(a, b)
