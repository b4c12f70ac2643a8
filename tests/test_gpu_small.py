"""Lattices around the size below which one launch does a stage and one a
measurement (4736 sites), at extents and volumes that leave partial 32-site
groups: links and rows against the oracle's flow."""
import numpy as np
import pytest

from conftest import topc_tolerance

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1, 3), (1, 2, 3, 4), (2, 2, 2, 2), (33, 1, 1, 2), (5, 3, 7, 4), (37, 2, 8, 8), (3, 5, 7, 45),
         (8, 8, 2, 38)]


@pytest.mark.parametrize("precision", ["fp64", "fp32_18", "fp32_12"])
@pytest.mark.parametrize("n", SIZES, ids=str)
def test_flow_matches_oracle(oracle, n, precision):
    from latticeyangmills_b200 import GluonField

    U = oracle.gen_expiah(n, 0.35, 17, 0)
    with GluonField(n, precision) as f:
        f.upload(U)
        rows = f.flow(0.02, 3, 1)
        links = f.download()
    want = oracle.flow(U, n, 0.02, 3, 1)  # flows U in place
    # FP64: rounding of 3 steps; FP32: the links' own rounding (6e-8) and a few
    # roundings of 9 stages' updates of size <= eps |Z|
    link_tol, rel = (1e-13, 1e-12) if precision == "fp64" else (5e-6, 1e-6)
    assert np.abs(links - U).max() < link_tol
    np.testing.assert_array_equal(rows[:, 0], want[:, 0])
    scale = 18.0 * oracle.volume(n)  # extent-1 planes: sums of rounding only
    for got, ref in zip(rows, want):
        assert abs(got[2] - ref[2]) <= rel
        assert abs(got[4] - ref[4]) <= rel * max(abs(ref[4]), scale)
        assert abs(got[3] - ref[3]) <= topc_tolerance(-max(abs(ref[4]), scale), rel)
