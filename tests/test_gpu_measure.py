"""Observables through the stored plaquette field (contexts on the two-kernel
stage): against the oracle's SuperObs (src/Observables/superobs.cpp:31-128),
and the field a measurement leaves for the next step."""
import numpy as np
import pytest

from conftest import topc_tolerance

pytestmark = pytest.mark.gpu

# extents 1 and 2 (a site is its own neighbour, or both neighbours are one
# site), partial 32-site groups, odd extents, and more 32-site groups than the
# energy and charge kernel has blocks
SIZES = [(1, 2, 3, 4), (2, 2, 2, 2), (32, 1, 1, 1), (3, 5, 7, 2), (5, 4, 6, 11), (8, 8, 8, 8), (32, 32, 16, 8)]


def split_context(n, precision):
    from latticeyangmills_b200 import GluonField, _native as N

    f = GluonField(n, precision)
    f.set_option(N.OPT_STAGE_FORM, N.STAGE_SPLIT)
    return f


@pytest.mark.parametrize("precision", ["fp64", "fp32_18", "fp32_12"])
@pytest.mark.parametrize("n", SIZES, ids=str)
def test_measurement_matches_oracle(oracle, n, precision):
    U = oracle.gen_expiah(n, 0.35, 11, 0)
    plaq, topc, energy = oracle.superobs(U, n)
    with split_context(n, precision) as f:
        f.upload(U)
        o = f.observables()
    if precision == "fp64":
        rel = 1e-12
    else:
        # sums of V random FP32 roundings over sums of V terms: a few ulp for one site, less for more
        rel = 16 * 2.0**-24
    # a lattice whose plaquettes are trivial (extent-1 planes) sums to rounding, not to a relative error
    scale = 18.0 * oracle.volume(n)
    assert abs(o.plaq - plaq) <= rel
    assert abs(o.energy - energy) <= rel * max(abs(energy), scale)
    assert abs(o.topc - topc) <= topc_tolerance(-max(abs(energy), scale), rel)


@pytest.mark.parametrize("precision", ["fp64", "fp32_18", "fp32_12"])
@pytest.mark.parametrize("graph", [1, 0])
def test_measured_steps_flow_the_same_links(precision, graph):
    """A measured step's stage 0 reads the measurement's plaquette field: the
    links are those of a flow measured at its end only, bit for bit."""
    from latticeyangmills_b200 import _native as N

    n, out = (6, 5, 4, 7), []
    for every in (1, 3, 0):
        with split_context(n, precision) as f:
            f.set_option(N.OPT_GRAPH, graph)
            f.init_links("expiah", 0.35, 5)
            rows = f.flow(0.02, 6, every, reunit_every=2)
            out.append((rows[-1], f.download()))
    for rows, links in out[1:]:
        np.testing.assert_array_equal(links, out[0][1])
        np.testing.assert_array_equal(rows, out[0][0])


@pytest.mark.parametrize("precision", ["fp64", "fp32_12"])
@pytest.mark.parametrize("steps", [14, 15, 16, 32])
def test_rows_folded_together(precision, steps):
    """A call folds its rows 16 at a time: each row of a call of 15 (fewer than
    a fold), 16, 17 and 33 rows is that of its step flowed in a call of its own."""
    n = (8, 8, 8, 10)
    with split_context(n, precision) as f, split_context(n, precision) as one:
        f.init_links("expiah", 0.35, 5)
        one.init_links("expiah", 0.35, 5)
        rows = f.flow(0.01, steps, 1)
        assert len(rows) == steps + 1
        for k in range(steps):
            apart = one.flow(0.01, 1, 1)
            np.testing.assert_array_equal(rows[k : k + 2, 2:5], apart[:, 2:5])
