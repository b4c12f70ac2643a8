"""FP64 flows pass links from step to step as their first two rows: one call of
n steps gives the links of n calls of one step, which read and leave whole
links, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [1, 0])
@pytest.mark.parametrize("n", [(1, 2, 3, 5), (4, 4, 4, 4), (7, 5, 3, 6), (16, 8, 4, 9)], ids=str)
def test_one_call_equals_single_steps(n, graph):
    from latticeyangmills_b200 import GluonField, _native as N

    steps = 5
    out = []
    for calls in ([steps], [1] * steps, [2, 3]):
        with GluonField(n, "fp64") as f:
            f.set_option(N.OPT_STAGE_FORM, N.STAGE_SPLIT)
            f.set_option(N.OPT_GRAPH, graph)
            f.init_links("expiah", 0.35, 3)
            rows = [f.flow(0.02, k, 1) for k in calls]
            out.append((np.concatenate([rows[0][:1]] + [r[1:] for r in rows]), f.download()))
    for rows, links in out[1:]:
        np.testing.assert_array_equal(links, out[0][1])
        np.testing.assert_array_equal(rows, out[0][0])


def test_uploaded_links_are_read_whole():
    """Links that are unitary to FP32 only: the first stage uses their own row 2,
    as a single-step call does."""
    from latticeyangmills_b200 import GluonField

    n = (4, 6, 4, 4)
    with GluonField(n, "fp64") as f:
        f.init_links("expiah", 0.35, 7)
        U = f.download().astype(np.float32).astype(np.float64)
        f.upload(U)
        np.testing.assert_array_equal(f.download(), U)
        f.flow(0.01, 3, 1)
        three = f.download()
        f.upload(U)
        for _ in range(3):
            f.flow(0.01, 1, 1)
        np.testing.assert_array_equal(f.download(), three)
