"""The autotuners time the launches that a flow makes: a tuned context or
ensemble steps no slower than an untuned one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def step_us(*timers):
    """The fastest of eight 50-step bursts of each, taken in turn."""
    best = [np.inf] * len(timers)
    for _ in range(8):
        for i, t in enumerate(timers):
            best[i] = min(best[i], t(50) / 50 * 1e3)
    return best


@pytest.mark.parametrize("n,precision", [((12, 12, 12, 12), "fp64"), ((8, 8, 8, 10), "fp64"),
                                         ((8, 8, 8, 16), "fp32_18"), ((8, 8, 8, 8), "fp32_12")], ids=str)
def test_tuned_contexts_are_not_slower(n, precision):
    from latticeyangmills_b200 import GluonField

    with GluonField(n, precision) as plain, GluonField(n, precision) as tuned:
        for f in (plain, tuned):
            f.init_links("expiah", 0.35, 1)
        U = tuned.download()
        form = tuned.autotune(0.01)
        np.testing.assert_array_equal(tuned.download(), U)
        a, b = step_us(lambda k: plain.time_steps(0.01, k)[0], lambda k: tuned.time_steps(0.01, k)[0])
    print(n, precision, "untuned", a, "tuned", form, b)
    assert b < 1.2 * a  # the clock's and the host's spread; a wrong form costs 1.3 and more


@pytest.mark.parametrize("sizes", [[(6, 6, 6, 6)] * 5, [(8, 8, 8, 8)] * 6 + [(6, 10, 12, 14)] * 4], ids=["one", "two"])
@pytest.mark.parametrize("precision", ["fp64", "fp32_12"])
def test_tuned_ensembles_are_not_slower(sizes, precision):
    from latticeyangmills_b200 import Ensemble

    with Ensemble(sizes, precision) as plain, Ensemble(sizes, precision) as tuned:
        for ens in (plain, tuned):
            for c in range(len(sizes)):
                ens.init_links(c, "expiah", 0.35, 1 + c)
        U = [tuned.download(c) for c in range(len(sizes))]
        tuned.autotune(0.01)
        for c in range(len(sizes)):
            np.testing.assert_array_equal(tuned.download(c), U[c])
        a, b = step_us(lambda k: plain.time_steps(0.01, k), lambda k: tuned.time_steps(0.01, k))
        forms = plain.tuning(), tuned.tuning()
    print(precision, "untuned", forms[0], a, "tuned", forms[1], b)
    assert b < 1.2 * a
