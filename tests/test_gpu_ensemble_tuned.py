"""Tuned ensembles: a choice tuned with the plane-generator pool is not taken by
an ensemble without it, whose two-kernel stage has nowhere to store."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_a_tuned_two_kernel_form_is_not_shared_without_the_pool():
    import torch

    from latticeyangmills_b200 import Ensemble

    sizes = [(16, 16, 16, 16)] * 8
    sites = sum(np.prod(n) for n in sizes)
    need = int(2 * 4 * sites * 144 + 4 * sites * 64)  # both link pools and the generators
    pool = int(6 * sites * 64)                        # the plane generators

    def flow(ens):
        for c in range(len(sizes)):
            ens.init_links(c, "expiah", 0.35, 5 + c)
        rows = ens.flow(0.01, 3, 1)
        return rows, ens.download(3)

    with Ensemble(sizes, "fp64") as ens:
        ens.set_tuning(0)
        want = flow(ens)
        ens.autotune()
        form = ens.tuning()[0]
    assert form in (1, 3)  # 1.2 x faster than the others at this size
    free, _ = torch.cuda.mem_get_info()
    filler = torch.empty(free - need - pool // 2, dtype=torch.uint8, device="cuda")
    try:
        with Ensemble(sizes, "fp64") as ens:
            assert ens.tuning()[0] == 0
            got = flow(ens)
            ens.autotune()
            assert ens.tuning()[0] not in (1, 3)
    finally:
        del filler
        torch.cuda.empty_cache()
    np.testing.assert_array_equal(got[1], want[1])
    np.testing.assert_allclose(got[0][:, :, [2, 4]], want[0][:, :, [2, 4]], rtol=1e-12)  # measured from the links alone
    with Ensemble(sizes, "fp64") as ens:  # one with the pool takes the choice
        assert ens.tuning()[0] == form
