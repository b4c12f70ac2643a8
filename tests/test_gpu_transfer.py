"""Transfers through the pinned slots: whole and partial chunks, worker shares of
different lengths, repeated and concurrent transfers, bit for bit."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# bytes 576 V: below the direct limit, and fields of 17 to 60 chunks that end
# inside one
SIZES = [(6, 5, 4, 7), (16, 16, 16, 8), (15, 16, 17, 9), (16, 13, 17, 31)]


def random_links(n, seed):
    return np.random.default_rng(seed).standard_normal((n[3], n[2], n[1], n[0], 4, 18))


@pytest.mark.parametrize("n", SIZES, ids=str)
def test_round_trip_is_exact(n):
    from latticeyangmills_b200 import GluonField

    with GluonField(n, "fp64") as f:
        for seed in range(6):  # past the transfers that earn the slots
            U = random_links(n, seed)
            f.upload(U)
            np.testing.assert_array_equal(f.download(), U)


def test_concurrent_round_trips():
    from latticeyangmills_b200 import GluonField

    n, bad = (16, 13, 17, 31), []

    def work(seed):
        with GluonField(n, "fp64") as f:
            for k in range(4):
                U = random_links(n, 10 * seed + k)
                f.upload(U)
                if not np.array_equal(f.download(), U):
                    bad.append(seed)

    threads = [threading.Thread(target=work, args=(s,)) for s in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
