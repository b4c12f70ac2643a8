"""Lattices above the size up to which one launch does a stage and one a
measurement (kSmallSites, csrc/kernels.h), where single contexts, slabs and
blocks run the fused and the two-kernel stage and measure from the links or
through the stored plaquette field: odd extents, extents 1 and 2 and volumes that
leave a partial 32-site group, against the oracle, and every path against
another one that must give the same links."""
import re

import numpy as np
import pytest

from conftest import ROOT, topc_tolerance

pytestmark = pytest.mark.gpu

# 4812 and 6000 sites with extents of 1 and 2; 9009 and 16575 with odd ones
SIZES = [(2, 2, 3, 401), (1, 2, 50, 60), (7, 9, 11, 13), (15, 13, 17, 5)]
PRECISIONS = ["fp64", "fp32_18", "fp32_12"]
SLABS = (16, 8, 8, 10)
BLOCKS = (9, 8, 10, 8)


def small_limit():
    """The line below which none of the kernels meant here runs."""
    src = (ROOT / "latticeyangmills_b200" / "csrc" / "kernels.h").read_text()
    a, b = re.search(r"kSmallSites = (\d+) \* (\d+);", src).groups()
    return int(a) * int(b)


@pytest.fixture(scope="module", autouse=True)
def sizes_are_above_the_line():
    for n in SIZES + [SLABS, BLOCKS]:
        assert np.prod(n) > small_limit()


def context(n, precision, form):
    from latticeyangmills_b200 import GluonField, _native as N

    f = GluonField(n, precision)
    f.set_option(N.OPT_STAGE_FORM, form)
    return f


def assert_rows(got, want, sites, rel):
    scale = 18.0 * sites  # extent-1 planes: sums of rounding only
    np.testing.assert_array_equal(got[:, 0], want[:, 0])
    for g, w in zip(got, want):
        assert abs(g[2] - w[2]) <= rel
        assert abs(g[4] - w[4]) <= rel * max(abs(w[4]), scale)
        assert abs(g[3] - w[3]) <= topc_tolerance(-max(abs(w[4]), scale), rel)


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("n", SIZES, ids=str)
def test_both_forms_match_oracle(oracle, n, precision):
    """Links and rows of three measured steps.  FP64: rounding; FP32: the links'
    own rounding (6e-8) and a few roundings of nine stages' updates."""
    link_tol, rel = (1e-13, 1e-12) if precision == "fp64" else (5e-6, 1e-6)
    U = oracle.gen_expiah(n, 0.35, 17, 0)
    out = []
    for form in (0, 1):
        with context(n, precision, form) as f:
            f.upload(U)
            out.append((f.flow(0.02, 3, 1), f.download()))
    want = oracle.flow(U, n, 0.02, 3, 1)  # flows U in place
    for rows, links in out:
        assert np.abs(links - U).max() < link_tol
        assert_rows(rows, want, oracle.volume(n), rel)
    # two algorithms: equal bits would mean that one kernel ran for both
    assert not np.array_equal(out[0][1], out[1][1])
    assert not np.array_equal(out[0][0], out[1][0])


@pytest.mark.parametrize("n", SIZES, ids=str)
def test_fp64_one_call_equals_single_steps(n):
    """The links that a call passes from step to step as two rows: those of
    calls of one step, which read and leave whole links, bit for bit."""
    out = []
    for calls in ([5], [1] * 5, [2, 3]):
        with context(n, "fp64", 1) as f:
            f.init_links("expiah", 0.35, 3)
            rows = [f.flow(0.02, k, 1) for k in calls]
            out.append((np.concatenate([rows[0][:1]] + [r[1:] for r in rows]), f.download()))
    for rows, links in out[1:]:
        np.testing.assert_array_equal(links, out[0][1])
        np.testing.assert_array_equal(rows, out[0][0])


def test_fp64_uploaded_links_are_read_whole():
    """Links that are unitary to FP32 only: a call's first stage uses their own
    row 2, as a single-step call does."""
    n = (7, 9, 11, 13)
    with context(n, "fp64", 1) as f:
        f.init_links("expiah", 0.35, 7)
        U = f.download().astype(np.float32).astype(np.float64)
        f.upload(U)
        f.flow(0.01, 3, 1)
        three = f.download()
        f.upload(U)
        for _ in range(3):
            f.flow(0.01, 1, 1)
        np.testing.assert_array_equal(f.download(), three)


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("n", SIZES, ids=str)
def test_measured_steps_flow_the_same_links(n, precision):
    """A measured step's stage 0 reads the measurement's plaquette field."""
    out = []
    for every in (1, 3, 0):
        with context(n, precision, 1) as f:
            f.init_links("expiah", 0.35, 5)
            rows = f.flow(0.02, 6, every, reunit_every=2)
            out.append((rows[-1], f.download()))
    for rows, links in out[1:]:
        np.testing.assert_array_equal(links, out[0][1])
        np.testing.assert_array_equal(rows, out[0][0])


def test_fp64_switching_forms_mid_flow_continues_the_flow():
    n, out = (7, 9, 11, 13), []
    for forms in ((0, 1, 0), (0, 0, 0)):
        with context(n, "fp64", 0) as f:
            f.init_links("expiah", 0.4, 9)
            for form, steps in zip(forms, (3, 3, 2)):
                f.set_option(4, form)
                rows = f.flow(0.02, steps, 0)
            out.append((rows, f.download()))
    assert out[0][0][-1, 0] == 8
    assert np.abs(out[0][1] - out[1][1]).max() < 1e-13
    assert not np.array_equal(out[0][1], out[1][1])


def assert_decomposed(got, links, want, want_links, precision):
    # FP64 is bit-identical; the FP32 halo kernels are compiled apart, so the
    # compiler may contract a few multiply-adds differently
    diff = np.abs(links - want_links).max()
    print(precision, "max |dU|", diff)
    assert diff == 0.0 if precision == "fp64" else diff < 1e-5
    rel = 1e-12 if precision == "fp64" else 1e-6
    np.testing.assert_array_equal(got[:, :2], want[:, :2])
    np.testing.assert_allclose(got[:, [2, 4, 5]], want[:, [2, 4, 5]], rtol=rel, atol=1e-15)
    assert np.abs(got[:, 3] - want[:, 3]).max() < rel


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("parts,exchange", [((10,), "fused"), ((4, 3, 3), "fused"), ((1, 2, 7), "fused"),
                                            ((4, 3, 3), "copy")], ids=str)
def test_slabs_match_the_whole_lattice(parts, exchange, form, precision, monkeypatch):
    from latticeyangmills_b200 import GluonField, _native as N, slab_group_flow

    reunit = 3 if precision != "fp64" else 0
    with context(SLABS, precision, form) as f:
        f.init_links("expiah", 0.4, 11)
        want, want_links = f.flow(0.02, 6, 2, reunit_every=reunit), f.download()
    if exchange == "copy":
        monkeypatch.setenv("YMFLOW_SLAB_COPY_EXCHANGE", "1")
    slabs = [GluonField.slab(SLABS, sum(parts[:i]), nt, precision) for i, nt in enumerate(parts)]
    try:
        for s in slabs:
            s.set_option(N.OPT_STAGE_FORM, form)
            s.init_links("expiah", 0.4, 11)
        got = slab_group_flow(slabs, 0.02, 6, 2, reunit_every=reunit)
        links = np.concatenate([s.download() for s in slabs])
    finally:
        for s in slabs:
            s.close()
    assert_decomposed(got, links, want, want_links, precision)


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("form", [0, 1])
def test_connected_slab_matches_the_whole_lattice(form, precision):
    """One rank that exchanges its halos with itself through NCCL: the steps
    and measurements of a slab that flows by itself (ymflow_flow)."""
    from latticeyangmills_b200 import GluonField, _native as N, nccl_unique_id

    reunit = 3 if precision != "fp64" else 0
    with context(SLABS, precision, form) as f:
        f.init_links("expiah", 0.4, 11)
        want, want_links = f.flow(0.02, 6, 2, reunit_every=reunit), f.download()
    with GluonField.slab(SLABS, 0, SLABS[3], precision) as s:
        s.set_option(N.OPT_STAGE_FORM, form)
        s.init_links("expiah", 0.4, 11)
        s.connect(nccl_unique_id(), 0, 1, 0, 0)
        got, links = s.flow(0.02, 6, 2, reunit_every=reunit), s.download()
    assert_decomposed(got, links, want, want_links, precision)


# uneven cuts of (9, 8, 10, 8): z and t; x and t; every direction
CUTS = {"zt": ([9], [8], [4, 6], [3, 5]), "xt": ([4, 5], [8], [10], [1, 7]), "xyzt": ([4, 5], [3, 5], [8, 2], [5, 3])}


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("cut", list(CUTS))
def test_blocks_equal_the_whole_lattice(cut, form, precision):
    from latticeyangmills_b200 import GluonField, _native as N, block_group_flow

    reunit = 2 if precision != "fp64" else 0
    with context(BLOCKS, precision, form) as f:
        f.init_links("expiah", 0.4, 5)
        U = f.download()
        want, want_links = f.flow(0.02, 4, 2, reunit_every=reunit), f.download()
    sizes = CUTS[cut]
    cells = np.ndindex(*[len(s) for s in sizes[::-1]])  # t slowest, x fastest
    boxes = []
    for t, z, y, x in cells:
        at = [sum(s[:i]) for s, i in zip(sizes, (x, y, z, t))]
        boxes.append((at, [s[i] for s, i in zip(sizes, (x, y, z, t))]))
    links = np.empty_like(want_links)
    blocks = [GluonField.block(BLOCKS, at, ext, precision) for at, ext in boxes]
    parts = [tuple(slice(a, a + e) for a, e in zip(at[::-1], ext[::-1])) for at, ext in boxes]
    try:
        for b, part in zip(blocks, parts):
            b.set_option(N.OPT_STAGE_FORM, form)
            b.upload(np.ascontiguousarray(U[part]))
        got = block_group_flow(blocks, [len(s) for s in sizes], 0.02, 4, 2, reunit_every=reunit)
        for b, part in zip(blocks, parts):
            links[part] = b.download()
    finally:
        for b in blocks:
            b.close()
    np.testing.assert_array_equal(links, want_links)
    np.testing.assert_allclose(got[:, [2, 4, 5]], want[:, [2, 4, 5]], rtol=1e-12)
    assert np.abs(got[:, 3] - want[:, 3]).max() < 1e-12
