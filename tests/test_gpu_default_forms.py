"""The default stage form of slabs and blocks goes by the whole configuration's
volume (FP32: the two-kernel stage above 8192 sites), whatever the parts' own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# 12,288 sites in parts of 6144 and 14,336 local ones; 8192 sites whose parts
# hold 9216 (all of t) or 5120 and 7168 with their halos
CASES = [((32, 8, 8, 6), (1, 5), 1), ((16, 8, 8, 8), (3, 5), 0), ((16, 8, 8, 8), (8,), 0)]


@pytest.mark.parametrize("precision", ["fp32_18", "fp32_12"])
@pytest.mark.parametrize("kind", ["slabs", "blocks"])
@pytest.mark.parametrize("n,parts,form", CASES, ids=str)
def test_parts_take_the_whole_lattices_form(n, parts, form, kind, precision):
    from latticeyangmills_b200 import GluonField, _native as N, block_group_flow, slab_group_flow

    with GluonField(n, precision) as f:
        assert f.get_option(N.OPT_STAGE_FORM) == form
        f.init_links("expiah", 0.4, 11)
        U = f.download()
        want, want_links = f.flow(0.02, 4, 2), f.download()
    cuts = [(sum(parts[:i]), nt) for i, nt in enumerate(parts)]
    ctxs = []
    try:
        for t0, nt in cuts:
            ctxs.append(GluonField.slab(n, t0, nt, precision) if kind == "slabs" else
                        GluonField.block(n, (0, 0, 0, t0), n[:3] + (nt,), precision))
            assert ctxs[-1].get_option(N.OPT_STAGE_FORM) == form
            ctxs[-1].upload(np.ascontiguousarray(U[t0:t0 + nt]))
        if kind == "slabs":
            got = slab_group_flow(ctxs, 0.02, 4, 2)
        else:
            got = block_group_flow(ctxs, [1, 1, 1, len(parts)], 0.02, 4, 2)
        links = np.concatenate([c.download() for c in ctxs])
    finally:
        for c in ctxs:
            c.close()
    # the halo kernels are compiled apart: equal to FP32 rounding
    assert np.abs(links - want_links).max() < 1e-5
    np.testing.assert_allclose(got[:, [2, 4, 5]], want[:, [2, 4, 5]], rtol=1e-6, atol=1e-15)
