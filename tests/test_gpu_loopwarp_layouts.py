"""The loop-parallel kernel's two layouts (one and two warps per pair of loop
and instance) give a loop the same sums, for loops shorter than a warp's lanes,
with a ragged last turn, and with an odd last CTA."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prof,fe,nint", [("smooth", 0, 50), ("smooth", 1, 6), ("gaussian", 1, 4),
                                          ("lattice", 1, 4), ("fixflux", 1, 8)])
@pytest.mark.parametrize("ppl", [4, 132])
def test_many_and_single_instances_agree(prof, fe, nint, ppl):
    import wltube

    Nl, n = 1001, 12
    pairs_of_two_warps = 4 * 152 * 4 * 4  # above it, one warp each
    assert Nl <= pairs_of_two_warps < n * Nl
    fld = wltube.field(prof, fermion=fe, nint=nint, lambda2=0.5, tubedist=2.0)
    loops = O.vloops(53, Nl, ppl)
    rng = np.random.default_rng(ppl)
    cx, cy, T = rng.uniform(0, 1, n), rng.uniform(-0.2, 0.2, n), rng.uniform(0.1, 1.0, n)
    with wltube.Context(0) as ctx:
        h = ctx.upload(loops)
        g, _, _ = ctx.eval(h, fld, cx, cy, T, [0.7, 0.2], 1)
        for k in (0, 11):
            g1, _, _ = ctx.eval(h, fld, cx[k], cy[k], T[k], [0.7, 0.2], 1)
            assert np.array_equal(g1[0], g[k])
