"""The loop-parallel kernel with one and with two warps per (loop, instance):
the choice follows the number of pairs and may not change a loop's sums; EV()'s
fingerprint from the sweep itself equals the one of the separate pass."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prof,fe,nint", [("smooth", 0, 50), ("smooth", 1, 6), ("gaussian", 1, 4),
                                          ("lattice", 1, 4), ("fixflux", 1, 8)])
@pytest.mark.parametrize("Nl,ppl", [(3, 4), (4, 132), (1000, 64)])
def test_one_and_two_warps_per_loop_agree(prof, fe, nint, Nl, ppl):
    import wltube

    fld = wltube.field(prof, fermion=fe, nint=nint, lambda2=0.5, tubedist=2.0)
    loops = O.vloops(51, Nl, ppl)
    rng = np.random.default_rng(Nl)
    cx, cy, T = rng.uniform(0, 1, 12), rng.uniform(-0.2, 0.2, 12), rng.uniform(0.1, 1.0, 12)
    with wltube.Context(0) as ctx:
        h = ctx.upload(loops)
        # 12 x 1000 pairs: one warp each; alone, or with few loops: two
        g, _, _ = ctx.eval(h, fld, cx, cy, T, [0.7, 0.2], 1)
        for k in (0, 11):
            g1, _, _ = ctx.eval(h, fld, cx[k], cy[k], T[k], [0.7, 0.2], 1)
            assert np.array_equal(g1[0], g[k])


def test_EV_fingerprint_hits_and_misses():
    """A repeated EV() of the first group recomputes only when a point changed."""
    import torch

    import wltube

    Nl, ppl = 260, 36
    wltube.legacy_configure("smooth", nint=50)
    loops = torch.tensor(O.vloops(52, Nl, ppl), device="cuda")
    scal = torch.zeros(Nl * 4, device="cuda")
    p = wltube.Wparams()
    p.Nl, p.Nppl, p.F, p.l2, p.fermion, p.ng = Nl, ppl, 1.0, 0.7, 0, 2
    p.worldlines, p.Wsscal_d, p.xcm.x = loops.data_ptr(), scal.data_ptr(), 0.3
    first = np.arange(128)
    a = wltube.EV(1.0, p, first)
    scal.zero_()
    torch.cuda.synchronize()
    assert wltube.EV(1.0, p, first) == a and not scal.any()  # cached: no sweep
    loops[259, 35, 1] += 1e-3                                # the last point of the last loop
    torch.cuda.synchronize()
    assert wltube.EV(1.0, p, first) == a and scal.any()      # another ensemble: swept again
