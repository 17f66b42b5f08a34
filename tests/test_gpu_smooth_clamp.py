"""The smooth profile's clamp of |z|^2 (1e-8 in the reference's mode) at 4
intervals, where kernels without the clamp exist: widths at which it decides
the result (lambda^2 = 1e-7: <W> off by 0.7 without it), and both sides of
lambda^2 = 0.25, where it stops changing a bit of lambda^2 + |z|^2."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

W_TOL = 1e-5  # of max(|W|, 1e-2 of its terms), the tolerance of every <W> here


@pytest.mark.parametrize("mode", [0, 1])  # the reference's clamps, none
@pytest.mark.parametrize("fe", [0, 1])
@pytest.mark.parametrize("lam2", [1e-7, 0.2499999, 0.25])
def test_clamped_widths_match_the_oracle(lam2, fe, mode):
    import wltube

    n, Nl, ppl = 40, 64, 64
    loops = O.vloops(61, Nl, ppl)
    rt = np.sqrt(np.geomspace(1e-9, 1e-6, n)).astype(np.float32).astype(np.float64)
    cx, T = np.zeros(n), rt * rt
    fld = wltube.field("smooth", fermion=fe, nint=4, lambda2=lam2, mode=mode)
    with wltube.Context(0) as ctx:
        h = ctx.upload(loops)
        g, _, _ = ctx.eval(h, fld, cx, cx, T, [1.0], 16)
        (b, _, _), = ctx.batch_eval([{"handle": h, "field": fld, "cx": cx, "cy": cx, "T": T,
                                      "F": [1.0], "group": 16}])
    ref, S = O.eval_groups(loops, cx, cx, T, [1.0],
                           O.field("smooth", fermion=fe, nint=4, lambda2=lam2, mode=mode),
                           group=16, return_scale=True)
    for w in (g, b):  # b sums its groups of 16 as one chunk, g as two
        assert np.max(np.abs(w - ref) / np.maximum(np.abs(ref), 1e-2 * S)) < W_TOL
