"""The reduction of partial sums to <W>, mean and standard error where its
thread layout changes: instance counts around the powers of two it gives a CTA,
group counts below, at and above the rounds it sums them in."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 33, 70])
@pytest.mark.parametrize("ng,group", [(1, 24), (7, 8), (64, 2), (257, 1), (600, 3)])
def test_group_mean_and_sem(n, ng, group):
    import torch

    import wltube

    rng = np.random.default_rng(n + ng)
    w = np.cumsum(rng.standard_normal((ng * group, 8, 4)) * 0.5, axis=1)
    w -= w.mean(axis=1, keepdims=True)
    cx, cy = rng.uniform(0, 2, n), rng.uniform(-0.3, 0.3, n)
    T = rng.uniform(0.1, 3.0, n)
    fld = wltube.field("smooth", fermion=1, nint=4)
    with wltube.Context(0) as ctx:
        h = ctx.upload(w.astype(np.float32))
        g, m, s = ctx.eval(h, fld, cx, cy, T, [0.5, 1.0], group)
        # the same group by group: loops of one group alone in an ensemble
        k = ng // 2
        h1 = ctx.upload(w[k * group:(k + 1) * group].astype(np.float32))
        g1, _, s1 = ctx.eval(h1, fld, cx, cy, T, [0.5, 1.0], group)
        # mean and error when no group values are asked for (recomputed or kept)
        dev = [torch.tensor(v, device="cuda") for v in (cx, cy, T)]
        om, os_ = (torch.zeros((n, 2), dtype=torch.float64, device="cuda") for _ in range(2))
        torch.cuda.synchronize()
        ctx.eval_device(h, fld, n, *(d.data_ptr() for d in dev), [0.5, 1.0], group, 0,
                        om.data_ptr(), os_.data_ptr())
        ctx.synchronize()
    assert np.array_equal(g[:, :, k], g1[:, :, 0]) and np.all(s1 == 0.0)
    # at most 600 FP64 terms of size ~1: 600 * 1.1e-16 < 1e-13
    np.testing.assert_allclose(m, g.mean(axis=2), rtol=0, atol=1e-13 * np.abs(g).max())
    ref = g.std(axis=2, ddof=1) / np.sqrt(ng) if ng > 1 else np.zeros_like(m)
    np.testing.assert_allclose(s, ref, rtol=1e-10, atol=1e-13 * np.abs(g).max())
    assert np.array_equal(om.cpu().numpy(), m) and np.array_equal(os_.cpu().numpy(), s)
