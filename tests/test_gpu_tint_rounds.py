"""The proper-time integral where its kernel goes through several rounds: more
proper times and more groups than threads, and the fewest of each."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def weights(T):
    """Simpson in ln T, the 3/8 rule on the last three intervals of an odd count."""
    n, du = len(T), np.log(T[1] / T[0])
    w = np.zeros(n)
    m = n - 1 if n % 2 else n - 4
    for k in range(0, m, 2):
        w[k:k + 3] += du / 3 * np.array([1.0, 4.0, 1.0])
    if m < n - 1:
        w[m:] += 3 * du / 8 * np.array([1.0, 3.0, 3.0, 1.0])
    return w * T


@pytest.mark.parametrize("nT", [3, 4, 127, 128, 129, 258])
@pytest.mark.parametrize("ng,nbins", [(2, 2), (130, 13), (128, 4)])
def test_integral_and_jackknife_from_the_integrand(nT, ng, nbins):
    import wltube

    rho, T, F = np.array([0.0, 0.7, 2.0]), np.geomspace(1e-3, 80.0, nT), [0.5, 2.0]
    fld = wltube.field("smooth", fermion=1, nint=4)
    with wltube.Context(0) as ctx:
        h = ctx.upload(O.vloops(61, 2 * ng, 16))
        leff, err, ig = ctx.tint(h, fld, rho, T, F, 2, nbins, want_igrand=True)
    I = np.einsum("k,rjkg->rjg", weights(T), ig)
    per = ng // nbins
    loo = (I.sum(2, keepdims=True) - I.reshape(3, 2, nbins, per).sum(3)) / (ng - per)
    jk = np.sqrt((nbins - 1) / nbins * ((loo - I.mean(2, keepdims=True)) ** 2).sum(2))
    # FP64 sums of at most 258 and 130 terms in another order: 400 * 1.1e-16 of
    # the largest term's sum
    tol = 1e-13 * np.abs(weights(T)[:, None] * ig).sum(2).max()
    np.testing.assert_allclose(leff, I.mean(2) / (4 * np.pi), rtol=0, atol=tol)
    np.testing.assert_allclose(err, jk / (4 * np.pi), rtol=0, atol=10 * tol)
