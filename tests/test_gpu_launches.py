"""Kernels that a call reports: a heavy profile's sweep with few units runs as
two (its loops cut at their Kahan blocks), with many as one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_launch_counts():
    import wltube

    n = 40
    cx, cy, T = np.linspace(0, 1, n), np.zeros(n), np.linspace(0.1, 2, n)
    count = {}
    with wltube.Context(0) as ctx:
        few, many = ctx.generate(1, 9, 64), ctx.generate(1, 4912, 64)
        for name, prof, h in (("cut", "fixflux", few), ("whole", "fixflux", many),
                              ("light", "smooth", few), ("lattice", "lattice", few)):
            fld = wltube.field(prof, nint=4, lambda2=0.5, tubedist=2.0)
            ctx.eval(h, fld, cx, cy, T, [0.7], 1)
            count[name] = ctx.last_launches()[0]
    # sweep (two kernels if cut) and reduction; the lattice orders its instances
    assert count == {"cut": 3, "whole": 2, "light": 2, "lattice": 3}
