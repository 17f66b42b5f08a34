"""Where the pair kernel leaves out the smooth profile's clamp of |z|^2: the
host's condition l2 + clamp == l2 (float32) makes l2 + max(a, clamp) and l2 + a
the same float for every a >= 0, because rounding is monotone."""
import numpy as np
import pytest


@pytest.mark.parametrize("lam2", [0.2, 0.2500001, 0.4999999, 0.5, 0.75, 1.0, 3.0, 1e4])
def test_clamp_changes_no_bit_where_it_is_left_out(lam2):
    l2, c = np.float32(lam2), np.float32(1e-8)
    a = np.concatenate([[0.0], np.geomspace(1e-45, 1e-8, 4000), np.geomspace(1e-8, 1e6, 4000)])
    a = np.unique(a.astype(np.float32))
    same = (l2 + np.maximum(a, c)) == (l2 + a)
    assert (l2 + c == l2) == (lam2 > 0.25)
    assert np.all(same) or l2 + c != l2
