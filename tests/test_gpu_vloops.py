"""The loop generator where its thread layout changes: fewer points than
threads, uneven runs of steps per thread, increments kept in shared memory
(up to 6400 points) and drawn twice (above)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ppl,Nl", [(4, 5), (32, 3), (36, 7), (252, 2), (260, 2), (1028, 3),
                                    (1540, 2), (6400, 2), (6404, 2), (8192, 1)])
def test_generated_loops_match_the_oracle(ppl, Nl):
    import wltube

    with wltube.Context(0) as ctx:
        dev = ctx.download(ctx.generate(2 ** 33 + 5, Nl, ppl, first=11))
    host = O.vloops(2 ** 33 + 5, Nl, ppl, first=11)
    # the same FP64 walk up to its rounding (~1e-14), then one float32 rounding
    # of values below 8: at most one ulp there
    assert np.abs(host).max() < 8.0
    np.testing.assert_allclose(dev, host, rtol=0, atol=2.0 ** -21)
    assert np.mean(dev != host) < 1e-3
