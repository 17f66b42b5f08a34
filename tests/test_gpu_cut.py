"""Single loops and whole chunks give the same bits: wl_eval cuts these launches
into single loops, wl_eval_device, which may run beside others, keeps chunks."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prof,fe", [("smooth", 0), ("smooth", 1), ("step", 0), ("quadratic", 0)])
@pytest.mark.parametrize("n,ppl", [(512, 256), (500, 244)])
def test_blocking_and_asynchronous_calls_agree(prof, fe, n, ppl):
    import torch

    import wltube

    Nl, F = 1024, [0.9, 0.3, 0.1, 0.03]
    fld = wltube.field(prof, fermion=fe, nint=4)
    rng = np.random.default_rng(n)
    rt = np.sqrt(rng.uniform(0.05, 2.0, n)).astype(np.float32).astype(np.float64)
    inst = (rng.uniform(0, 2, n).astype(np.float32).astype(np.float64), np.zeros(n), rt * rt)
    with wltube.Context(0) as ctx:
        h = ctx.upload(O.vloops(54, Nl, ppl))
        g, m, s = ctx.eval(h, fld, *inst, F, 128)
        dev = [torch.tensor(v, device="cuda") for v in inst]
        out = [torch.zeros(v.shape, dtype=torch.float64, device="cuda") for v in (g, m, s)]
        torch.cuda.synchronize()
        ctx.eval_device(h, fld, n, *(d.data_ptr() for d in dev), F, 128,
                        *(o.data_ptr() for o in out))
        ctx.synchronize()
    for a, b in zip((g, m, s), out):
        assert np.isfinite(a).all() and np.array_equal(a, b.cpu().numpy())
