"""The sweep's warp units: loop pairs with odd remainders, chunks of 1 to 8
loops, loops shorter and longer than a staged piece, and the choice between
whole chunks and single loops, which may not change a result."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def instances(n, seed, span=2.0):
    rng = np.random.default_rng(seed)
    rt = np.sqrt(rng.uniform(0.05, 2.0, n)).astype(np.float32).astype(np.float64)
    f = lambda v: v.astype(np.float32).astype(np.float64)  # noqa: E731
    return f(rng.uniform(0, span, n)), f(rng.uniform(-0.3, 0.3, n)), rt * rt


@pytest.mark.parametrize("Nl,group,ppl", [(7, 7, 64), (5, 5, 132), (9, 3, 128), (12, 12, 124),
                                          (6, 6, 260), (16, 16, 516), (2, 2, 4)])
@pytest.mark.parametrize("prof,fe,nint,n", [("smooth", 1, 4, 33), ("gaussian", 0, 50, 64),
                                            ("smooth", 1, 6, 40), ("quadratic", 1, 2, 65),
                                            ("gaussian", 1, 14, 32), ("step", 0, 64, 32), ("lattice", 1, 4, 97),
                                            ("periodic", 0, 8, 40)])
def test_remainders_equal_loops_on_their_own(prof, fe, nint, n, Nl, group, ppl):
    """A group is the mean of its loops, each evaluated as an ensemble of its own
    (no neighbour in its pair or chunk), up to the FP64 rounding of at most 16
    terms of size <= 5 max|W|: below 1e-14 of it."""
    import wltube

    fld = wltube.field(prof, fermion=fe, nint=nint, lambda2=0.8, tubedist=3.0)
    loops = O.vloops(41, Nl, ppl)
    cx, cy, T = instances(n, Nl + ppl)
    with wltube.Context(0) as ctx:
        g, _, _ = ctx.eval(ctx.upload(loops), fld, cx, cy, T, [0.7, 0.2], group)
        one = [ctx.eval(ctx.upload(loops[k:k + 1]), fld, cx, cy, T, [0.7, 0.2], 1)[0][:, :, 0]
               for k in range(Nl)]
    w = np.stack(one, axis=2).reshape(n, 2, -1, group)
    assert np.max(np.abs(g - w.mean(axis=3))) < 1e-14 * max(1.0, np.abs(w).max())


@pytest.mark.parametrize("prof,fe,nint,n", [("smooth", 1, 4, 700), ("gaussian", 0, 10, 700)])
def test_single_loops_and_whole_chunks_agree_bit_for_bit(prof, fe, nint, n):
    """wl_eval_device stores these loops one by one; the fixed scratch of
    wl_eval_noalloc holds only chunk sums."""
    import torch

    import wltube

    Nl, ppl, F = 2048, 64, [1.0, 0.3]
    fld = wltube.field(prof, fermion=fe, nint=nint)
    dev = [torch.tensor(v, device="cuda") for v in instances(n, 3)]
    loops = torch.tensor(O.vloops(42, Nl, ppl), device="cuda")
    out = [torch.zeros((n, 2, Nl // 128), dtype=torch.float64, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    with wltube.Context(0) as ctx:
        h = ctx.wrap(loops.data_ptr(), Nl, ppl)
        ctx.eval_device(h, fld, n, *(d.data_ptr() for d in dev), F, 128, out[0].data_ptr())
        ctx.synchronize()
    wltube.eval_noalloc(loops.data_ptr(), Nl, ppl, fld, n, *(d.data_ptr() for d in dev), F, 128,
                        out[1].data_ptr())
    assert torch.isfinite(out[0]).all() and torch.equal(out[0], out[1])


@pytest.mark.parametrize("ppl", [4, 8, 36, 256, 260, 288, 1028])
@pytest.mark.parametrize("prof,fe,ffv", [("periodic", 0, 0), ("periodic", 1, 0),
                                         ("spline", 1, 0), ("fixflux", 1, 0),
                                         ("fixflux", 0, 1)])
def test_heavy_profiles_cut_at_their_blocks(prof, fe, ffv, ppl):
    """wl_eval cuts these loops at their Kahan blocks (few units); among many
    loops (two tiles of 4912) it walks them whole: the same bits."""
    import wltube

    fld = wltube.field(prof, fermion=fe, nint=4, lambda2=0.5, tubedist=1.0, ff_variant=ffv)
    few = O.vloops(43, 9, ppl)
    many = np.concatenate([few, O.vloops(44, 4903, ppl)])
    cx, cy, T = instances(40, ppl)
    with wltube.Context(0) as ctx:
        g, _, _ = ctx.eval(ctx.upload(few), fld, cx, cy, T, [0.7], 1)
        w, _, _ = ctx.eval(ctx.upload(many), fld, cx, cy, T, [0.7], 1)
    assert np.isfinite(g).all() and np.array_equal(g, w[:, :, :9])


def test_a_job_beside_a_large_one_equals_it_alone():
    """Alone the batch stores single loops, beside a job of 40960 units whole
    chunks."""
    import wltube

    with wltube.Context(0) as ctx:
        h, big = ctx.generate(5, 256, 64), ctx.generate(6, 16384, 4)
        jobs = []
        for k, (prof, fe) in enumerate([("smooth", 1), ("lattice", 0), ("gaussian", 1)]):
            cx, cy, T = instances(90, k)
            jobs.append({"handle": h, "cx": cx, "cy": cy, "T": T, "F": [1.0], "group": 128,
                         "field": wltube.field(prof, fermion=fe, nint=4, tubedist=3.0)})
        cx, cy, T = instances(640, 9)
        jobs.append({"handle": big, "cx": cx, "cy": cy, "T": T, "F": [1.0], "group": 8,
                     "field": wltube.field("smooth", fermion=0, nint=4)})
        mixed = ctx.batch_eval(jobs)
        for j, want in zip(jobs[:3], mixed):
            for a, b in zip(ctx.batch_eval([j])[0], want):
                np.testing.assert_array_equal(a, b)
