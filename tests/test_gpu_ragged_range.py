"""Disparity ranges that are not a multiple of 8 in the cross-based pipeline: the view
kernels' results against the C oracle, bit for bit, over costs, forms, colours and
sizes; and where the call must fall back to the module kernels."""
import numpy as np
import pytest

from conftest import bits_equal

pytestmark = pytest.mark.gpu


def pair(seed, W, H, D, colour):
    import rtstereo_gb300 as R
    L, Rr, _ = R.synth_pair(seed, W, H, D, 3, 0, 2.0, min(4, D - 1))
    if not colour:
        return (L, Rr), (R.gray_to_rgb(L), R.gray_to_rgb(Rr))
    rng = np.random.default_rng(seed)
    # blocks of one colour: long arms
    base = np.repeat(np.repeat(rng.integers(0, 200, (H // 11 + 1, W // 11 + 1, 3)), 11, 0), 11, 1)[:H, :W]
    Lc = (base + L[..., None] // 16).astype(np.uint8)
    Rc = np.ascontiguousarray(np.roll(Lc, -min(2, W - 1), 1))
    return (L, Rr), (Lc, Rc)


def check(ctx, O, W, H, D, colour, **kw):
    import rtstereo_gb300 as R
    (L, Rr), (Lc, Rc) = pair(W + H + D, W, H, D, colour)
    p = R.params(disp_range=D, **kw)
    got = ctx.pipeline(p, L, Rr, Lc, Rc) if colour else ctx.pipeline(p, L, Rr)
    o = O.pipeline(O.params(cost1=p.cost1, cost2=p.cost2, aggr=3, lambda1=p.lambda1, lambda2=p.lambda2, D=D,
                            rank_rad=p.rank_rad, cross_L=p.cross_arm, cross_tau=p.cross_tau, ad_trunc=p.ad_trunc,
                            right_view=p.right_view), L, Rr, Lc, Rc)
    assert bits_equal(got[0], o[0])
    if p.right_view:
        assert bits_equal(got[1], o[1]) and bits_equal(got[2], o[2])


@pytest.mark.parametrize("W,H,D", [(9, 12, 1), (20, 11, 7), (61, 40, 20), (90, 33, 60), (140, 20, 129), (300, 9, 255)])
@pytest.mark.parametrize("colour", [False, True])
@pytest.mark.parametrize("precision", [0, 1])
def test_sizes(ctx, oracle_mod, W, H, D, colour, precision):
    # the FP16 form of such a range has always been the plain one
    check(ctx, oracle_mod, W, H, D, colour, precision=precision)


@pytest.mark.parametrize("kw", [dict(cost1=3, cost2=0), dict(cost1=1, cost2=0), dict(cost1=2, cost2=3, rank_rad=3),
                                dict(ad_trunc=7.5), dict(cost1=3, cost2=1), dict(right_view=0), dict(cross_arm=23),
                                dict(cross_arm=24), dict(lambda1=-5.0, lambda2=30.0), dict(ad_trunc=-3.0),
                                dict(cost1=1, cost2=0, ad_trunc=1000.0)], ids=str)
def test_options(ctx, oracle_mod, kw):
    check(ctx, oracle_mod, 70, 45, 20, True, **kw)


def test_captured_call(oracle_mod):
    """On a captured stream the call records the module kernels; replays give the same results."""
    torch = pytest.importorskip("torch")
    import rtstereo_gb300 as R
    import ctypes as C
    W, H, D = 70, 45, 20
    (L, Rr), _ = pair(5, W, H, D, False)
    s = torch.cuda.Stream()
    with R.Context(0) as ctx:
        ctx.set_stream(s.cuda_stream)
        l, r = torch.from_numpy(L).cuda(), torch.from_numpy(Rr).cuda()
        outs = [torch.empty(H, W, dtype=torch.uint8, device="cuda") for _ in range(3)]
        p = R.params(disp_range=D)
        prm = (R.Pair(W, H, l.data_ptr(), r.data_ptr(), None, None, None, None), p,
               R.Out(*[t.data_ptr() for t in outs], None))
        torch.cuda.synchronize()
        call = lambda: ctx.call("pipeline_run", R.DEVICE, *[C.byref(x) for x in prm])
        call()
        s.synchronize()
        want = [t.cpu().numpy().copy() for t in outs]
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            call()
        for t in outs:
            t.zero_()
        g.replay()
        torch.cuda.synchronize()
        for a, b in zip(outs, want):
            assert bits_equal(a.cpu().numpy(), b)
        ctx.set_stream(None)
    o = oracle_mod.pipeline(oracle_mod.params(D=D), L, Rr, *pair(5, W, H, D, False)[1])
    assert bits_equal(want[0], o[0]) and bits_equal(want[1], o[1])


# adaptive weights: volumes whose pixels are not whole 16-byte runs, one and two disparity chunks
@pytest.mark.parametrize("D", [1, 5, 20, 62, 67])
@pytest.mark.parametrize("rad", [3, 16])
def test_adaptive_weights(ctx, oracle_mod, D, rad):
    import rtstereo_gb300 as R
    W, H = 90, 21
    (L, Rr), (Lc, Rc) = pair(D, W, H, D, True)
    ll, rl = R.rgb_to_lab(Lc), R.rgb_to_lab(Rc)
    got = ctx.pipeline(R.params(disp_range=D, aggr=2, aw_rad=rad), L, Rr, Lc, Rc, ll, rl, want_cost=True)
    o = oracle_mod.pipeline(oracle_mod.params(D=D, aggr=2, aw_rad=rad), L, Rr, Lc, Rc, ll, rl, want_cost=True)
    for a, b in zip(got, o):
        assert bits_equal(a, b)
    # FP16: an entry does not depend on the range it is computed in
    wide = (D + 7) // 8 * 8
    f = [ctx.pipeline(R.params(disp_range=d, aggr=2, aw_rad=rad, precision=1), L, Rr, Lc, Rc, ll, rl, want_cost=True)
         for d in (D, wide)]
    assert bits_equal(f[0][3], np.ascontiguousarray(f[1][3][:, :, :D]))
    assert bits_equal(f[0][0], oracle_mod.wta(f[0][3]))


# the AD + census volume under box and adaptive weights: disparity groups of four and remainders, pixels
# past a block's 64, single tables (small pairs) and copied ones (many items)
@pytest.mark.parametrize("W,H,D", [(9, 9, 3), (70, 33, 37), (200, 20, 64), (257, 12, 256), (129, 1500, 6)])
@pytest.mark.parametrize("colour", [False, True])
def test_ad_census_volume(ctx, oracle_mod, W, H, D, colour):
    import rtstereo_gb300 as R
    (L, Rr), (Lc, Rc) = pair(W, W, H, D, colour)
    for prec in (0, 1):
        p = R.params(disp_range=D, aggr=1, box_rad=2, precision=prec)
        got = ctx.pipeline(p, L, Rr, Lc, Rc)
        o = oracle_mod.pipeline(oracle_mod.params(D=D, aggr=1, box_rad=2), L, Rr, Lc, Rc)
        assert bits_equal(got[0], o[0])
        if prec == 0:
            assert bits_equal(got[1], o[1]) and bits_equal(got[2], o[2])


@pytest.mark.parametrize("kw", [dict(aggr=1, box_rad=3), dict(aggr=1, box_rad=9), dict(aggr=1, cost1=3, cost2=0),
                                dict(aggr=1, cost1=3, cost2=1, lambda2=25.0), dict(aggr=2, aw_rad=4),
                                dict(aggr=2, aw_rad=4, cost1=1, cost2=0), dict(aggr=2, aw_rad=4, cost1=2, rank_rad=3),
                                dict(aggr=0)], ids=str)
@pytest.mark.parametrize("colour", [False, True])
@pytest.mark.parametrize("want_cost", [False, True])
def test_right_view_from_shared_records(ctx, oracle_mod, kw, colour, want_cost):
    """Both views where the right one reads the left one's records, and where it cannot."""
    import rtstereo_gb300 as R
    W, H, D = 83, 30, 36
    (L, Rr), (Lc, Rc) = pair(77, W, H, D, colour)
    ll, rl = R.rgb_to_lab(Lc), R.rgb_to_lab(Rc)
    p = R.params(disp_range=D, **kw)
    imgs = (L, Rr, Lc, Rc) if colour else (L, Rr, None, None)
    got = ctx.pipeline(p, *imgs, ll, rl, want_cost=want_cost)
    o = oracle_mod.pipeline(oracle_mod.params(D=D, **kw), L, Rr, Lc, Rc, ll, rl, want_cost=want_cost)
    for a, b in zip(got, o):
        assert a is None or bits_equal(a, b)
