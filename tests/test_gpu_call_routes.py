"""Calls whose route depends on the stream, the context's memory or the parameters' signs: the
results are the oracle's on every route, and no route refuses what another takes."""
import ctypes as C

import numpy as np
import pytest

from conftest import bits_equal

pytestmark = pytest.mark.gpu


def images(seed, W, H, D):
    """Random dots, and a colour pair of flat blocks (long arms)."""
    import rtstereo_gb300 as R
    L, Rr, _ = R.synth_pair(seed, W, H, D, 3, 0, 2.0, min(4, D - 1))
    rng = np.random.default_rng(seed)
    base = np.repeat(np.repeat(rng.integers(0, 200, (H // 11 + 1, W // 11 + 1, 3)), 11, 0), 11, 1)[:H, :W]
    Lc = (base + L[..., None] // 16).astype(np.uint8)
    return L, Rr, Lc, np.ascontiguousarray(np.roll(Lc, -2, 1))


def oracle_params(O, p):
    return O.params(cost1=p.cost1, cost2=p.cost2, aggr=p.aggr, lambda1=p.lambda1, lambda2=p.lambda2, D=p.disp_range,
                    rank_rad=p.rank_rad, box_rad=p.box_rad, cross_L=p.cross_arm, cross_tau=p.cross_tau,
                    ad_trunc=p.ad_trunc, right_view=p.right_view, median_ksize=p.median_ksize)


class DeviceCall:
    """One rts_pipeline_run on device buffers."""

    def __init__(self, ctx, p, imgs, cost=False):
        import torch
        import rtstereo_gb300 as R
        H, W = imgs[0].shape
        self.ctx, self.p = ctx, p
        self.ims = [torch.from_numpy(i).cuda() for i in imgs]
        self.outs = [torch.zeros(H, W, dtype=torch.uint8, device="cuda") for _ in range(3)]
        self.vol = torch.empty(H, W, p.disp_range, device="cuda") if cost else None
        ptr = [i.data_ptr() for i in self.ims] + [None] * (4 - len(imgs))
        self.pair = R.Pair(W, H, *ptr, None, None)
        self.out = R.Out(*[t.data_ptr() for t in self.outs], self.vol.data_ptr() if cost else None)
        torch.cuda.synchronize()

    def __call__(self):
        import rtstereo_gb300 as R
        self.ctx.call("pipeline_run", R.DEVICE, C.byref(self.pair), C.byref(self.p), C.byref(self.out))

    def check(self, want):
        import torch
        torch.cuda.synchronize()
        for t, w in zip(self.outs, want[:3] if self.p.right_view else want[:1]):
            assert bits_equal(t.cpu().numpy(), w)


def last_error(ctx):
    return ctx._lib.rts_ctx_last_error(ctx.h)


@pytest.mark.parametrize("median", [0, 3])
def test_recorded_after_calls_for_the_volume(oracle_mod, median):
    """A context that has only made the volume (module kernels) can record the same pair without
    it, and records nothing besides that call's kernels."""
    torch = pytest.importorskip("torch")
    import rtstereo_gb300 as R
    W, H, D = 70, 45, 20
    im = images(5, W, H, D)
    s = torch.cuda.Stream()
    with R.Context(0) as ctx:
        ctx.set_stream(s.cuda_stream)
        p = R.params(disp_range=D, median_ksize=median)
        warm, call = DeviceCall(ctx, p, im, cost=True), DeviceCall(ctx, p, im)
        n0 = ctx.kernel_launches
        warm()
        n1, msg = ctx.kernel_launches, last_error(ctx)
        s.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            call()
        # as many kernels as the volume's call (its cross aggregation adds up to three a view)
        assert ctx.kernel_launches - n1 <= n1 - n0
        assert last_error(ctx) == msg
        g.replay()
        call.check(oracle_mod.pipeline(oracle_params(oracle_mod, p), *im))
        ctx.set_stream(None)


def test_recorded_after_another_range(oracle_mod):
    """The same after calls of a larger range that went through the view kernels."""
    torch = pytest.importorskip("torch")
    import rtstereo_gb300 as R
    W, H = 70, 45
    s = torch.cuda.Stream()
    with R.Context(0) as ctx:
        ctx.set_stream(s.cuda_stream)
        p = R.params(disp_range=13)
        im = images(6, W, H, 13)
        DeviceCall(ctx, R.params(disp_range=21), im)()
        s.synchronize()
        for cost in (False, True):  # both forms find their scratch
            call = DeviceCall(ctx, p, im, cost)
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=s):
                call()
            g.replay()
            call.check(oracle_mod.pipeline(oracle_params(oracle_mod, p), *im))
        ctx.set_stream(None)


@pytest.mark.parametrize("D", [20, 61])
def test_default_stream_handles(oracle_mod, D):
    """The legacy default stream cannot be captured; calls on it and on the per-thread one work."""
    torch = pytest.importorskip("torch")
    import rtstereo_gb300 as R
    im = images(7, 80, 40, D)
    p = R.params(disp_range=D)
    want = oracle_mod.pipeline(oracle_params(oracle_mod, p), *im)
    with R.Context(0) as ctx:
        for handle in (1, 2):  # cudaStreamLegacy, cudaStreamPerThread
            ctx.set_stream(handle)
            call = DeviceCall(ctx, p, im)
            for _ in range(3):
                call()
                call.check(want)
        torch.cuda.synchronize()
        ctx.set_stream(None)


@pytest.mark.parametrize("kw", [dict(), dict(right_view=0), dict(cost1=3, cost2=0), dict(median_ksize=5)], ids=str)
def test_ragged_ranges_of_changing_size(oracle_mod, kw):
    """Larger and smaller pairs in turn over the same scratch, with and without colour."""
    import rtstereo_gb300 as R
    with R.Context(0) as ctx:
        for W, H, D in ((40, 30, 9), (90, 50, 33), (40, 30, 9), (61, 70, 60), (90, 50, 33)):
            im = images(W, W, H, D)
            p = R.params(disp_range=D, **kw)
            for rgb in (True, False):
                got = ctx.pipeline(p, *(im if rgb else im[:2]))
                gray = [np.repeat(g[..., None], 3, 2) for g in im[:2]]
                want = oracle_mod.pipeline(oracle_params(oracle_mod, p), *im[:2], *(im[2:] if rgb else gray))
                for a, b in zip(got[:3] if p.right_view else got[:1], want):
                    assert bits_equal(a, b)


# lambdas and truncations that make costs negative: the general division and signed keys
NEGATIVE = [dict(lambda1=-5.0, lambda2=30.0), dict(lambda1=-5.0, lambda2=-20.0), dict(ad_trunc=-3.0),
            dict(cost1=1, cost2=0, ad_trunc=-3.0), dict(cost1=1, cost2=0, ad_trunc=-2.5),
            dict(cost1=2, cost2=3, rank_rad=3, lambda2=-9.0), dict(cost1=4, cost2=3, lambda1=-9.0),
            dict(cost1=3, cost2=1, lambda2=-25.0)]


@pytest.mark.parametrize("kw", NEGATIVE, ids=str)
@pytest.mark.parametrize("aggr", [3, 1])
@pytest.mark.parametrize("D", [24, 36, 40])
def test_negative_costs(ctx, oracle_mod, kw, aggr, D):
    import rtstereo_gb300 as R
    im = images(D, 70, 45, D)
    p = R.params(disp_range=D, aggr=aggr, box_rad=2, **kw)
    want = oracle_mod.pipeline(oracle_params(oracle_mod, p), *im)
    got = ctx.pipeline(p, *im)
    assert all(bits_equal(a, b) for a, b in zip(got[:3], want))


@pytest.mark.parametrize("kw", NEGATIVE[:2], ids=str)
def test_negative_costs_fp16_batch_and_server(ctx, oracle_mod, kw):
    """A batch and the serving loop give what single calls give.  FP16 winners: a row segment of costs
    of one sign is rounded by 2^-11 of itself at most, so a mean is, and a winner's plain cost lies
    within twice that of the least one (and 2^-14 for the plain form's own roundings)."""
    pytest.importorskip("torch")
    import rtstereo_gb300 as R
    dims = [(70, 45, 24), (90, 30, 40)]
    data = [images(D, W, H, D) for W, H, D in dims]
    for prec in (R.PREC_F32, R.PREC_F16):
        ps = [R.params(disp_range=D, precision=prec, **kw) for _, _, D in dims]
        single = [ctx.pipeline(p, *im)[:3] for p, im in zip(ps, data)]
        for p, im, s in zip(ps, data, single):
            plain = oracle_mod.pipeline(oracle_params(oracle_mod, p), *im, want_cost=True)
            if prec == R.PREC_F32:
                assert all(bits_equal(a, b) for a, b in zip(s, plain))
            elif kw["lambda1"] < 0 and kw["lambda2"] < 0:
                c = plain[3]
                tol = (2.0 ** -10 + 2.0 ** -14) * np.abs(c).max(2)
                won = c[:, :, 0] > c.min(2) + tol  # a winner of its own, whatever the roundings
                lead = np.take_along_axis(c, s[0][..., None].astype(np.int64), 2)[..., 0] - c.min(2)
                assert won.mean() > 0.5 and (lead[won] <= tol[won]).all()
        calls = [DeviceCall(ctx, p, im) for p, im in zip(ps, data)]
        ctx.batch_run([c.pair for c in calls], ps, [c.out for c in calls])
        for c, s in zip(calls, single):
            c.check(s)
        srv = R.Server(ctx, hbm_budget=1 << 28, max_inflight=4, max_batch=2, precision=prec)
        try:
            tickets = [srv.submit(p, *im) for p, im in zip(ps, data)]
            for t, _ in tickets:
                srv.wait(t)
            for (_, outs), s in zip(tickets, single):
                assert all(bits_equal(a, b) for a, b in zip(outs, s))
        finally:
            srv.close()


def test_ragged_pairs_hold_no_second_volume():
    """A ragged range through the view kernels holds the module kernels' volumes and 100 bytes a
    pixel (each slot an eighth and two pages more), whatever the range."""
    import rtstereo_gb300 as R
    W, H, D = 130, 70, 61
    im = images(2, W, H, D)
    with R.Context(0) as a, R.Context(0) as b:
        a.pipeline(R.params(disp_range=D), *im)
        b.pipeline(R.params(disp_range=D), *im, want_cost=True)
        out = W * H * D * 4  # b's volume on its way to the host
        assert a.bytes_in_use - (b.bytes_in_use - out) <= 1.125 * (100 * W * H + 16384) + 3 * 8192


def test_more_shapes_than_graphs(oracle_mod):
    """Ragged shapes met again and again, more of them than graphs are kept."""
    import rtstereo_gb300 as R
    dims = [(130 + 3 * i, 20 + i, 9 + i) for i in range(19)]
    data = [images(W, W, H, D) for W, H, D in dims]
    with R.Context(0) as ctx:
        ps = [R.params(disp_range=D) for _, _, D in dims]
        want = [oracle_mod.pipeline(oracle_params(oracle_mod, p), *im) for p, im in zip(ps, data)]
        for order in (range(19), range(19), (0, 0, 0, 18, 18, 5, 5, 0), reversed(range(19))):
            for i in order:
                got = ctx.pipeline(ps[i], *data[i])
                assert all(bits_equal(a, b) for a, b in zip(got[:3], want[i]))


def test_batch_of_narrow_and_wide_pairs(ctx, oracle_mod):
    """Narrow pairs beside a wide one share the vertical kernel; alone they do not."""
    pytest.importorskip("torch")
    import rtstereo_gb300 as R
    dims = [(9, 12, 8), (33, 20, 24), (140, 21, 128), (40, 30, 40), (260, 10, 256)]
    data = [images(W, W, H, D) for W, H, D in dims]
    ps = [R.params(disp_range=D) for _, _, D in dims]
    want = [oracle_mod.pipeline(oracle_params(oracle_mod, p), *im) for p, im in zip(ps, data)]
    for n in (2, 3, 5):
        calls = [DeviceCall(ctx, p, im) for p, im in zip(ps[:n], data)]
        ctx.batch_run([c.pair for c in calls], ps[:n], [c.out for c in calls])
        for c, w in zip(calls, want):
            c.check(w)


@pytest.mark.parametrize("rows", [16, 24, 33, 64, 4096])
@pytest.mark.parametrize("W,H,D", [(128, 97, 16), (300, 70, 60), (131, 50, 128)])
def test_strips(ctx, oracle_mod, rows, W, H, D):
    import rtstereo_gb300 as R
    im = images(W, W, H, D)
    p = R.params(disp_range=D)
    want = oracle_mod.pipeline(oracle_params(oracle_mod, p), *im)
    ctx.force_cross_tune(rows)
    try:
        got = ctx.pipeline(p, *im)
    finally:
        ctx.force_cross_tune(0)
    assert all(bits_equal(a, b) for a, b in zip(got[:3], want))


class Aggregation:
    """One rts_cross_stereo_aggregation on device buffers, large enough for the kernels with scratch."""

    def __init__(self, O, seed, H=90, W=200, D=33):
        import torch
        rng = np.random.default_rng(seed)
        a, b = images(seed, W, H, 16)[2:]
        arms = [x for im in (a, b) for x in O.find_cross(im, 17, 20)]
        pre = O.prefix_h(rng.normal(0.5, 1.0, (H, W, D)).astype(np.float32))
        self.want = O.cross_aggr(pre, arms[0], arms[2], arms[1], arms[3])
        self.dev = [torch.from_numpy(x).cuda() for x in (pre, arms[0], arms[2], arms[1], arms[3])]
        self.out = torch.zeros(H, W, D, device="cuda")
        self.dims = (H, W, D)
        torch.cuda.synchronize()

    def call(self, ctx):
        import rtstereo_gb300 as R
        ctx.call("cross_stereo_aggregation", R.DEVICE, self.dev[0], self.out, *self.dev[1:], *self.dims)

    def check(self):
        assert bits_equal(self.out.cpu().numpy(), self.want)
        self.out.zero_()


def test_more_streams_than_scratch_buffers(oracle_mod):
    """Calls on any number of streams, destroyed ones among them, all get scratch and do not
    overwrite each other's."""
    torch = pytest.importorskip("torch")
    import rtstereo_gb300 as R
    jobs = [Aggregation(oracle_mod, i, D=33 + 2 * i) for i in range(7)]
    with R.Context(0) as ctx:
        held = []
        for rnd in range(3):
            streams = [torch.cuda.Stream() for _ in jobs]
            for s, j in zip(streams, jobs):
                ctx.set_stream(s.cuda_stream)
                n = ctx.kernel_launches
                j.call(ctx)
                assert ctx.kernel_launches - n == 4
            torch.cuda.synchronize()
            for j in jobs:
                j.check()
            held.append(ctx.bytes_in_use)
            del streams
        assert max(held) <= 4 * 1.2 * max(4 * (np.prod(j.dims) + 4 * j.dims[0] * j.dims[1]) for j in jobs)
        ctx.set_stream(None)


def test_scratch_within_a_budget(oracle_mod):
    """Without room for scratch the general kernel makes the same result, and no error is left;
    scratch stays where another call fits at its exact size, and goes where it does not."""
    pytest.importorskip("torch")
    import rtstereo_gb300 as R
    job = Aggregation(oracle_mod, 11)
    H, W, D = job.dims
    with R.Context(0, 1 << 20) as ctx:
        n, msg = ctx.kernel_launches, last_error(ctx)
        job.call(ctx)
        assert ctx.kernel_launches - n == 1 and last_error(ctx) == msg
        ctx.synchronize()
        job.check()
    with R.Context(0) as ctx:
        job.call(ctx)
        work = ctx.bytes_in_use
    vol = H * W * D * 4
    cost = np.random.default_rng(1).normal(0, 1, (H, W, D)).astype(np.float32)
    tall = np.concatenate([cost, cost])[: H + H // 2]
    with R.Context(0, work + vol) as ctx:
        job.call(ctx)
        assert bits_equal(ctx.aggregate_cost_horizontal(cost), oracle_mod.prefix_h(cost))
        assert ctx.bytes_in_use == work + vol
        n = ctx.kernel_launches
        job.call(ctx)
        assert ctx.kernel_launches - n == 4
        assert bits_equal(ctx.aggregate_cost_horizontal(tall), oracle_mod.prefix_h(tall))
        assert ctx.bytes_in_use <= work + vol
        job.call(ctx)
        ctx.synchronize()
        job.check()


@pytest.mark.parametrize("kw", [dict(disp_range=21), dict(disp_range=13, cost1=3, cost2=0),
                                dict(disp_range=21, aggr=2, aw_rad=3), dict(disp_range=21, aggr=2, aw_rad=3, precision=1),
                                dict(disp_range=21, aggr=2, aw_rad=17)], ids=str)
def test_smaller_budgets(kw):
    """Every budget gives the same bits or is refused; what a call needs at least does not grow
    with the room there is."""
    import rtstereo_gb300 as R
    im = images(9, 90, 40, 24)
    p = R.params(**kw)
    lab = [R.rgb_to_lab(i) for i in im[2:]] if p.aggr == R.AGGR_AW else [None, None]
    with R.Context(0) as ctx:
        want = ctx.pipeline(p, *im, *lab)[:3]
        full = ctx.bytes_in_use
    refused = False
    for k in range(40, 0, -1):
        with R.Context(0, full * k // 40) as ctx:
            try:
                got = [ctx.pipeline(p, *im, *lab)[:3] for _ in range(2)]
            except R.RtsError:
                refused = True
                continue
            assert not refused
            assert all(bits_equal(a, b) for g in got for a, b in zip(g, want))
    assert refused


@pytest.mark.parametrize("prec", [0, 1])
def test_padded_adaptive_weight_volume_is_the_only_one(prec):
    """A range that is no multiple of 16 bytes holds no more than the padded range does."""
    import rtstereo_gb300 as R
    im = images(4, 90, 30, 24)
    lab = [R.rgb_to_lab(i) for i in im[2:]]
    held = []
    for D in (21, 24):
        with R.Context(0) as ctx:
            ctx.pipeline(R.params(disp_range=D, aggr=2, aw_rad=4, precision=prec), *im, *lab)
            held.append(ctx.bytes_in_use)
    assert held[0] <= held[1]


@pytest.mark.parametrize("prec", [0, 1])
def test_recorded_adaptive_weights(oracle_mod, prec):
    torch = pytest.importorskip("torch")
    import rtstereo_gb300 as R
    im = images(4, 90, 30, 21)
    lab = [torch.from_numpy(R.rgb_to_lab(i)).cuda() for i in im[2:]]
    s = torch.cuda.Stream()
    with R.Context(0) as ctx:
        ctx.set_stream(s.cuda_stream)
        p = R.params(disp_range=21, aggr=2, aw_rad=4, precision=prec)
        call = DeviceCall(ctx, p, im)
        call.pair.left_lab, call.pair.right_lab = (t.data_ptr() for t in lab)
        call()
        torch.cuda.synchronize()
        want = [t.cpu().numpy() for t in call.outs]
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            call()
        for t in call.outs:
            t.zero_()
        g.replay()
        call.check(want)
        ctx.set_stream(None)


def test_tiles_of_other_threads(oracle_mod):
    """Contexts on threads of their own whose kernels want different amounts of shared memory."""
    import threading
    import rtstereo_gb300 as R
    L, Rr, Lc, Rc = images(3, 300, 40, 64)
    disp = np.random.default_rng(0).integers(0, 64, (40, 300), dtype=np.uint8)
    failures = []

    def work(D, arm, rad):
        try:
            with R.Context(0) as c:
                horz, vert = c.findCross(Lc, 17, 20)
                jobs = [(lambda: (c.disp_refinement(disp, horz, vert, D),)),
                        (lambda: c.pipeline(R.params(disp_range=D, cross_arm=arm), L, Rr, Lc, Rc)[:3]),
                        (lambda: c.pipeline(R.params(disp_range=D, aggr=R.AGGR_AW, aw_rad=rad), L, Rr, Lc, Rc, Lc, Rc)[:3])]
                want = [j() for j in jobs]
                for _ in range(150):
                    for j, w in zip(jobs, want):
                        assert all(bits_equal(a, b) for a, b in zip(j(), w))
        except Exception as e:  # noqa: BLE001 (reported below)
            failures.append(e)

    ts = [threading.Thread(target=work, args=a) for a in ((256, 23, 16), (8, 3, 1), (64, 17, 5), (128, 20, 12))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not failures
