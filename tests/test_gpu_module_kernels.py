"""GPU parity of the tiled module kernels at the sizes where their splits can go
wrong (edges of tiles, remainders, the smallest and largest of a range), against
the C oracle; the bar is bit-exact."""
import numpy as np
import pytest

from conftest import bits_equal, smooth

pytestmark = pytest.mark.gpu


def patches(seed, H, W, ch=3, step=9):
    """Piecewise-constant image with a little noise: long cross arms."""
    rng = np.random.default_rng(seed)
    g = rng.integers(0, 256, (H // step + 1, W // step + 1, ch))
    im = np.repeat(np.repeat(g, step, 0), step, 1)[:H, :W]
    return np.ascontiguousarray(np.clip(im + rng.integers(-3, 4, im.shape), 0, 255).astype(np.uint8))


# runs that end at, cross and start at the aligned 32; arms up to 17 and 40 (runs are cut at xr)
@pytest.mark.parametrize("H,W,D,arm", [(1, 1, 1, 17), (9, 31, 7, 17), (23, 64, 33, 17), (40, 97, 64, 40), (12, 300, 256, 17)])
def test_disp_refinement(ctx, oracle_mod, H, W, D, arm):
    O = oracle_mod
    rgb = patches(H, H, W)
    horz, vert = ctx.findCross(rgb, arm, 20)
    rng = np.random.default_rng(W)
    for disp in (rng.integers(0, D, (H, W)), np.repeat(rng.integers(0, D, (H, W // 40 + 1)), 40, 1)[:, :W],
                 rng.integers(0, 256, (H, W))):  # votes at or above D count for nothing
        disp = np.ascontiguousarray(disp.astype(np.uint8))
        assert bits_equal(ctx.disp_refinement(disp, horz, vert, D), O.disp_refinement(disp, horz, vert, D))


def patches_pair(seed, H, W):
    a, b = patches(seed, H, W), patches(seed + 100, H, W)
    b[:, : W // 2] = np.roll(a, 3, 1)[:, : W // 2]  # half of it matches: arms of both lengths
    return a, b


# one chunk, ragged chunks, strips (64 rows and more of few columns), one row and column; arms above
# kModArm = 20 and foreign arms (outside the image, negative) take the general kernel
@pytest.mark.parametrize("H,W,D", [(1, 1, 1), (6, 33, 32), (131, 40, 33), (200, 9, 5), (50, 300, 70), (9, 257, 256)])
@pytest.mark.parametrize("arm", [0, 17, 20, 21])
def test_cross_aggregation(ctx, oracle_mod, H, W, D, arm):
    O = oracle_mod
    a, b = patches_pair(H + W, H, W)
    ha, va = ctx.findCross(a, arm, 20)
    hb, vb = ctx.findCross(b, arm, 20)
    assert bits_equal(ha, O.find_cross(a, arm, 20)[0]) and bits_equal(va, O.find_cross(a, arm, 20)[1])
    cost = np.random.default_rng(D).normal(0.5, 1.0, (H, W, D)).astype(np.float32)  # sums of either sign
    pre = ctx.aggregate_cost_horizontal(cost)
    want = O.prefix_h(cost)
    assert bits_equal(pre, want)
    assert bits_equal(ctx.cross_stereo_aggregation(pre, ha, hb, va, vb), O.cross_aggr(want, ha, hb, va, vb))


def test_cross_aggregation_foreign_arms(ctx, oracle_mod):
    """Arms that leave the image go to the general kernel, whatever image they are in."""
    H, W, D = 20, 50, 12
    a, b = patches_pair(3, H, W)
    (ha, va), (hb, vb) = ctx.findCross(a, 17, 20), ctx.findCross(b, 17, 20)
    pre = ctx.aggregate_cost_horizontal(np.random.default_rng(1).random((H, W, D), dtype=np.float32))
    for arr, at, v in ((ha, (0, 0, 0), 5), (hb, (3, 7, 1), 60), (va, (H - 1, 4, 1), 2), (vb, (2, 2, 0), 19)):
        arms = [x.copy() for x in (ha, hb, va, vb)]
        arms[[id(ha), id(hb), id(va), id(vb)].index(id(arr))][at] = v
        assert bits_equal(ctx.cross_stereo_aggregation(pre, *arms), oracle_mod.cross_aggr(pre, *arms))


# rows shorter than a warp's 32 pixels, warps that end a row, a ragged last warp; rows without a winner
@pytest.mark.parametrize("H,W,D", [(1, 1, 1), (7, 3, 3), (5, 33, 32), (9, 40, 33), (3, 299, 256), (40, 64, 2)])
def test_wta(ctx, oracle_mod, H, W, D):
    O = oracle_mod
    rng = np.random.default_rng(H * W + D)
    cost = rng.integers(0, 6, (H, W, D)).astype(np.float32)  # ties
    cost[rng.random((H, W)) < 0.3, 0] = -1.0                 # no winner of their own: carried
    cost[H // 2] = 0.0                                       # a whole row carried
    special = rng.random((H, W, D)) < 0.03
    cost[special] = rng.choice(np.array([np.nan, np.inf, -np.inf, -0.0, 3.4028235e38], np.float32), special.sum())
    assert bits_equal(ctx.WTA(cost), O.wta(cost))
    assert bits_equal(ctx.WTA_NCC(cost), O.wta(cost, True))


# batches of 32 columns: shorter, exact, one more; chains across a block's end
@pytest.mark.parametrize("H,W,D", [(1, 1, 1), (3, 31, 5), (2, 32, 33), (5, 33, 64), (1, 65, 256), (70, 100, 3)])
def test_prefix(ctx, oracle_mod, H, W, D):
    cost = np.random.default_rng(W).normal(0.0, 1.0, (H, W, D)).astype(np.float32)
    cost[0, 0, 0] = -0.0
    assert bits_equal(ctx.aggregate_cost_horizontal(cost), oracle_mod.prefix_h(cost))


# both lane widths, odd and ragged disparities, tiles inside (TMA where D % 4 == 0) and at the wrap,
# the smallest and largest tiled radius, radius 9 and 0 (untiled)
@pytest.mark.parametrize("H,W,D,r", [(10, 11, 1, 1), (40, 70, 32, 4), (41, 50, 33, 4), (33, 67, 64, 2), (40, 60, 68, 8),
                                     (25, 45, 130, 3), (20, 30, 31, 8), (24, 50, 12, 5), (21, 40, 9, 9), (5, 6, 40, 0)])
def test_box(ctx, oracle_mod, H, W, D, r):
    rng = np.random.default_rng(D * r)
    cost = rng.normal(0.2, 1.0, (H, W, D)).astype(np.float32)
    assert bits_equal(ctx.boxAggregate(cost, r), oracle_mod.box(cost, r))
    cost[rng.random(cost.shape) < 0.9] = 0.0  # zero and tiny sums, then infinite and NaN ones
    cost *= np.float32(1e-37)
    cost[rng.random(cost.shape) < 0.001] = np.inf
    cost[rng.random(cost.shape) < 0.001] = -np.inf
    got, want = ctx.boxAggregate(cost, r), oracle_mod.box(cost, r)
    assert np.array_equal(np.isnan(got), np.isnan(want)) and bits_equal(np.nan_to_num(got), np.nan_to_num(want))


# means of signed sums beside flat areas (sums of exactly zero), partial blocks of disparities,
# tiles inside and at the wrap
@pytest.mark.parametrize("H,W,D,r", [(40, 70, 64, 4), (21, 50, 34, 1), (24, 150, 130, 8)])
def test_ncc_box_flat(ctx, oracle_mod, H, W, D, r):
    import rtstereo_gb300 as R
    O = oracle_mod
    L, Rr, _ = R.synth_pair(D + r, W, H, D, 3, 0, 2.0, 4)
    L[:, W // 2:] = 90
    Rr[:, W // 2:] = 90
    p = R.params(disp_range=D, cost1=R.COST_NCC, cost2=R.COST_NONE, aggr=R.AGGR_BOX, box_rad=r, ncc_hrad=2, ncc_wrad=2)
    got = ctx.pipeline(p, L, Rr)
    c = (R.gray_to_rgb(L), R.gray_to_rgb(Rr))
    want = O.pipeline(O.params(cost1=5, cost2=0, aggr=1, D=D, box_rad=r, ncc_hrad=2, ncc_wrad=2), L, Rr, *c)
    assert all(bits_equal(got[i], want[i]) for i in range(3))


# whole and partial pixel blocks of a row, every code width, both directions
@pytest.mark.parametrize("H,W,D", [(1, 1, 1), (3, 31, 9), (2, 64, 64), (5, 33, 33), (2, 300, 256), (70, 20, 20)])
def test_cost_rows(ctx, oracle_mod, H, W, D):
    O = oracle_mod
    rng = np.random.default_rng(W + D)
    L, R = rng.integers(0, 256, (2, H, W), dtype=np.uint8)
    Lc, Rc = rng.integers(0, 256, (2, H, W, 3), dtype=np.uint8)
    Lf, Rf = rng.normal(0, 90, (2, H, W)).astype(np.float32)
    for d, gray, colour, fl in ((O.L2R, ctx.pixelBasedL2R, ctx.pixelBasedCostL2R_Color, ctx.pixelBasedCostL2R_Float),
                                (O.R2L, ctx.pixelBasedR2L, ctx.pixelBasedR2L_Color, ctx.pixelBasedCostR2L_Float)):
        assert bits_equal(gray(L, R, D), O.ad_gray(L, R, D, d))
        assert bits_equal(colour(Lc, Rc, D, 1, 100.5), O.ad_color(Lc, Rc, D, d, 100.5, 1))
        assert bits_equal(fl(Lf, Rf, D), O.ad_float(Lf, Rf, D, d))
    for nb in ((0, 0), (0, 4), (0, 60)):  # 1, 9 and 121 bits; nonzero bytes count as set
        b = rng.integers(0, 3, (2, H, W, 2 * nb[1] + 1), dtype=np.uint8)
        want = O.hamming((b[0] != 0).astype(np.uint8), (b[1] != 0).astype(np.uint8), D, *nb)
        assert bits_equal(ctx.calcHammingDist(b[0], b[1], D, *nb), want)


# windows up to and above the 256 bits of the pixel kernel, images narrower than a block of 128
@pytest.mark.parametrize("H,W,hr,wr", [(1, 1, 0, 0), (9, 15, 4, 3), (40, 33, 7, 8), (30, 130, 8, 7), (20, 40, 3, 18), (30, 40, 9, 9)])
def test_census_bits(ctx, oracle_mod, H, W, hr, wr):
    img = np.random.default_rng(W).integers(0, 9, (H, W), dtype=np.uint8)
    assert bits_equal(ctx.calcCensusTrans(img, hr, wr), oracle_mod.census(img, hr, wr))


@pytest.mark.parametrize("n", [1, 3, 4, 7, 1025])
def test_combine_remainders(ctx, oracle_mod, n):
    c1 = np.arange(n, dtype=np.float32).reshape(1, n, 1)
    assert bits_equal(ctx.combineCost(c1, c1[:, ::-1].copy(), 10.0, 30.0), oracle_mod.combine(c1, c1[:, ::-1].copy(), 10.0, 30.0))


def test_device_buffers_without_vector_alignment(ctx, oracle_mod):
    """Device buffers aligned to their element alone: the wide loads and stores must not be used."""
    torch = pytest.importorskip("torch")
    import rtstereo_gb300 as R
    O, dev = oracle_mod, R.DEVICE
    H, W, D = 21, 50, 36
    rng = np.random.default_rng(5)

    def put(a):
        """The array one element past an aligned address."""
        t = torch.empty(a.size + 1, dtype=torch.from_numpy(a).dtype, device="cuda")[1:].view(a.shape)
        return t.copy_(torch.from_numpy(a))

    img = rng.integers(0, 256, (H, W), dtype=np.uint8)
    c1, c2 = rng.integers(0, 60, (2, H, W, D)).astype(np.float32)
    rgb = patches(8, H, W)
    bits, cost, comb = put(np.zeros((H, W, 63), np.uint8)), put(c1), put(c1)
    horz, vert = (put(np.zeros((H, W, 2), np.int32)) for _ in range(2))
    disp = put(img % 16)
    ham, fin = put(c2), put(c2)
    args = [put(x) for x in (img, c2, rgb)]
    torch.cuda.synchronize()
    ctx.call("calcCensusTrans", dev, args[0], bits, 4, 3, H, W)
    ctx.call("calcHammingDist", dev, bits, bits, ham, 4, 3, H, W, D)
    ctx.call("combineCost", dev, comb, args[1], 10.0, 10.0, H, W, D)
    ctx.call("boxAggregate", dev, cost, H, W, D, 3)
    ctx.call("findCross", dev, args[2], horz, vert, H, W)
    ctx.call("cross_stereo_aggregation", dev, cost, fin, horz, horz, vert, vert, H, W, D)
    ctx.call("disp_refinement", dev, disp, horz, vert, H, W, D)
    ctx.synchronize()
    b, box = O.census(img, 4, 3), O.box(c1, 3)
    h, v = O.find_cross(rgb)
    assert bits_equal(bits.cpu().numpy(), b) and bits_equal(ham.cpu().numpy(), O.hamming(b, b, D, 4, 3))
    assert bits_equal(comb.cpu().numpy(), O.combine(c1, c2, 10.0, 10.0)) and bits_equal(cost.cpu().numpy(), box)
    assert bits_equal(horz.cpu().numpy(), h) and bits_equal(vert.cpu().numpy(), v)
    assert bits_equal(fin.cpu().numpy(), O.cross_aggr(box, h, h, v, v))
    assert bits_equal(disp.cpu().numpy(), O.disp_refinement(img % 16, h, v, D))


# both tile widths, pixels and disparities past their tiles' ends, windows below and above a warp's 32
# taps; weights of any value, outside the image too
@pytest.mark.parametrize("H,W,D,r", [(1, 1, 1, 0), (3, 64, 32, 1), (7, 65, 33, 2), (20, 140, 64, 16), (17, 90, 66, 5),
                                     (18, 40, 7, 17), (3, 260, 129, 2), (47, 80, 33, 46)])
def test_adaptive_weight_tiles(ctx, oracle_mod, H, W, D, r):
    O = oracle_mod
    rng = np.random.default_rng(W + r)
    lab = patches(r, H, W)
    pw = O.prox_weight(36.0, r)
    assert bits_equal(ctx.computeWeights(pw, lab, 7.0, r), O.compute_weights(pw, lab, 7.0, r))
    wl, wr = rng.normal(0.5, 0.5, (2, H, W, (2 * r + 1) ** 2)).astype(np.float32)
    cost = rng.normal(0.0, 1.0, (H, W, D)).astype(np.float32)
    assert bits_equal(ctx.calcAWCostL2R(wl, wr, cost, r), O.aw_l2r(wl, wr, cost, r))
    if r + D <= W:
        assert bits_equal(ctx.calcAWCostR2L(wl, wr, cost, r), O.aw_r2l(wl, wr, cost, r))


# radii whose window passes the tiled kernels' shared memory: weights above 46
@pytest.mark.parametrize("r", [46, 47])
def test_compute_weights_large_window(ctx, oracle_mod, r):
    lab = patches(r, r + 2, 20 + r)
    pw = oracle_mod.prox_weight(36.0, r)
    assert bits_equal(ctx.computeWeights(pw, lab, 7.0, r), oracle_mod.compute_weights(pw, lab, 7.0, r))


# tiles' ends, wraps, radii as constants (2, 3) and not, borders above the tile's 64
@pytest.mark.parametrize("H,W,r", [(1, 1, 0), (17, 65, 1), (33, 130, 2), (16, 64, 3), (40, 70, 3), (70, 90, 9), (66, 68, 65)])
def test_window_filters(ctx, oracle_mod, H, W, r):
    O = oracle_mod
    rng = np.random.default_rng(H)
    img = rng.integers(0, 256, (H, W), dtype=np.uint8)
    assert bits_equal(ctx.calculateRankFilt(img, r), O.rank(img, r))
    mask = rng.normal(0, 0.2, (2 * r + 1) ** 2).astype(np.float32)
    assert bits_equal(ctx.convolveImage(img, mask, r, r), O.convolve(img, mask, r, r))
    D = min(5, W - r)
    if D > 0 and r < 20:  # blocks whose windows wrap and, in the widest image, blocks inside
        other = rng.integers(0, 256, (H, W), dtype=np.uint8)
        assert bits_equal(ctx.calcNCCDispL2R(img, other, D, r, r, fill=-7.0), O.ncc(img, other, D, r, r, fill=-7.0))


@pytest.mark.parametrize("hr,wr", [(3, 3), (1, 5), (4, 4)])
def test_ncc_inside_and_wrapped_blocks(ctx, oracle_mod, hr, wr):
    rng = np.random.default_rng(hr)
    L, R = rng.integers(0, 256, (2, 20, 330), dtype=np.uint8)
    L[:, 100:150] = R[:, 100:150] = 7  # zero denominators
    for D in (10, 70):
        assert bits_equal(ctx.calcNCCDispL2R(L, R, D, hr, wr, fill=-7.0), oracle_mod.ncc(L, R, D, hr, wr, fill=-7.0))


# tiles' ends, arms longer than the image, the longest tiled arm and one above, thresholds at their ends
@pytest.mark.parametrize("H,W", [(1, 1), (16, 64), (17, 65), (50, 131)])
@pytest.mark.parametrize("arm,tau", [(0, 20), (17, 20), (32, 60), (33, 60), (17, 0), (17, -3), (17, 1), (17, 255), (17, 256), (17, 1000)])
def test_find_cross(ctx, oracle_mod, H, W, arm, tau):
    rgb = patches(W, H, W)
    got, want = ctx.findCross(rgb, arm, tau), oracle_mod.find_cross(rgb, arm, tau)
    assert bits_equal(got[0], want[0]) and bits_equal(got[1], want[1])


def test_disp_refinement_crosses_above_16_bits(ctx, oracle_mod):
    """Arms of 255 on a flat image: crosses of more than 65535 pixels."""
    H, W, D = 300, 520, 5
    horz, vert = ctx.findCross(np.zeros((H, W, 3), np.uint8), 255, 20)
    disp = np.random.default_rng(0).integers(0, 2, (H, W), dtype=np.uint8) * 4
    assert bits_equal(ctx.disp_refinement(disp, horz, vert, D), oracle_mod.disp_refinement(disp, horz, vert, D))


# columns side by side in a warp (D up to 8 and 16) and their remainders, strips of 24 rows and
# more, volumes below the size that takes three kernels
@pytest.mark.parametrize("H,W,D", [(300, 601, 3), (170, 403, 8), (97, 651, 9), (130, 257, 16), (100, 310, 17), (49, 331, 33)])
@pytest.mark.parametrize("arm", [17, 21])
def test_cross_aggregation_few_disparities(ctx, oracle_mod, H, W, D, arm):
    O = oracle_mod
    a, b = patches_pair(H + W, H, W)
    (ha, va), (hb, vb) = O.find_cross(a, arm, 20), O.find_cross(b, arm, 20)
    pre = O.prefix_h(np.random.default_rng(D).normal(0.5, 1.0, (H, W, D)).astype(np.float32))
    assert bits_equal(ctx.cross_stereo_aggregation(pre, ha, hb, va, vb), O.cross_aggr(pre, ha, hb, va, vb))


def test_cross_aggregation_foreign_arms_in_a_large_volume(ctx, oracle_mod):
    """One arm that leaves the image or passes the rings sends the whole call to the general kernel."""
    H, W, D = 100, 400, 16
    a, b = patches_pair(7, H, W)
    arms = list(oracle_mod.find_cross(a, 17, 20)) + list(oracle_mod.find_cross(b, 17, 20))  # horz, vert; horz, vert
    pre = oracle_mod.prefix_h(np.random.default_rng(1).random((H, W, D), dtype=np.float32))
    for k, at, v in ((0, (0, 0, 0), 5), (0, (50, 100, 0), 21), (1, (H - 1, 4, 1), 2), (2, (3, 7, 1), -1), (None, None, 0)):
        m = [x.copy() for x in arms]
        if k is not None:
            m[k][at] = v
        args = (pre, m[0], m[2], m[1], m[3])
        assert bits_equal(ctx.cross_stereo_aggregation(*args), oracle_mod.cross_aggr(*args))


# 16-bit counters (D above 128) at their end: two disparities of 78000 votes each (the first where
# they tie), and one of 117000
@pytest.mark.parametrize("D", [129, 256])
def test_disp_refinement_16_bit_counters(ctx, oracle_mod, D):
    H, W = 300, 520
    horz, vert = ctx.findCross(np.zeros((H, W, 3), np.uint8), 255, 20)
    x, y = np.arange(W)[None], np.arange(H)[:, None]
    for disp in ((x + y) % 2 * (D - 1), np.where(x % 4 == 0, 7, D - 1) + 0 * y):
        disp = np.ascontiguousarray(disp.astype(np.uint8))
        assert bits_equal(ctx.disp_refinement(disp, horz, vert, D), oracle_mod.disp_refinement(disp, horz, vert, D))


# the blocks of 128 and 256 pixels of small ranges: whole, partial, one pixel past
@pytest.mark.parametrize("H,W,D", [(2, 256, 8), (3, 257, 5), (2, 513, 1), (3, 128, 16), (2, 129, 12), (1, 300, 9), (2, 40, 4)])
def test_cost_rows_of_small_ranges(ctx, oracle_mod, H, W, D):
    test_cost_rows(ctx, oracle_mod, H, W, D)


# enough tiles for the tiled kernels, ranges on both sides of the line to a thread per entry
@pytest.mark.parametrize("H,W,D,r", [(80, 64, 32, 1), (90, 70, 33, 5), (78, 70, 20, 17), (30, 260, 129, 2), (41, 140, 64, 2),
                                     (80, 70, 9, 3), (80, 70, 1, 4), (77, 65, 33, 0), (79, 66, 12, 8)])
def test_adaptive_weight_routes(ctx, oracle_mod, H, W, D, r):
    O = oracle_mod
    rng = np.random.default_rng(W + r)
    wl, wr = rng.normal(0.5, 0.5, (2, H, W, (2 * r + 1) ** 2)).astype(np.float32)
    cost = rng.normal(0.0, 1.0, (H, W, D)).astype(np.float32)
    assert bits_equal(ctx.calcAWCostL2R(wl, wr, cost, r), O.aw_l2r(wl, wr, cost, r))
    assert bits_equal(ctx.calcAWCostR2L(wl, wr, cost, r), O.aw_r2l(wl, wr, cost, r))


# the smallest and largest tiled windows and their neighbours
@pytest.mark.parametrize("r", [2, 3, 51, 52])
def test_compute_weights_window_limits(ctx, oracle_mod, r):
    test_compute_weights_large_window(ctx, oracle_mod, r)


# images of at least as many 64 x 16 tiles as SMs, and one tile fewer
@pytest.mark.parametrize("H,W", [(16 * 39, 4 * 64 - 3), (16 * 14 + 1, 640)])
@pytest.mark.parametrize("r", [1, 2, 3, 7])
def test_window_filters_of_large_images(ctx, oracle_mod, H, W, r):
    rng = np.random.default_rng(r)
    img = rng.integers(0, 256, (H, W), dtype=np.uint8)
    assert bits_equal(ctx.calculateRankFilt(img, r), oracle_mod.rank(img, r))
    mask = rng.normal(0, 0.2, (2 * r + 1) ** 2).astype(np.float32)
    assert bits_equal(ctx.convolveImage(img, mask, r, r), oracle_mod.convolve(img, mask, r, r))


# both sides of the line between the tiled and the entry's kernel, all tiled radii
@pytest.mark.parametrize("D,r", [(7, 1), (8, 1), (5, 2), (6, 2), (4, 3), (5, 3), (3, 4), (4, 4), (2, 5), (3, 6), (3, 7), (2, 8), (1, 8)])
def test_box_of_small_ranges(ctx, oracle_mod, D, r):
    cost = np.random.default_rng(D * r).normal(0.2, 1.0, (30, 45, D)).astype(np.float32)
    assert bits_equal(ctx.boxAggregate(cost, r), oracle_mod.box(cost, r))
