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
