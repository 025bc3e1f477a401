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
