"""The tiled motion kernels at the sizes where their staging can go wrong, on
smooth textured planes moved by a known shift (no near-ties): tiles that do not
divide the plane, tiles past the staged refinement (per-thread kernels), a
search past the staged coarse pass, planes narrower than a tile, and lines too
long for the row blur's shared memory. Vectors within the 1e-4 px that the FP64
oracle and the float reference agree to; the confidence is a ratio of float
sums over at most tile^2 pixels, 1e-3."""
import numpy as np
import pytest

from oracle import hvd_oracle as O

pytestmark = pytest.mark.gpu


def _planes(h, w, dy, dx, seed):
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:h + 24, 0:w + 24].astype(np.float64)
    p = np.zeros_like(y)
    for _ in range(14):
        fy, fx = rng.uniform(-0.25, 0.25, 2)
        p += rng.uniform(2, 6) * np.cos(2 * np.pi * (fy * y + fx * x) + rng.uniform(0, 6.3))
    a = p[12:12 + h, 12:12 + w]
    b = p[12 + dy:12 + dy + h, 12 + dx:12 + dx + w]
    return (50 + a).astype(np.float32), (50 + b).astype(np.float32)


@pytest.mark.parametrize("h,w,tile,search", [
    (97, 131, 32, 16),     # remainders in both directions
    (64, 64, 16, 8),       # no remainder, smallest coarse tile
    (75, 203, 24, 11),
    (140, 150, 64, 16),    # the largest staged tile
    (150, 170, 72, 16),    # past it
    (120, 130, 32, 24),    # a search past the staged coarse pass
    (20, 300, 32, 6),      # shorter than a tile
    (16, 26000, 32, 4),    # rows past shared memory
])
def test_float_motion_matches_oracle(ctx, h, w, tile, search):
    a, b = _planes(h, w, 2, -3, h * w)
    dy, dx, cf = ctx.estimate_motion(a, b, tile=tile, search=search)
    oy, ox, oc = O.estimate_motion(a, b, tile=tile, search=search)
    assert np.abs(dy - oy).max() <= 1e-4 and np.abs(dx - ox).max() <= 1e-4
    assert np.abs(cf - oc).max() <= 1e-3


@pytest.mark.parametrize("h,w,tile", [(97, 131, 32), (40, 70, 48), (33, 65, 33)])
def test_verify_motion_matches_full_sums(ctx, h, w, tile):
    """The prediction wins exactly where its sum over the blurred planes is the
    smaller one."""
    a, b = _planes(h, w, 2, -3, 5)
    th, tw = -(-h // tile), -(-w // tile)
    rng = np.random.default_rng(1)
    pdy = rng.choice([-2.0, 0.4, 3.0], (th, tw)).astype(np.float32)
    pdx = rng.choice([3.0, -1.0], (th, tw)).astype(np.float32)
    dy, dx, _ = ctx.verify_motion(a, b, pdy, pdx, tile=tile)
    A, B = O.box_blur_same(b, 2), O.box_blur_same(a, 2)

    def ssd(ty, tx, sy, sx):
        y = np.arange(ty * tile, min((ty + 1) * tile, h))
        x = np.arange(tx * tile, min((tx + 1) * tile, w))
        r = B[np.clip(y - sy, 0, h - 1)][:, np.clip(x - sx, 0, w - 1)]
        return float(((A[y][:, x] - r) ** 2).sum())

    for ty in range(th):
        for tx in range(tw):
            p = (pdy[ty, tx], pdx[ty, tx])
            won = ssd(ty, tx, int(np.round(p[0])), int(np.round(p[1]))) < ssd(ty, tx, 0, 0)
            want = p if won else (0.0, 0.0)
            assert (dy[ty, tx], dx[ty, tx]) == want, (ty, tx)
