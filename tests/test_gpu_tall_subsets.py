"""Rectangular subsets of at most 16 columns: two windows per warp where a CTA has room for them,
else one.  Either way, and without windows, a POI's record is the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def solve(dic, pr, q, rx, ry, tune=False, **shape):
    with dic.Engine(rx, ry) as e:
        e.set_autotune(tune)
        if shape:
            e.set_launch_shape(dic.Engine.WALK_COLUMN_PX, **shape)
        e.set_ref(pr.ref)
        e.set_tar(pr.tar)
        return e.icgn(q.copy())


def grid(dic, xs, ys):
    return dic.make_queue(*[a.ravel().astype(np.float32) for a in np.meshgrid(xs, ys)])


# two windows per warp fit up to ry = 70 with 8 warps and up to 145 with 4
@pytest.mark.parametrize("rx,ry", [(7, 30), (7, 70), (7, 71), (5, 100), (7, 124), (7, 140), (7, 150)])
def test_tall_subsets(dic, rx, ry):
    from fasticgn_gb300 import speckle
    w, h = 96, 2 * ry + 48
    pr = speckle.pair_bumps(seed=ry, width=w, height=h, max_disp=1.0, max_strain=0.01)
    q = grid(dic, range(rx + 2, w - rx - 2, 5), range(ry + 2, h - ry - 2, 7))
    want = solve(dic, pr, q, rx, ry, warps_per_cta=4, tile=0)
    assert (want["zncc"] >= 0).mean() > 0.5
    for warps in (2, 4, 8):
        if warps == 8 and ry == 150:
            continue                       # eight windows of this height do not fit in a CTA
        for tile in (1, 2) if ry <= 124 else (2,):   # a TMA box has at most 256 rows
            got = solve(dic, pr, q, rx, ry, warps_per_cta=warps, tile=tile)
            np.testing.assert_array_equal(got.view(np.uint8), want.view(np.uint8))


def test_autotune_of_a_tall_subset(dic):
    """The tuner tries eight warps per CTA too."""
    from fasticgn_gb300 import speckle
    pr = speckle.pair_bumps(seed=9, width=128, height=240, max_disp=1.0, max_strain=0.01)
    q = grid(dic, range(9, 119), range(102, 138))
    assert len(q) >= 2048
    want, got = solve(dic, pr, q, 7, 100), solve(dic, pr, q, 7, 100, tune=True)
    np.testing.assert_array_equal(got.view(np.uint8), want.view(np.uint8))
