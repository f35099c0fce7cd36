"""The pixel-sampled IC-GN's row loops against its general loop.

A staged window whose samples are all covered runs px_column_rows (four rows a group, support
pixels kept from row to row and reloaded where a lane's warp crosses a pixel boundary) or, from a
whole-pixel seed, px_column_lattice; without a window every sample goes through the tested
general loop.  Both read the same floats in the same order, so the records are the same bytes.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [260, 263])           # TMA on the plane itself, and on its padded copy
@pytest.mark.parametrize("radius", [1, 2, 3, 7, 8, 14, 15, 16, 17, 30, 31])   # last groups of one and three rows
def test_row_loops_equal_the_general_loop(dic, radius, width):
    from fasticgn_gb300 import speckle
    pr = speckle.pair_bumps(seed=300 + radius, width=width, height=220, max_disp=4.0, max_strain=0.02)
    rng = np.random.default_rng(radius)
    q0 = dic.grid_queue(width, 220, radius, 3 if radius < 16 else 7)
    q0["u"], q0["v"] = rng.uniform(-3, 3, (2, len(q0)))
    for f in ("ux", "uy", "vx", "vy"):                  # up to a pixel boundary crossed every few rows
        q0[f] = rng.uniform(-0.08, 0.08, len(q0))
    whole = rng.random(len(q0)) < 0.4                   # these start on the pixel lattice
    for f in ("u", "v"):
        q0[f][whole] = np.rint(q0[f][whole])
    for f in ("ux", "uy", "vx", "vy"):
        q0[f][whole] = 0
    walk = dic.Engine.WALK_COLUMN_PX if radius <= 15 else dic.Engine.WALK_PAIR_PX
    got = []
    for tile in (0, 1, 2):
        with dic.Engine(radius) as e:
            e.set_launch_shape(walk, warps_per_cta=2, tile=tile, warps_per_poi=1 if radius <= 15 else 2)
            e.set_ref(pr.ref)
            e.set_tar(pr.tar)
            got.append(e.icgn(q0.copy()))
    for q in got[1:]:
        np.testing.assert_array_equal(q.view(np.uint8), got[0].view(np.uint8))
    if radius >= 7:
        assert (got[0]["zncc"] >= 0).mean() > 0.2


@pytest.mark.parametrize("radius,drop", [(1, 0), (2, 1), (5, 0), (7, 0), (7, 1)])
def test_two_pois_per_warp_equal_one(dic, radius, drop):
    """Subsets of at most 16 columns: two POIs per warp for a queue, one per warp in a batch.  An
    odd queue leaves its last warp with one; rejected and unconverged POIs share warps with solved
    ones."""
    from fasticgn_gb300 import speckle
    pr = speckle.pair_bumps(seed=400 + radius, width=232, height=200, max_disp=3.0, max_strain=0.03)
    q = dic.grid_queue(232, 200, radius, 3)
    q = np.ascontiguousarray(q[:len(q) - (len(q) + drop + 1) % 2])     # odd (drop 0) or even
    assert len(q) % 2 == 1 - drop
    rng = np.random.default_rng(radius)
    far = rng.random(len(q)) < 0.1
    q["x"][far] += rng.integers(-40, 40, far.sum())                     # some subsets leave the image
    q["zncc"][rng.random(len(q)) < 0.05] = -3
    want, got = q.copy(), q.copy()
    with dic.Engine(radius) as e:
        e.batch_process([(pr.ref, pr.tar, radius, want)])
    with dic.Engine(radius) as e:
        e.set_ref(pr.ref)
        e.set_tar(pr.tar)
        e.process_pair(got)
    np.testing.assert_array_equal(got.view(np.uint8), want.view(np.uint8))
