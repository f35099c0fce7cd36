"""Two POIs per warp (subsets of at most 16 columns): a window copy that never arrives, in both
halves of a warp or with one half without a POI, ends in the bounded wait as for one POI."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius,count", [(7, 200), (7, 201), (5, 1)])
def test_window_timeout_of_a_half_is_reported(dic, monkeypatch, radius, count):
    from fasticgn_gb300 import _lib, speckle
    pr = speckle.pair_bumps(seed=9, width=192, height=160, max_disp=3.0, max_strain=0.01)
    q0 = dic.grid_queue(192, 160, radius, 8)[:count]
    assert len(q0) == count

    def solve(e):
        e.set_ref(pr.ref)
        e.set_tar(pr.tar)
        return e.process_pair(q0.copy())

    with dic.Engine(radius) as e:
        want = solve(e)
    monkeypatch.setenv("DIC_TEST_WAIT_FAULT", "1")      # arms the wait and skips the copy
    e = dic.Engine(radius)
    monkeypatch.delenv("DIC_TEST_WAIT_FAULT")
    with pytest.raises(_lib.DicError) as info:
        solve(e)
    assert info.value.code == _lib.DIC_ERR_CUDA and "TMA tile copy" in str(info.value)
    e.close()
    with dic.Engine(radius) as e:
        np.testing.assert_array_equal(solve(e).view(np.uint8), want.view(np.uint8))
