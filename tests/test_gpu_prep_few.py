"""Short queues take eight POIs per CTA in the per-POI prep, a batch's jobs and queues above 96
POIs per SM 32: the same queue as a pair and as a batch gives the same bytes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius", [7, 15, 20, 32])     # shared columns (column, pair walk), per POI (flat walk)
@pytest.mark.parametrize("count", [1, 8, 9, 31, 1000, None, "line"])
def test_few_pois_per_cta_equal_32(dic, radius, count):
    import torch
    from fasticgn_gb300 import speckle
    line = 96 * torch.cuda.get_device_properties(0).multi_processor_count
    size = 448 if count in (None, "line") else 260
    pr = speckle.pair_bumps(seed=700 + radius, width=size, height=size - 20, max_disp=4.0, max_strain=0.01)
    q = dic.grid_queue(size, size - 20, radius, 3 if size == 448 else 5)
    if size == 448:                                      # the last short queue and the first long one
        q = np.resize(q, line + (count is None))
    else:
        q = q[:count]
    q = np.ascontiguousarray(q)
    q["x"][::13] -= 3 * radius                           # some subsets leave the image
    want, got = q.copy(), q.copy()
    with dic.Engine(radius) as e:
        e.batch_process([(pr.ref, pr.tar, radius, want)])
    with dic.Engine(radius) as e:
        e.set_ref(pr.ref)
        e.set_tar(pr.tar)
        e.process_pair(got)
    assert got.tobytes() == want.tobytes()
