"""Other calls on an engine between the frames of a sequence: a longer queue, a larger layout and
another pixel type move buffers that a captured frame names, so the next frame is captured again
and equals the eager one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# the FFTCC in the plain order (7; 20 with 396 POIs), without near ties (10) and with their list
@pytest.mark.parametrize("radius,step", [(7, 6), (10, 6), (20, 6), (20, 9)])
def test_calls_between_frames(dic, radius, step):
    from fasticgn_gb300 import speckle
    pr = speckle.pair_bumps(seed=radius, width=240, height=200, max_disp=2.0, max_strain=0.01)
    ref = pr.ref.copy()
    ref[:, :80] = np.tile(np.random.default_rng(3).integers(0, 255, (2, 2)), (100, 40))   # every shift ties
    jump = np.roll(ref, (radius // 2, radius - 2), (0, 1))             # the whole frame is solved again
    frames = [pr.tar, ref, pr.tar, jump, pr.tar.astype(np.float32), jump.astype(np.float32)]
    tmpl = dic.grid_queue(240, 200, radius, step)
    more = dic.grid_queue(240, 200, radius, 2)
    runs = []
    for graphs in (True, False):
        with dic.Engine(radius) as e:
            e.set_graphs(graphs)
            e.set_ref(ref)
            e.sequence_begin(tmpl)
            seq = []
            for k, tar in enumerate(frames):
                res = np.zeros_like(tmpl)
                rep = e.sequence_frame(tar, res)
                seq.append((res.tobytes(), rep["frame_fallback_used"], rep["repaired_recovered"]))
                if k == 2:
                    e.fftcc(more.copy())
                    e.prepare_ref(more)
                    e.prepare_ref(tmpl)
            runs.append(seq)
    assert runs[0] == runs[1]
    assert any(used for _, used, _ in runs[0])
