"""FFTCC of flat windows: constant in both images (the map is zero, the guess stays) or in one (the
map is rounding noise, whose peak the plain order decides)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def plain_seeds(dic, ref, tar, q, r):
    """u, v of the allocation-free entry point's FFTCC: the plain order for 2r = 2 x prime above 32."""
    torch = pytest.importorskip("torch")
    from fasticgn_gb300 import _lib
    h, w = ref.shape
    cfg = _lib.DicConfig(r, r, 0.001, 10, 0, 1.0)
    dt = {np.uint8: _lib.DIC_U8, np.float32: _lib.DIC_F32}[ref.dtype.type]
    dev = [torch.from_numpy(a).cuda() for a in (ref, tar, q.view(np.uint8).copy())]
    err = ctypes.create_string_buffer(256)
    rc = _lib.load().dic_process_pair_noalloc(ctypes.byref(cfg), dev[0].data_ptr(), dev[1].data_ptr(), w, h, dt,
                                              dev[2].data_ptr(), len(q), torch.cuda.current_stream().cuda_stream, err, 256)
    assert rc == _lib.DIC_OK, err.value
    torch.cuda.synchronize()
    return dev[2].cpu().numpy().view(dic.POI_DTYPE)


@pytest.mark.parametrize("dtype,flat_ref,flat_tar", [(np.uint8, 255, 0), (np.float32, 0.1, 0.7)])
@pytest.mark.parametrize("r", [7, 11, 14, 17, 20, 24, 27, 30, 31, 32])
def test_flat_windows(dic, r, dtype, flat_ref, flat_tar):
    rng = np.random.default_rng(r)
    h, w = 2 * r + 36, 9 * r + 60
    ref = rng.integers(0, 255, (h, w)).astype(dtype)
    tar = np.roll(ref, (1, 2), (0, 1))
    a, b = 3 * r + 20, 6 * r + 40
    tar[:, :b] = flat_tar                   # [0, a): both flat, [a, b): the target alone
    ref[:, :a] = flat_ref
    q0 = dic.grid_queue(w, h, r, 3)
    q0["u"], q0["v"] = 1, -1
    q0 = np.tile(q0, 5000 // len(q0) + 1)                       # long enough for the faster kernels
    q0 = np.ascontiguousarray(q0[rng.permutation(len(q0))])     # the three kinds share CTAs and warps
    with dic.Engine(r) as e:
        e.set_ref(ref)
        e.set_tar(tar)
        got = e.fftcc(q0.copy())
        rest = e.fftcc(np.tile(q0[q0["x"] - r > b + 1], 5)).reshape(5, -1)[2]
    x = q0["x"]
    left, mid, right = x + r < a - 2, (x - r >= a) & (x + r < b - 2), x - r > b + 1
    assert min(left.sum(), mid.sum(), right.sum()) > 10
    if dtype == np.uint8:                   # sums exact in any order: the map is zero
        for f, want in (("u", 1), ("v", -1), ("u0", 1), ("v0", -1)):
            assert (got[f][left] == want).all()
        assert np.isnan(got["zncc"][left]).all()
    np.testing.assert_array_equal(got[right].view(np.uint8), rest.view(np.uint8))
    assert ((got["u"] == 2) & (got["v"] == 1))[right].mean() > 0.9
    if r in (17, 31):                       # (where IC-GN ran, u0, v0 are its seed)
        want = plain_seeds(dic, ref, tar, q0, r)
        ran = want["iteration"] > 0
        assert ran[mid].any() or ran[left].any()
        for f, seed in (("u", "u0"), ("v", "v0")):
            np.testing.assert_array_equal(got[f][ran], want[seed][ran])
