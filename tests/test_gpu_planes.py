"""Planes at sizes around the preparation kernels' tiles (64 x 16 reference pixels, 128 x 4 target
pixels) equal the CPU's bit for bit, the target's without its table (pixel sampling)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height", [(5, 5), (63, 15), (64, 16), (65, 17), (127, 6), (128, 33), (129, 18), (259, 50)])
@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.float32])
def test_planes_at_tile_edges(dic, oracle_mod, dtype, width, height):
    rng = np.random.default_rng(width)
    top = {np.uint8: 255, np.uint16: 4095, np.float32: 300}[dtype]
    ref, tar = (rng.uniform(0, top, (2, height, width))).astype(dtype)
    with dic.Engine(7) as e:
        e.set_ref(ref)
        e.set_tar(tar)
        tarf = e.read_plane(dic._lib.DIC_PLANE_TAR, width, height)
        reff = e.read_plane(dic._lib.DIC_PLANE_REF, width, height)
        pack = e.read_plane(dic._lib.DIC_PLANE_REF_PACK, width, height)
    gx, gy = oracle_mod.gradient(ref.astype(np.float32))
    assert np.array_equal(tarf, tar.astype(np.float32))
    assert np.array_equal(reff, ref.astype(np.float32))
    assert np.array_equal(pack, np.stack([ref.astype(np.float32), gx, gy, np.zeros_like(gx)], -1))
