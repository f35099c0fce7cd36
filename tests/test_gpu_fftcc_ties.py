"""Near ties of the correlation peak: the faster FFTCC kernels leave them to a second pass in the
plain order, so a map with equal peaks gives one of them and two runs give the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def correlation(ref, tar, x, y, r):
    """The POI's circular correlation map in 64 bits, divided by a perfect match's value."""
    f, g = (im[y - r:y + r, x - r:x + r].astype(np.float64) for im in (ref, tar))
    f, g = f - f.mean(), g - g.mean()
    c = np.fft.ifft2(np.conj(np.fft.fft2(f)) * np.fft.fft2(g)).real
    return c / np.sqrt((f * f).sum() * (g * g).sum())


# one length per kernel: a prime factor above 5 in k_fftcc2, k_fftcc_line with its looped and
# unrolled stages (2 x prime, coprime pairs, 64), POIs per CTA of 8, 4, 2 and 1
@pytest.mark.parametrize("r", [7, 11, 17, 20, 24, 27, 30, 31, 32])
def test_peaks_of_maps_with_ties(dic, r):
    rng = np.random.default_rng(r)
    period = next(p for p in range(4, 2 * r + 1) if (2 * r) % p == 0)
    tile = rng.integers(0, 255, (period, period)).astype(np.float32)
    h, w = 4 * r + 40, 4 * r + 72
    ref = np.tile(tile, (h // period + 1, w // period + 1))[:h, :w].copy()   # every shift by the period ties
    tar = np.roll(ref, (1, 2), (0, 1))
    half = ref[:, w // 2:]
    ref[:, w // 2:] = rng.integers(0, 255, half.shape)                        # textured: no ties
    tar[:, w // 2:] = np.roll(ref[:, w // 2:], (-1, 1), (0, 1))
    tar[: h // 3, w // 2 + 3 * w // 8:] = 77                                  # flat target, textured reference
    q0 = dic.grid_queue(w, h, r, 3)
    runs = []
    for _ in range(2):
        with dic.Engine(r) as e:
            e.set_ref(ref.astype(np.uint8))
            e.set_tar(tar.astype(np.uint8))
            runs.append(e.fftcc(q0.copy()))
    np.testing.assert_array_equal(runs[0].view(np.uint8), runs[1].view(np.uint8))
    ties = 0
    for p in runs[0][:: max(1, len(q0) // 150)]:
        x, y = int(p["x"]), int(p["y"])
        if tar[y - r:y + r, x - r:x + r].std() < 1:
            continue
        c = correlation(ref, tar, x, y, r)
        got = c[int(p["v"]) % (2 * r), int(p["u"]) % (2 * r)]
        # FP32 rounding of a map is below 1e-5 of a perfect match
        assert got >= c.max() - 2e-5 and abs(p["zncc"] - c.max()) <= 2e-5
        ties += (c >= c.max() - 1e-6).sum() > 1
    assert ties > 0
