"""FFTCC by queue length: a short queue takes the plain order of operations alone, a long one the
faster kernels, which leave near ties to that order.  Ties and flat windows get the same bytes
either way, every other POI the same peak."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# every length with two forms; short: POIs that 2 (prime factors above 5) or 4 per SM allow
RADII = [7, 11, 14, 18, 20, 21, 22, 24, 25, 26, 27, 28, 30, 32]


def scene(r):
    """Tied, flat and textured areas, and POIs whose windows leave the image."""
    rng = np.random.default_rng(r)
    h, w = 2 * r + 40, 8 * r + 90
    period = next(p for p in range(4, 2 * r + 1) if (2 * r) % p == 0)
    ref = rng.integers(0, 255, (h, w)).astype(np.uint8)
    tiles = np.tile(rng.integers(0, 255, (period, period)), (h // period + 1, w // period + 1))
    a = 3 * r + 40
    ref[:, :a] = tiles[:h, :a]                                     # every shift by the period ties
    tar = np.roll(ref, (1, 2), (0, 1))
    tar[:, a:] = np.clip(tar[:, a:] + rng.normal(0, 3, (h, w - a)), 0, 255)
    tar[: h // 2, a + r:a + 3 * r + 20] = 200                      # flat target
    ys, xs = np.meshgrid(np.arange(r + 2, h - r - 2, 3), np.arange(r - 2, w - r + 2, 3), indexing="ij")
    return ref, tar, xs.ravel().astype(np.float32), ys.ravel().astype(np.float32)


@pytest.mark.parametrize("r", RADII)
def test_short_and_long_queues_agree(dic, r):
    ref, tar, xs, ys = scene(r)
    keep = np.random.default_rng(0).permutation(len(xs))[:299]     # odd: a last CTA that is not full
    q0 = dic.make_queue(xs[keep], ys[keep])
    q0["u"], q0["zncc"] = -1, 0.5
    with dic.Engine(r) as e:
        e.set_ref(ref)
        e.set_tar(tar)
        short = e.fftcc(q0.copy())
        long = e.fftcc(np.tile(q0, 17)).reshape(17, -1)
    for copy in long[1:]:                                          # other neighbours in the CTA, same bytes
        np.testing.assert_array_equal(copy.view(np.uint8), long[0].view(np.uint8))
    long = long[0]
    for f in ("x", "y", "u", "v", "u0", "v0"):
        np.testing.assert_array_equal(long[f], short[f])
    out = short["zncc"] == 0.5                                     # left untouched
    assert out.any() and (~out).sum() > 100
    np.testing.assert_array_equal(long[out].view(np.uint8), short[out].view(np.uint8))
    tied = ~out & (short["x"] + r < 3 * r + 36) & (short["x"] >= r + 4)
    assert tied.sum() > 10
    np.testing.assert_array_equal(long[tied].view(np.uint8), short[tied].view(np.uint8))
    # values that moved by half the margin of a near tie, 1e-5 (rn + tn) / 2 M^2, could pass each other
    for p, z in zip(short[~out], long["zncc"][~out]):
        x, y = int(p["x"]), int(p["y"])
        rn, tn = (float(im[y - r:y + r, i - r:i + r].astype(np.float64).var()) for im, i in ((ref, x), (tar, x - 1)))
        if rn > 0 and tn > 0:
            assert abs(float(z) - float(p["zncc"])) <= 5e-6 * (rn + tn) / 2 / np.sqrt(rn * tn)


@pytest.mark.parametrize("r", [8, 15, 19, 23, 29])
def test_other_lengths_match_the_oracle(dic, oracle_mod, r):
    """Lengths that the radii of the oracle test leave out, among them 2 x prime ones with 5, 2 and
    1 POIs per CTA; out-of-range POIs share CTAs with valid ones."""
    O = oracle_mod
    from fasticgn_gb300 import speckle
    from test_gpu_parity import check_fftcc, to_oracle
    pr = speckle.pair_affine(seed=r, width=256, height=224)
    q = dic.grid_queue(256, 224, r, 7)
    q["u"], q["v"] = -3.0, 1.0
    q["u"][::7] = 300.0                                            # these target windows leave the image
    q = np.ascontiguousarray(q[:len(q) - (len(q) + 1) % 2])
    oq = to_oracle(O, q)
    with dic.Engine(r) as e:
        e.set_ref(pr.ref)
        e.set_tar(pr.tar)
        before = q.copy()
        e.fftcc(q)
    out = before["u"] == 300
    np.testing.assert_array_equal(q[out].view(np.uint8), before[out].view(np.uint8))
    ref, tar = pr.ref.astype(np.float32), pr.tar.astype(np.float32)
    O.fftcc2d(ref, tar, oq, r)
    check_fftcc(O, ref, tar, r, q[~out], oq[~out])


@pytest.mark.parametrize("r", [14, 17, 20, 27, 31, 32])
def test_maps_beyond_float_range(dic, r):
    """Pixels so large that the peak, and with it the margin of a near tie, is infinite: still the
    plain order's peak, in short and in long queues."""
    m = 2 * r
    rng = np.random.default_rng(r)
    h, w = 4 * r + 30, 4 * r + 40
    # peak of a perfect match: m^4 var, 2.5 times beyond the range; the rest of the map stays within
    ref = (rng.normal(size=(h, w)) * np.sqrt(2.5 * 3.4e38) / m ** 2).astype(np.float32)
    tar = np.roll(ref, (1, 2), (0, 1))
    q0 = dic.grid_queue(w, h, r, 4)[:299]
    with dic.Engine(r) as e:
        e.set_ref(ref)
        e.set_tar(tar)
        short, long = e.fftcc(q0.copy()), e.fftcc(np.tile(q0, 5100 // len(q0) + 1))[:len(q0)]
    for f in ("u", "v"):
        np.testing.assert_array_equal(long[f], short[f])
    assert ((long["u"] == 2) & (long["v"] == 1)).all()


@pytest.mark.parametrize("r", [20, 24, 28, 30, 32])
def test_zncc_error_is_the_plain_orders(dic, r):
    """Rms distance of zncc from 64 bits: the long queue's form within 5 % of the plain order's."""
    rng = np.random.default_rng(5)
    h, w = 260, 420
    ref = rng.normal(size=(h, w))
    for _ in range(3):
        ref = (ref + np.roll(ref, 1, 0) + np.roll(ref, 1, 1)) / 3
    ref = 128 + 50 * ref / ref.std()
    a, b = (np.clip(np.rint(im + rng.normal(0, 2, (h, w))), 0, 255).astype(np.uint8)
            for im in (ref, np.roll(ref, (1, 2), (0, 1))))
    q0 = dic.grid_queue(w, h, r, 4)
    q0 = np.ascontiguousarray(q0[:: max(1, len(q0) // 1500)])
    with dic.Engine(r) as e:
        e.set_ref(a)
        e.set_tar(b)
        plain = np.concatenate([e.fftcc(q0[k:k + 299].copy()) for k in range(0, len(q0), 299)])
        long = e.fftcc(np.tile(q0, 2000 // len(q0) + 1))[:len(q0)]
    exact = []
    for p in q0:
        x, y = int(p["x"]), int(p["y"])
        f, g = (im[y - r:y + r, x - r:x + r].astype(np.float64) for im in (a, b))
        f, g = f - f.mean(), g - g.mean()
        c = np.fft.irfft2(np.conj(np.fft.rfft2(f)) * np.fft.rfft2(g), s=f.shape)
        exact.append(c.max() / np.sqrt((f * f).sum() * (g * g).sum()))
    rms = [float(np.sqrt(np.mean((q["zncc"] - np.array(exact)) ** 2))) for q in (plain, long)]
    assert rms[1] <= 1.05 * rms[0], rms
