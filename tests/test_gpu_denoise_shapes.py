"""The denoise tile kernel on images of more than two 16 x 16 blocks an SM, the
sizes it takes at every radius, thin ones among them whose taps wrap several
times: against the oracle, and across CTAs that a planted infinity sends to the
per-pixel kernel, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def denoise(rt, ctx, img, sigma, ksigma, threshold=0.1, mix=0.75):
    import torch
    h, w = img.shape[:2]
    d_in = torch.from_numpy(np.ascontiguousarray(img)).cuda()
    d_out = torch.full_like(d_in, 7.0)
    torch.cuda.synchronize()
    rt.denoise_image(ctx, d_in, w, h, d_out, sigma, ksigma, threshold, mix)
    ctx.synchronize()
    return d_out.cpu().numpy()


SHAPES = [(3, 20000), (20000, 3), (1, 5000), (700, 301), (65, 1700)]


@pytest.mark.parametrize("radius", [0, 1, 4, 8])
@pytest.mark.parametrize("w,h", SHAPES)
def test_tiles_match_the_oracle_and_the_per_pixel_kernel(rt, orc, ctx, w, h, radius):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert ((w + 15) // 16) * ((h + 15) // 16) > 2 * sms
    img = np.random.default_rng(w + radius).uniform(0, 1, (h, w, 4)).astype(np.float32)
    sigma, ksigma = (float(radius), 1.0) if radius else (0.4, 0.5)
    plain = denoise(rt, ctx, img, sigma, ksigma)
    want = orc.denoise(img, sigma, ksigma, 0.1, 0.75)
    assert (np.abs(plain.astype(np.float64) - want) / (1.0 + np.abs(want))).max() <= 2e-5
    for y, x in ((0, 0), (h // 2, w // 2), (h - 1, w - 1)):
        bad = img.copy()
        bad[y, x, 1] = np.inf
        got = denoise(rt, ctx, bad, sigma, ksigma)
        near = np.zeros((h, w), bool)  # taps reach radius + 1 texels around
        ys, xs = np.arange(y - radius - 1, y + radius + 2) % h, np.arange(x - radius - 1, x + radius + 2) % w
        near[np.ix_(ys, xs)] = True
        assert np.array_equal(got[~near].view(np.uint32), plain[~near].view(np.uint32))
        assert (~near).any() and not np.isfinite(got[y, x]).all()


@pytest.mark.parametrize("w,h", [(40, 30), (640, 480)])
def test_a_radius_that_is_no_number_has_no_taps(rt, ctx, w, h):
    img = np.random.default_rng(1).uniform(0, 1, (h, w, 4)).astype(np.float32)
    assert np.isnan(denoise(rt, ctx, img, np.inf, 0.0)).all()
