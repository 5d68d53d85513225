"""The shared-memory denoise kernel (radius up to 8, images of some hundred
16 x 16 blocks up) against the per-pixel one, which takes over in CTAs that see a texel that is not finite: planted
infinities switch 32 x 16 pixel blocks from one to the other, and every pixel
whose taps do not meet one keeps its value bit for bit."""
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


@pytest.mark.parametrize("radius", [0, 1, 2, 3, 4, 5, 7, 8])
@pytest.mark.parametrize("w,h", [(96, 80), (31, 17), (400, 223), (351, 229), (33, 1700), (1703, 31)])
def test_tile_kernel_equals_per_pixel(rt, ctx, w, h, radius):
    img = np.random.default_rng(w + radius).uniform(0, 2, (h, w, 4)).astype(np.float32)
    img[::7, ::5] = -0.0
    sigma, ksigma = (float(radius), 1.0) if radius else (0.4, 0.5)
    plain = denoise(rt, ctx, img, sigma, ksigma)
    assert np.isfinite(plain).all()
    switched = np.zeros((h, w), bool)
    for y, x in ((0, 0), (h // 2, w // 2), (h - 1, w - 1), (h // 3, w - 1)):
        bad = img.copy()
        bad[y, x, 2] = np.inf
        got = denoise(rt, ctx, bad, sigma, ksigma)
        # Taps reach radius + 1 texels around, wrapping at the edges.
        near = np.zeros((h, w), bool)
        for dy in range(-radius - 1, radius + 2):
            for dx in range(-radius - 1, radius + 2):
                near[(y + dy) % h, (x + dx) % w] = True
        assert np.array_equal(got[~near].view(np.uint32), plain[~near].view(np.uint32))
        assert not np.isfinite(got[y, x]).all()
        switched |= ~near
    assert switched.any()


@pytest.mark.parametrize("w,h", [(1, 1), (3, 2), (33, 5), (64, 33)])
@pytest.mark.parametrize("radius", [2, 8, 9])
def test_small_images_match_oracle(rt, orc, ctx, w, h, radius):
    # Images smaller than the kernel wrap several times.
    img = np.random.default_rng(w * h).uniform(0, 1, (h, w, 4)).astype(np.float32)
    got = denoise(rt, ctx, img, float(radius), 1.0)
    want = orc.denoise(img, float(radius), 1.0, 0.1, 0.75)
    assert (np.abs(got.astype(np.float64) - want) / (1.0 + np.abs(want))).max() <= 2e-5


@pytest.mark.parametrize("radius", [1, 4, 8, 9])
@pytest.mark.parametrize("w,h", [(256, 144), (256, 160), (256, 304), (256, 320), (271, 305)])
def test_sizes_around_the_rule_match_oracle(rt, orc, ctx, w, h, radius):
    img = np.random.default_rng(w * h).uniform(0, 1, (h, w, 4)).astype(np.float32)
    got = denoise(rt, ctx, img, float(radius), 1.0)
    want = orc.denoise(img, float(radius), 1.0, 0.1, 0.75)
    assert (np.abs(got.astype(np.float64) - want) / (1.0 + np.abs(want))).max() <= 2e-5
