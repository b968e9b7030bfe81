"""The lanes of the differentiable kernels (32 / spp pixels to a warp, chunks
of 32 samples) and the replay record of the adjoint's first 8 vertices.

Samples are independent, so the image and the gradients at spp samples are the
means of those at one sample each.  Sizes: sample counts around the warp's 32
and its divisors, images whose pixels do not fill the last warp, depths within
and past the record.  Each float term is the same on both sides; only sums of
at most 40 terms differ in rounding, 40 x 2^-24 = 2.4e-6 of the sum of their
magnitudes, and terms have one sign in the image; the gradients' terms cancel
in part, so they are held to 1e-4 of the gradient vector's length."""
import numpy as np
import pytest

import wfpt
from wfpt import diff, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spp,depth,size", [(1, 3, (5, 3)), (3, 10, (7, 5)), (8, 4, (9, 7)), (16, 10, (4, 3)),
                                            (17, 3, (3, 3)), (31, 4, (5, 2)), (32, 9, (3, 2)), (33, 4, (3, 3)),
                                            (40, 12, (2, 1))])
def test_samples_average(cuda, spp, depth, size):
    torch = cuda
    w, h = size
    scene, cam, n, _ = scenes.cornell_inverse(w, h, cells=4)
    a, r = (torch.from_numpy(x).cuda() for x in scenes.inverse_parameters(scene, n, seed=9))
    dev = wfpt.DeviceScene(scene)
    g = torch.Generator(device="cuda").manual_seed(spp)
    d_image = torch.randn(h, w, 3, device="cuda", generator=g)
    d_image[0, 0] = 0.0

    def both(samples, start, weight):
        cfg = diff.diff_config(w, h, samples, depth, n, sample_start=start)
        img = diff.forward(dev, cam, cfg, a, r, 1.3)
        grads = diff.backward(dev, cam, cfg, a, r, 1.3, d_image * weight)
        return img.double().cpu().numpy(), np.concatenate([x.cpu().numpy().ravel() for x in grads])

    image, grads = both(spp, 5, 1.0)
    parts = [both(1, 5 + k, 1.0 / spp) for k in range(spp)]
    want = sum(p[0] for p in parts) / spp
    assert np.abs(image - want).max() <= 2.4e-6 * np.abs(want).max() + 1e-12
    want = sum(p[1] for p in parts)
    assert np.linalg.norm(want) > 0
    assert np.linalg.norm(grads - want) <= 1e-4 * np.linalg.norm(want)
    dev.close()


@pytest.mark.parametrize("spp,pixels", [(1, 32), (1, 7), (8, 4), (3, 10), (32, 2)])
def test_pixels_meet_in_double(cuda, spp, pixels):
    """Gradients are sums of float terms of the single pixels, added in
    double.  A pixel's terms do not depend on the other pixels' adjoints, so
    the gradient of a large adjoint (2^24) at one pixel and small ones at its
    neighbours in the warp is the sum of the two gradients.  In double the
    sums lose at most spp x pixels x depth = 128 times 2^-53 of the large
    terms, which may be some 2^6 of their sum: 2^-40 of it.  A float sum across
    pixels would lose 2^-24 of it, as much as the small ones' terms are.
    Samples of one pixel always have the same adjoint here, so how they meet
    is not what is tested."""
    torch = cuda
    scene, cam, n, _ = scenes.cornell_inverse(256, 256, cells=1)  # few large triangles: one for many lanes
    a, r = (torch.from_numpy(x).cuda() for x in scenes.inverse_parameters(scene, n, seed=9))
    dev = wfpt.DeviceScene(scene)
    depth = 4
    cfg = diff.diff_config(256, 256, spp, depth, n, sample_start=5, crop=(100, 200, pixels, 1))
    small = torch.zeros(256, 256, 3, device="cuda")
    small[200, 100:100 + pixels] = 1.0
    small[200, 100] = 0.0
    large = torch.zeros(256, 256, 3, device="cuda")
    large[200, 100] = 2.0 ** 24

    def gradient(adjoint):
        return np.concatenate([x.double().cpu().numpy().ravel()
                               for x in diff.backward(dev, cam, cfg, a, r, 1.0, adjoint)])

    g_small, g_large, g_both = gradient(small), gradient(large), gradient(small + large)
    bound = 2.0 ** -40 * np.abs(g_large).max()
    assert np.abs(g_small).max() > 1e3 * bound
    assert np.abs(g_both - (g_large + g_small)).max() <= bound
    dev.close()
