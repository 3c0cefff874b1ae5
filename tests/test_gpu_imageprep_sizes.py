"""The preparation's transforms over the box sizes: the smallest, one of each radix mix of the one-CTA path
(up to 128), and both ends and the odd radices of the two-pass path (144 .. 512), with the noise background
(which runs every kernel of a path), an odd batch and a window of less than the box.  Oracle, checks and
tolerances of test_gpu_imageprep.  The noise spectrum is that of the images' own noise, 0.49 / N^2 a
coefficient: the masked and the unmasked image are transformed as one complex sequence, so each is exact to
FP32 rounding of the larger of the two (noise of variance 1 a coefficient, N times the image's, leaves the
unmasked image 3e-5 at 500, with these transforms and with block-wide ones)."""
import numpy as np
import pytest

import imageprep_oracle as ipo
from test_gpu_imageprep import _check, _images
from test_imageprep_oracle import base_cfg, params

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(t2b):
    es = t2b.EStep(0)
    yield es
    es.close()


@pytest.mark.parametrize("N", [8, 12, 54, 90, 108, 128, 144, 150, 162, 270, 384, 486, 500, 512])
def test_prep_sizes(ctx, N):
    rng = np.random.default_rng(N)
    s = max(4, N // 3 * 2 // 2 * 2)
    cfg = base_cfg(N, s, sigma2_noise=0.49 / N ** 2 * (0.3 + np.linspace(1.0, 0.05, N // 2 + 1) ** 2), zero_mask=0, mask_radius=0.4 * N,
                   width_mask_edge=min(5.0, 0.1 * N))
    imgs = _images(N, 3, rng)
    par = params(3, rng, offset=2.0)
    pid = np.arange(3, dtype=np.int64) * 37 + 5
    ctx.configure_prep(max_batch=3, **cfg)
    _check(ctx.prepare_images(imgs, par, pid), ipo.prepare(imgs.astype(np.float64), par, pid, cfg), N, s, cfg)
