"""Gradients of each convolution by itself: a wrong bias row or a dropped tile of
a small layer carries little of the whole vector's norm."""
import numpy as np
import pytest
import torch

from nostrum_pray_gb300 import native
from test_denoise_gpu import CONVS, LEVELS, random_batch, rel

pytestmark = pytest.mark.gpu


def _check_layers(got, want, n, h, w):
    """Per convolution, weights and bias. The tensor cores round every layer's
    output gradient to BF16 (2^-9 / sqrt(3) rms, up to 18 layers: 0.5 %), and a
    stored activation or ReLU sign that rounds the other way weighs the more the
    fewer pixels a level has: 3 % from 1,024 pixels on, 8 % from 32, 25 % below.
    A missing bias row, tap or tile of a level of few pixels is 30 % and more."""
    off = 0
    for i, ((cin, cout), level) in enumerate(zip(CONVS, LEVELS)):
        px = n * (h >> level) * (w >> level)
        tol = 0.03 if px >= 1024 else 0.08 if px >= 32 else 0.25
        nw = cout * 9 * cin
        for what, a, b in (("weights", off, off + nw), ("bias", off + nw, off + nw + cout)):
            assert rel(got[a:b], want[a:b]) < tol, (i, cin, cout, what, rel(got[a:b], want[a:b]))
        off += nw + cout
    assert off == len(got)


@pytest.mark.parametrize("shape", [(1, 16, 16), (1, 16, 48), (3, 48, 32), (2, 80, 48), (1, 144, 208), (2, 256, 256)])
def test_each_convolution_matches_cuda_cores(shape):
    n, h, w = shape
    den = native.Denoiser(seed=11)
    rad, feat, tgt = random_batch(7, n, h, w)
    t = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    got = {}
    for tc in (False, True):
        den.set_tensor_cores(tc)
        got[tc] = den.gradients(t(rad), t(feat), t(tgt))[1]
        den.check()
    _check_layers(got[True], got[False], n, h, w)
