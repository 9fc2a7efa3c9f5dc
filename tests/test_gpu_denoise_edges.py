"""The denoiser at the edges of its convolution tiles (126 pixels by 2, 4 or 8
rows) on every level of the U-Net, against the FP64 oracle."""
import numpy as np
import pytest

from oracle import denoise as D
from pfx_b200.denoise import Denoiser, write_tza
from test_gpu_denoise import TOL, gap, images, random_weights

pytestmark = pytest.mark.gpu


# widths whose padded tile ends just before, at and just after a tile's 126 pixels on levels 0, 1 and 2
@pytest.mark.parametrize("h,w", [(16, 112), (17, 126), (33, 128), (24, 252), (16, 256), (40, 272), (130, 16), (16, 512)])
def test_tile_edges(gpu, h, w):
    blob = write_tza(random_weights(seed=h + w))
    den = Denoiser(blob)
    color, albedo, normal = images(h, w, seed=w)
    out = den.denoise(color, albedo, normal)
    want = D.denoise(color, albedo, normal, D.build_net(D.parse_tza(blob)))
    assert gap(out, want) <= TOL, gap(out, want)
    assert np.array_equal(out.view(np.uint32), den.denoise(color, albedo, normal).view(np.uint32))

