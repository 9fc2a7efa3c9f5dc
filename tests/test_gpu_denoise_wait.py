"""The wait limit bounds a layer's own waits: the set-up of a layer overlaps the
layer before it, whose time the polls do not count."""
import numpy as np
import pytest

from pfx_b200.denoise import Denoiser, write_tza
from test_gpu_denoise import images, random_weights

pytestmark = pytest.mark.gpu


def test_polls_do_not_count_the_layer_before(gpu):
    """Waits of 517 x 391 take about 70 polls in a layer of its own; with the rest
    of the layer before it they took 830."""
    den = Denoiser(write_tza(random_weights(seed=5)))
    color, albedo, normal = images(391, 517, seed=5)
    good = den.denoise(color, albedo, normal)
    den.set_wait_limit(400)
    for _ in range(5):
        assert np.array_equal(den.denoise(color, albedo, normal).view(np.uint32), good.view(np.uint32))
