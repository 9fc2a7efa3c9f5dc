"""Several samples of a pixel in one wave: the accumulation and the films equal
those of the same samples taken one call at a time, bit for bit, whatever the
sample count, the launch choices, the mask and the converged pixels."""
import numpy as np
import pytest

from pfx_b200 import synth
from pfx_b200.trace import Adaptive, Trace

pytestmark = pytest.mark.gpu


def images(t):
    out = t.readback()
    return [t.read_accum(), out.color, out.albedo, out.normal]


def same(a, b):
    return all(np.array_equal(x.view(np.uint32), y.view(np.uint32)) for x, y in zip(images(a), images(b)))


@pytest.mark.parametrize("sampler", ["sobol", "pcg"])
@pytest.mark.parametrize("count", [2, 3, 7, 16, 21])
def test_one_call_equals_single_samples(gpu, sampler, count):
    w = synth.small("instanced_1080", (61, 37), sampler)
    a, b = (Trace(w.scene, w.settings, w.width, w.height) for _ in range(2))
    a.sample(count, 5)
    a.sample(count, 6)
    for seed in (5, 6):
        for _ in range(count):
            b.sample(1, seed)
    # a sample's index counts on from the samples before it, whichever call took them
    assert a.samples() == b.samples() == 2 * count
    assert same(a, b)
    assert a.rays_traced() == b.rays_traced()


@pytest.mark.parametrize("choice", [{"split_shade": False}, {"shadow_queue": False}, {"slot_kernels": False},
                                    {"sort_rays": True}, {"graphs": False, "sort_shading": False}])
def test_launch_choices(gpu, choice):
    w = synth.small("plain_512", (48, 33), "sobol")
    a, b = (Trace(w.scene, w.settings, w.width, w.height) for _ in range(2))
    a.set_tuning(**choice)
    a.sample(6, 3)
    for _ in range(6):
        b.sample(1, 3)
    assert same(a, b)


def test_mask_and_converged_pixels(gpu):
    w = synth.small("plain_512", (64, 48), "pcg")
    a, b = (Trace(w.scene, w.settings, w.width, w.height) for _ in range(2))
    mask = np.random.default_rng(1).random((48, 64)) < 0.3
    for t in (a, b):
        t.set_pixel_mask(mask)
    a.sample(9, 2)
    for _ in range(9):
        b.sample(1, 2)
    assert same(a, b)
    for t in (a, b):
        t.set_pixel_mask(None)
    # adaptive: a keeper makes the second one take its samples one at a time

    class Keeper:
        def resume(self):
            return None

        def due(self, samples):
            return False

        def keep(self, data):
            raise AssertionError("never due")

    adaptive = Adaptive(threshold=0.05, min_samples=4, max_samples=40, growth=1.5)
    rounds = a.sample_adaptive(adaptive, 4).rounds
    kept = b.sample_adaptive_kept(adaptive, 4, "key", Keeper()).rounds
    assert rounds == kept and len(rounds) > 3 and 0 < rounds[-2].active < 64 * 48
    assert same(a, b)
