"""Waves of several samples a pixel take memory for the paths they hold, and
where there is none, or one sample's buffers already hold them, the same images
come out."""
import numpy as np
import pytest

from pfx_b200 import synth
from pfx_b200.trace import Adaptive, SceneBuffers, Trace

pytestmark = pytest.mark.gpu


def free_bytes():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def same(a, b):
    return np.array_equal(a.read_accum().view(np.uint32), b.read_accum().view(np.uint32))


@pytest.mark.parametrize("size,count", [((64, 36), 2), ((64, 36), 64), ((320, 180), 16)])
def test_memory_follows_the_paths(gpu, size, count):
    """At most 1 KB a path of the wave (its buffers are 208 + 56 x slots bytes),
    twice that for the power of two, and 64 MB for graphs and allocation units."""
    w = synth.small("plain_512", size, "sobol")
    trace = Trace(w.scene, w.settings, w.width, w.height)
    trace.sample(1, 1)
    before = free_bytes()
    trace.sample(count, 2)
    assert before - free_bytes() <= 2 * 1024 * size[0] * size[1] * count + (64 << 20)


def test_calls_that_grow(gpu):
    w = synth.small("plain_512", (61, 37), "pcg")
    a, b = (Trace(w.scene, w.settings, w.width, w.height) for _ in range(2))
    a.set_tuning(sort_shading=True)
    for count in (2, 1, 16, 3, 64, 5):
        a.sample(count, 9)
        for _ in range(count):
            b.sample(1, 9)
        assert same(a, b)


def keep_nothing():
    class Keeper:
        def resume(self):
            return None

        def due(self, samples):
            return False

    return Keeper()


@pytest.mark.parametrize("size", [(96, 64), (2100, 2000)])
def test_few_pixels_of_a_film(gpu, size):
    """Late adaptive rounds take several samples of the pixels that are left; the
    larger film's waves fit the buffers of one of its samples (4.2 M paths)."""
    w = synth.small("plain_512", size, "sobol")
    buffers = SceneBuffers(w.scene, w.settings)
    a, b = (Trace(w.scene, w.settings, *size, buffers=buffers) for _ in range(2))
    adaptive = Adaptive(threshold=0.2, min_samples=2, max_samples=24, growth=2.0)
    rounds = a.sample_adaptive(adaptive, 4).rounds
    assert rounds == b.sample_adaptive_kept(adaptive, 4, "key", keep_nothing()).rounds
    assert 0 < rounds[-2].active < size[0] * size[1] // 2
    assert same(a, b)
    before = free_bytes()
    a.sample_adaptive(adaptive, 5)
    assert before - free_bytes() <= 64 << 20


def test_without_room(gpu):
    """With 5 GB left, the quarter that a wave may take does not hold 4 M paths."""
    import torch
    w = synth.small("plain_512", (512, 512), "sobol")
    a, b = (Trace(w.scene, w.settings, 512, 512) for _ in range(2))
    for t in (a, b):
        t.sample(1, 3)
    filler = torch.empty(max(free_bytes() - (5 << 30), 1), dtype=torch.uint8, device="cuda")
    before = free_bytes()
    a.sample(16, 3)
    taken = before - free_bytes()
    a.sample(2, 3)  # a smaller wave fits
    del filler
    torch.cuda.empty_cache()
    assert taken <= 64 << 20
    for _ in range(18):
        b.sample(1, 3)
    assert same(a, b)
