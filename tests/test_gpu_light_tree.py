"""The light tree's descent on its own rows against the descent that reads the
reference's rows (the one-kernel light slots): the same images bit for bit over
tree sizes, point and spot lights, bulb radii from zero up and ranges that cut
lights off."""
import numpy as np
import pytest

from pfx_b200 import synth
from pfx_b200.trace import Settings, Trace

pytestmark = pytest.mark.gpu


def lights(rng, count, radius, reach):
    out = []
    for i in range(count):
        p = rng.uniform((-9, 1, -9), (9, 18, 9))
        if i % 2:
            d = rng.normal(size=3)
            out.append(synth.spot_light(p, d / np.linalg.norm(d), 40.0, float(rng.uniform(5, 80)), 4.0,
                                        (1.0, 0.8, 0.6), radius=radius, rng_range=reach))
        else:
            out.append(synth.point_light(p, float(rng.uniform(1, 50)), (0.6, 0.8, 1.0), radius=radius,
                                         rng_range=reach))
    return np.concatenate(out)


@pytest.mark.parametrize("sampler", ["sobol", "pcg"])
@pytest.mark.parametrize("count,radius,reach", [(1, 0.1, 30.0), (2, 0.0, 8.0), (3, 2.5, 30.0), (9, 0.0, 4.0),
                                                (33, 0.2, 12.0), (128, 0.2, 30.0), (700, 0.05, 6.0)])
def test_descents_agree(gpu, sampler, count, radius, reach):
    w = synth.small("plain_512", (56, 43), sampler)
    w.scene.lights = lights(np.random.default_rng(count), count, radius, reach)
    if count == 9:  # lights at one point: boxes of no extent
        w.scene.lights["position"][:5] = w.scene.lights["position"][0]
    images = []
    for slot_kernels in (True, False):
        t = Trace(w.scene, Settings.deep(3, sampler=sampler, sobol_samples=16), w.width, w.height)
        t.set_tuning(slot_kernels=slot_kernels)
        t.sample(3, 8)
        images.append(t.read_accum())
        t.close()
    assert images[0][..., :3].mean() > 0.0
    assert np.array_equal(images[0].view(np.uint32), images[1].view(np.uint32))
