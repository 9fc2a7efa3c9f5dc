"""The four-box walk at the sizes and rays where it can go wrong: trees of one
to a few nodes, trees that are one long chain, flat boxes, every class of ray
it hands over (degenerate axes, long directions, far origins) and limits that
are zero, negative, infinite or NaN, against the oracle bit for bit."""
import numpy as np
import pytest

import oracle
from pfx_b200 import synth
from pfx_b200.trace import SceneDesc, Settings, Trace, make_rays

F32 = np.float32


def rays_for(rng, lo, hi, n):
    o = rng.uniform(lo, hi, (n, 3)).astype(F32)
    d = rng.normal(size=(n, 3)).astype(F32)
    k = np.arange(n)
    d[k % 7 == 1, 0] = 0.0                      # degenerate axes
    d[k % 7 == 2, 1:] = 0.0
    d[k % 14 == 3] *= F32(3e6)                  # beyond the bounded directions
    d[k % 14 == 10, 2] = F32(-0.0)
    o[k % 28 == 4, 0] = F32(1e25)               # beyond the bounded origins
    o[k % 11 == 5] = np.round(o[k % 11 == 5])   # origins on box planes
    return o, d


def compare(trace, ref, batch):
    got = trace.trace_rays(batch)
    want = oracle.trace(ref, batch)
    assert np.array_equal(got["hit"], want["hit"])
    h = want["hit"] == 1
    assert np.array_equal(got["slot"][h], want["slot"][h])
    assert np.array_equal(got["record"][h], want["record"][h])
    assert np.array_equal(got["t"][h].view(np.uint32), want["t"][h].view(np.uint32))
    assert np.array_equal(trace.occluded(batch), oracle.trace(ref, batch, any_hit=True)["hit"] == 1)
    return h.sum()


@pytest.mark.gpu
@pytest.mark.parametrize("count", [1, 2, 3, 4, 5, 9, 17, 40, 300])
@pytest.mark.parametrize("shape", ["cloud", "flat", "chain"])
def test_small_trees(gpu, count, shape):
    rng = np.random.default_rng(count)
    v = rng.uniform(-4, 4, (count, 1, 3)) + rng.uniform(-1.5, 1.5, (count, 3, 3))
    if shape == "flat":       # boxes of no thickness, corners on whole numbers, some shared
        v = np.round(v)
        v[:, :, count % 3] = np.round(v[:, :1, count % 3])
    if shape == "chain":      # triangles at ever larger distances: a tree that is one long chain
        v = (v * 0.1 + 1.0) * (1.3 ** np.arange(count) if count < 150 else 1.05 ** np.arange(count))[:, None, None]
    scene = SceneDesc(synth.triangles(v.astype(F32)), synth.material(), synth.look_at((0, 0, 10), (0, 0, 0), 45, 1.0))
    trace = Trace(scene, Settings(), 8, 8)
    ref = oracle.scene_buffers(scene, Settings())
    top = float(np.abs(v).max())
    o, d = rays_for(rng, -top, top, 3000)
    aim = v[rng.integers(0, count, 3000)].mean(1).astype(F32)   # half of them towards a triangle
    d[::2] = (aim - o)[::2]
    hits = compare(trace, ref, make_rays(o, d, 1e20))
    assert hits > 0 or count < 9   # rounded to whole numbers, a few triangles may all be degenerate
    for limit in (0.0, -1.0, 1e-3, 0.5, np.inf):
        compare(trace, ref, make_rays(o, d, F32(limit)))
    nan = make_rays(o, d, F32(np.nan))
    assert not trace.occluded(nan).any() and not trace.trace_rays(nan)["hit"].any()


@pytest.mark.gpu
@pytest.mark.parametrize("count", [127, 128, 129, 257])
def test_the_last_triangles_of_a_block(gpu, count):
    """The triangles are laid out by blocks of 128: rays at the last ones of a full and of a short block."""
    rng = np.random.default_rng(count)
    v = rng.uniform(-4, 4, (count, 1, 3)) + rng.uniform(-0.5, 0.5, (count, 3, 3))
    scene = SceneDesc(synth.triangles(v.astype(F32)), synth.material(), synth.look_at((0, 0, 10), (0, 0, 0), 45, 1.0))
    aim = np.repeat(v.mean(1), 4, 0).astype(F32)
    o = rng.uniform(-6, 6, aim.shape).astype(F32)
    hits = compare(Trace(scene, Settings(), 8, 8), oracle.scene_buffers(scene, Settings()), make_rays(o, aim - o, 1e20))
    assert hits == len(o)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["doubled", "needles", "stacked", "grid", "mixed"])
def test_ties_and_slivers(gpu, kind):
    """Where the order of the walk could show: the same triangles twice, needles
    seen edge on, coplanar overlapping quads, rays through shared corners and
    edges, and all of it over six orders of magnitude."""
    rng = np.random.default_rng(len(kind))
    n = 400
    v = rng.uniform(-4, 4, (n, 1, 3)) + rng.uniform(-1.0, 1.0, (n, 3, 3))
    if kind == "doubled":
        v = np.concatenate([v, v[::-1], v[:, [1, 2, 0]]])
    if kind == "needles":
        v[:, 2] = v[:, 0] + (v[:, 1] - v[:, 0]) * rng.uniform(0.2, 0.9, (n, 1)) + rng.normal(size=(n, 3)) * 1e-5
    if kind == "stacked":
        v = np.round(v)
        v[:, :, 1] = (np.arange(n) % 4)[:, None]
    if kind == "grid":
        x, z = np.meshgrid(np.arange(-7, 7), np.arange(-7, 7))
        a = np.stack([x, 0.25 * ((x + z) % 3), z], -1).reshape(-1, 3).astype(float)
        v = np.concatenate([a[:, None] + np.array([[0, 0, 0], [1, 0, 0], [1, 0, 1]]),
                            a[:, None] + np.array([[0, 0, 0], [1, 0, 1], [0, 0, 1]])])
    if kind == "mixed":
        v *= 10.0 ** rng.uniform(-3, 3, (n, 1, 1))
    scene = SceneDesc(synth.triangles(v.astype(F32)), synth.material(), synth.look_at((0, 0, 10), (0, 0, 0), 45, 1.0))
    trace = Trace(scene, Settings(), 8, 8)
    ref = oracle.scene_buffers(scene, Settings())
    m = 40_000
    f = v.astype(F32)
    o = rng.uniform(-8, 8, (m, 3)).astype(F32)
    # at corners, at edges, at insides, and (every fourth) along the plane of a triangle
    t = rng.integers(0, len(f), m)
    w = rng.dirichlet((1, 1, 1), m).astype(F32)
    w[::3] = np.eye(3, dtype=F32)[rng.integers(0, 3, len(w[::3]))]
    w[1::3, 0] = 0.0
    aim = np.einsum("ij,ijk->ik", w / w.sum(1, keepdims=True), f[t]).astype(F32)
    o[::4] = (aim + (f[t, 0] - f[t, 1]) * rng.uniform(1, 3, (m, 1)).astype(F32))[::4]
    d = (aim - o).astype(F32)
    assert compare(trace, ref, make_rays(o, d, 1e20)) > m // 3
    compare(trace, ref, make_rays(o, d, rng.uniform(0.5, 1.5, m).astype(F32)))


@pytest.mark.gpu
def test_coincident_instances(gpu):
    """Instances placed on one another: hits tie across instances."""
    w = synth.instanced_1080(target=2000)
    w.scene.instances = np.concatenate([w.scene.instances, w.scene.instances[::-1], w.scene.instances[::3]])
    trace = Trace(w.scene, w.settings, 8, 8)
    ref = oracle.scene_buffers(w.scene, w.settings)
    o, d = rays_for(np.random.default_rng(4), (-60, 0, -60), (60, 40, 60), 20000)
    assert compare(trace, ref, make_rays(o, d, 1e20)) > 1000


@pytest.mark.gpu
def test_instances_with_every_ray_class(gpu):
    w = synth.instanced_1080(target=3000)
    trace = Trace(w.scene, w.settings, 8, 8)
    ref = oracle.scene_buffers(w.scene, w.settings)
    rng = np.random.default_rng(2)
    o, d = rays_for(rng, (-60, 0, -60), (60, 40, 60), 20000)
    assert compare(trace, ref, make_rays(o, d, 1e20)) > 1000
    compare(trace, ref, make_rays(o, d, rng.uniform(0.0, 60.0, len(o)).astype(F32)))


def test_the_loose_comparison_holds_every_box_that_passes_exactly():
    """Entry and exit by x * r with r an ulp off 1/d, the comparison scaled by
    1 + 2^-18, against the quotients (fp32 arithmetic, worst cases of r)."""
    rng = np.random.default_rng(9)
    n = 400_000
    o = rng.normal(size=(n, 3)).astype(F32) * F32(10.0) ** rng.integers(-3, 4, (n, 1)).astype(F32)
    lo = (o + rng.normal(size=(n, 3)).astype(F32) * F32(10.0) ** rng.integers(-4, 3, (n, 1)).astype(F32)).astype(F32)
    size = np.abs(rng.normal(size=(n, 3))).astype(F32) * F32(10.0) ** rng.integers(-6, 2, (n, 3)).astype(F32)
    size[rng.random((n, 3)) < 0.2] = 0.0
    hi = (lo + size).astype(F32)
    aim = (lo + size * rng.choice([0.0, 0.5, 1.0], (n, 3)).astype(F32)).astype(F32)  # at the corners and edges
    d = (aim - o).astype(F32)
    d = (d.view(np.int32) + rng.integers(-3, 4, (n, 3)).astype(np.int32)).view(F32)  # and a few ulps beside them
    ok = ((np.abs(d) >= 1e-12) & (np.abs(d) < 1e6)).all(1)
    o, lo, hi, d = o[ok], lo[ok], hi[ok], d[ok]
    a, b = (lo - o) / d, (hi - o) / d
    near = np.maximum(np.minimum(a, b).max(1), F32(0))
    far = np.maximum(a, b).min(1)
    exact = ~(near > far)
    assert 0.2 < exact.mean() < 1.0
    for ulps in (-1, 0, 1):
        r = F32(1.0) / d
        r = (r.view(np.int32) + np.int32(ulps)).view(F32)
        a, b = (lo - o) * r, (hi - o) * r
        n_l = np.maximum(np.minimum(a, b).max(1), F32(0))
        f_l = np.maximum(a, b).min(1)
        scale = F32(1.0) + F32(2.0) ** F32(-18)
        for limit in (np.full_like(near, np.inf), near):   # the tightest limit that the box passes
            assert (n_l <= np.minimum(f_l, limit) * scale)[exact].all()
