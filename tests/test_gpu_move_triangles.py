"""Where a move's traversal triangles come from: the blobs a tracer was created
from have the triangles that the device holds already; a host's own buffers are
read, as they may hold others."""
import ctypes as C

import numpy as np
import pytest

import oracle
from pfx_b200 import synth
from pfx_b200.trace import SceneBuffers, Trace, make_rays

pytestmark = pytest.mark.gpu


def compare(trace, buffers, rays):
    got, want = trace.trace_rays(rays), oracle.trace(buffers, rays)
    assert np.array_equal(got["hit"], want["hit"])
    h = want["hit"] == 1
    assert np.array_equal(got["slot"][h], want["slot"][h])
    assert np.array_equal(got["t"][h].view(np.uint32), want["t"][h].view(np.uint32))
    assert np.array_equal(trace.occluded(rays), oracle.trace(buffers, rays, any_hit=True)["hit"] == 1)
    return want["hit"].copy()


def test_a_move_keeps_or_reads_the_triangles(gpu):
    w = synth.instanced_1080(target=4000)
    buffers = SceneBuffers(w.scene, w.settings)
    trace = Trace(w.scene, w.settings, 8, 8, buffers=buffers)
    rng = np.random.default_rng(8)
    o = rng.uniform((-60, 0, -60), (60, 40, 60), (8000, 3)).astype(np.float32)
    rays = make_rays(o, rng.normal(size=(8000, 3)).astype(np.float32), 1e20)
    first = compare(trace, buffers, rays)
    moved = w.scene.instances["transform"].copy()
    moved[:, 12] += 5.0  # along x
    assert trace.set_instance_transforms(moved)
    second = compare(trace, buffers, rays)
    assert (first != second).any()
    # a host that shrinks every triangle a little in buffers of its own: the boxes still hold them
    b = buffers.buffers
    corners = np.ctypeslib.as_array((C.c_float * (b.triangles_bytes // 4)).from_address(b.triangles)).reshape(-1, 24)
    for k in range(3):
        corners[:, 4:7][:, k] = corners[:, k] + np.float32(0.75) * (corners[:, 4 + k] - corners[:, k])
    trace.finish_tops(buffers)
    third = compare(trace, buffers, rays)
    assert (second != third).any()
