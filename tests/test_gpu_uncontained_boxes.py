"""Host-packed nodes whose boxes do not hold their children's: the reference
tests every box on the way to a leaf, so a leaf that pokes out of one is missed
through the part outside.  The four-box walk, which passes over boxes, does not
take such scenes."""
import ctypes as C

import numpy as np
import pytest

import oracle
from pfx_b200 import abi, synth
from pfx_b200.trace import SceneBuffers, SceneDesc, Settings, Trace, make_rays

F32 = np.float32
NODE = np.dtype([("lo", "<f4", 4), ("hi", "<f4", 4), ("first", "<u4"), ("count", "<u4"), ("pad", "<u4", 2)])


def small(buffers):
    out, need = C.c_uint32(), C.c_uint32()
    abi.check(abi.load().pfxt_debug_layout(C.byref(buffers.buffers), C.byref(out), C.byref(need)))
    return out.value


def nodes_of(buffers):
    """The nodes in place."""
    b = buffers.buffers
    return np.ctypeslib.as_array((C.c_uint8 * b.nodes_bytes).from_address(b.nodes)).view(NODE)


def cloud():
    rng = np.random.default_rng(6)
    v = rng.uniform(-4, 4, (500, 1, 3)) + rng.uniform(-0.8, 0.8, (500, 3, 3))
    return SceneDesc(synth.triangles(v.astype(F32)), synth.material(), synth.look_at((0, 0, 10), (0, 0, 0), 45, 1.0))


def inner_nodes(nodes):
    """The root and every ninth inner node."""
    return [0] + [int(k) for k in np.flatnonzero((nodes["count"] == 0) & (nodes["pad"][:, 0] == 0))[1::9]]


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("side", ["lo", "hi"])
def test_a_box_that_does_not_hold_its_children_is_seen(axis, side):
    buffers = SceneBuffers(cloud(), Settings())
    nodes = nodes_of(buffers)
    assert small(buffers) == 1
    for k in inner_nodes(nodes):
        kept = nodes[side][k, axis]
        towards = nodes["hi" if side == "lo" else "lo"][k, axis]
        nodes[side][k, axis] = np.nextafter(kept, towards, dtype=F32)  # one ulp inside is enough
        assert small(buffers) == 0
        nodes[side][k, axis] = kept
    assert small(buffers) == 1


@pytest.mark.parametrize("name", ["plain_512", "instanced_1080", "room_4k"])
def test_built_scenes_hold_their_boxes(name):
    w = synth.small(name, (16, 16), "sobol")
    buffers = SceneBuffers(w.scene, w.settings)
    assert small(buffers) == 1
    if name == "instanced_1080":
        buffers.move_instances(np.ascontiguousarray(w.scene.instances["transform"][::-1]))
        assert small(buffers) == 1


@pytest.mark.gpu
def test_hits_equal_the_oracle(gpu):
    scene = cloud()
    buffers = SceneBuffers(scene, Settings())
    nodes = nodes_of(buffers)
    for k in inner_nodes(nodes)[1:]:
        nodes["lo"][k, k % 3] += F32(0.3) * (nodes["hi"][k, k % 3] - nodes["lo"][k, k % 3])
    trace = Trace(scene, Settings(), 8, 8, buffers=buffers)
    rng = np.random.default_rng(1)
    o, d = (rng.uniform(-6, 6, (20000, 3)).astype(F32) for _ in range(2))
    batch = make_rays(o, d, 1e20)
    got, want = trace.trace_rays(batch), oracle.trace(buffers, batch)
    whole = oracle.trace(oracle.scene_buffers(scene, Settings()), batch)
    assert (want["hit"] != whole["hit"]).sum() > 100  # the boxes decide
    assert np.array_equal(got["hit"], want["hit"])
    h = want["hit"] == 1
    assert np.array_equal(got["slot"][h], want["slot"][h])
    assert np.array_equal(got["t"][h].view(np.uint32), want["t"][h].view(np.uint32))
    assert np.array_equal(trace.occluded(batch), oracle.trace(buffers, batch, any_hit=True)["hit"] == 1)
