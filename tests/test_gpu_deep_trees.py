"""The four-box walk's stack.  The layout's bound on what a ray may hold is at
least what any ray holds, whichever order the walk takes; and on trees where a
ray holds more waiting entries than the stack has room for (QUAD_STACK in
pfxt_types.h), while the reference's own stack is far from full, hits and
occlusion equal the oracle's bit for bit."""
import ctypes as C

import numpy as np
import pytest

import oracle
from pfx_b200 import abi, synth
from pfx_b200.trace import INSTANCE, SceneBuffers, SceneDesc, Settings, Trace, make_rays

F32 = np.float32
NODE = np.dtype([("lo", "<f4", 4), ("hi", "<f4", 4), ("first", "<u4"), ("count", "<u4"), ("pad", "<u4", 2)])
QUAD_STACK = 64


def chain(sign, steps, ratio, copies, start):
    """Triangles ever larger and further off along (1, 1, 1): towards minus the
    tree leans right, and every box holds the neighbourhood of the origin's corner."""
    rng = np.random.default_rng(7)
    s = np.repeat(ratio ** np.arange(steps) * 2.0 ** start, copies)
    return (sign * s[:, None, None] * (1 + 0.05 * rng.uniform(-1, 1, (len(s), 3, 3)))).astype(F32)


def scene_of(sign, placed):
    with np.errstate(over="ignore"):  # the shading normals of the largest
        mesh = synth.triangles(chain(sign, 320, 1.3, 8, -69))
    world = synth.triangles(np.array([[[3, 0, 0], [4, 0, 0], [3, 1, 0]]], F32))
    inst = np.zeros(placed, INSTANCE)
    inst["two_sided"] = inst["casts_shadow"] = 1
    for k in range(placed):
        inst["transform"][k] = synth.transform_matrix(1.25 ** (k // 4), np.eye(3), np.zeros(3))
    camera = synth.look_at((0, 0, 10), (0, 0, 0), 45, 1.0)
    return SceneDesc(world, synth.material(), camera, meshes=[mesh], instances=inst)


def most_held(nodes, o, d, nearest):
    """The most entries that a ray which meets no triangle holds on the four-box
    nodes: nearest child first, or the first child first."""
    def boxes(i):
        out = []
        for c in (i + 1, int(nodes["first"][i])):
            inner = nodes["count"][c] == 0 and nodes["pad"][c, 0] == 0
            out += [c + 1, int(nodes["first"][c])] if inner else [c]
        return out

    world, stack, most, ref, inside = (o, d), [], 0, 0, None
    while True:
        oo, dd = inside or world
        n = nodes[ref]
        nxt, near = None, 0.0
        if n["pad"][0] == 1 and inside is None:
            stack.append(None)
            if n["pad"][1]:
                m = nodes[n["pad"][1]]
                last = np.array([m["first"], m["count"], m["pad"][0], m["pad"][1]], np.uint32).view(F32)
                rows = np.array([m["lo"], m["hi"], last], float)
                oo, dd = rows[:, :3] @ oo + rows[:, 3], rows[:, :3] @ dd
            inside = (oo, dd)
            nxt = int(n["first"])
        elif n["count"] == 0:
            for c in boxes(ref)[::-1]:
                with np.errstate(over="ignore"):
                    a, b = (nodes["lo"][c, :3] - oo) / dd, (nodes["hi"][c, :3] - oo) / dd
                entry, leave = max(np.minimum(a, b).max(), 0.0), np.maximum(a, b).min()
                if entry <= leave:
                    if nearest and nxt is not None and entry >= near:
                        stack.append(c)
                    else:
                        if nxt is not None:
                            stack.append(nxt)
                        nxt, near = c, entry
        most = max(most, len(stack))
        while nxt is None:
            if not stack:
                return most
            nxt = stack.pop()
            if nxt is None:
                inside = None
        ref = nxt


def rays(sign):
    rng = np.random.default_rng(3)
    o = (rng.normal(size=(600, 3)) * 10.0 ** rng.uniform(-18, 0, (600, 1))).astype(F32)
    o[:200] = 0.0
    d = (sign * (1 + 0.15 * rng.normal(size=(600, 3)) * rng.uniform(0, 1, (600, 1)))).astype(F32)
    d[500:] = rng.normal(size=(100, 3))
    return o, d


def layout(buffers):
    small, need = C.c_uint32(), C.c_uint32()
    abi.check(abi.load().pfxt_debug_layout(C.byref(buffers.buffers), C.byref(small), C.byref(need)))
    return small.value, need.value


@pytest.mark.parametrize("sign", [-1.0, 1.0])
def test_the_bound_holds_on_deep_trees(sign):
    """A ray holds more entries than the stack has, nearest child first (and on
    the left-leaning tree also first child first); the layout's figure says so."""
    buffers = SceneBuffers(scene_of(sign, 280), Settings())
    nodes = buffers.array("nodes").view(NODE)
    o, d = (x[0].astype(float) for x in rays(sign))
    held = most_held(nodes, o, d, True)
    small, need = layout(buffers)
    assert QUAD_STACK < held <= need and small == 1
    assert buffers.buffers.max_depth <= 64
    assert (most_held(nodes, o, d, False) > QUAD_STACK) == (sign > 0)


@pytest.mark.filterwarnings("ignore:overflow")
@pytest.mark.parametrize("shape", ["cloud", "left", "right", "instanced"])
def test_the_bound_holds_for_every_ray(shape):
    rng = np.random.default_rng(len(shape))
    if shape == "instanced":
        scene, top = synth.instanced_1080(target=4000).scene, 60.0
    else:
        v = rng.uniform(-4, 4, (300, 1, 3)) + rng.uniform(-0.5, 0.5, (300, 3, 3))
        if shape != "cloud":
            v = chain(1.0 if shape == "left" else -1.0, 90, 1.5, 2, -8)
        scene = SceneDesc(synth.triangles(v.astype(F32)), synth.material(),
                          synth.look_at((0, 0, 10), (0, 0, 0), 45, 1.0))
        top = float(np.abs(v).max())
    buffers = SceneBuffers(scene, Settings())
    nodes = buffers.array("nodes").view(NODE)
    small, need = layout(buffers)
    assert small == 1 and need <= QUAD_STACK  # the walk without the check
    held = [most_held(nodes, rng.uniform(-top, top, 3) * rng.choice([0.0, 1e-3, 1.0]), rng.normal(size=3), nearest)
            for _ in range(60) for nearest in (True, False)]
    if shape == "right":  # along the chain, from its small end
        held.append(most_held(nodes, np.zeros(3), np.array([-1.0, -1.01, -0.99]), True))
        assert held[-1] > 10
    assert max(held) <= need


@pytest.mark.gpu
@pytest.mark.parametrize("sign", [-1.0, 1.0])
@pytest.mark.parametrize("placed", [1, 280])
def test_deep_trees_equal_the_oracle(gpu, sign, placed):
    scene = scene_of(sign, placed)
    trace, ref = Trace(scene, Settings(), 8, 8), oracle.scene_buffers(scene, Settings())
    o, d = rays(sign)
    for limit in (1e20, 1e-3, np.inf):
        batch = make_rays(o, d, F32(limit))
        got, want = trace.trace_rays(batch), oracle.trace(ref, batch)
        assert np.array_equal(got["hit"], want["hit"])
        h = want["hit"] == 1
        assert np.array_equal(got["slot"][h], want["slot"][h])
        assert np.array_equal(got["record"][h], want["record"][h])
        assert np.array_equal(got["t"][h].view(np.uint32), want["t"][h].view(np.uint32))
        assert np.array_equal(trace.occluded(batch), oracle.trace(ref, batch, any_hit=True)["hit"] == 1)
