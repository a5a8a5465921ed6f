"""The ray casts of the G-buffer and the shadow map against the fp32 oracle, which
tests every primitive with every ray: the kernels skip primitives that the bounds of
a warp's rays miss, and every value must stay the same bits (the same operations in
the same order).  Images smaller than a warp's pixels and ragged ones; scenes of one
primitive, of more than one shared-memory stage, and of degenerate ones: the camera
inside a box and a sphere, flat boxes, faces in the camera's planes, primitives behind
it, corners at infinity and NaN; a camera along an axis, whose central rays have zero
components."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (5, 3), (8, 4), (33, 9), (65, 41)]


def _prims(gi, kind, cam):
    if kind != "degenerate":
        return gi.scene_generate(41, *{"room": (0, 0), "few": (9, 4), "many": (420, 180)}[kind])
    prims = gi.scene_generate(43, 12, 6)
    p, inf, nan = [cam.pos[k] for k in range(3)], float("inf"), float("nan")
    boxes = [([v - 0.05 for v in p], [v + 0.05 for v in p]),  # around the camera
             ([0.2, 0.3, 0.4], [0.6, 0.3, 0.7]), ([0.7, 0.1, 0.2], [0.7, 0.1, 0.2]),  # flat, a point
             ([p[0], 0.0, 0.0], [p[0] + 0.1, 0.2, 1.0]), ([0.1, p[1], 0.1], [0.4, p[1], 0.9]),
             ([-inf, 0.0, 0.0], [0.02, 0.1, 1.0]), ([nan, 0.1, 0.1], [0.5, 0.5, 0.5]),
             ([0.3, 0.1, nan], [0.5, 0.5, nan]), ([0.9, 0.9, 0.9], [0.8, 0.8, 0.8])]
    for q, (a, b) in zip(list(prims)[1:], boxes):
        q.kind = gi.GI_PRIM_BOX
        for k in range(3):
            q.a[k], q.b[k] = a[k], b[k]
    n = len(prims)
    for q, (c, r) in zip([prims[n - k] for k in (1, 2, 3)], [(p, 0.04), ([0.5, 0.5, 0.5], 0.0), ([0.2, 0.2, nan], 0.1)]):
        q.kind = gi.GI_PRIM_SPHERE
        for k in range(3):
            q.a[k] = c[k]
        q.b[0] = r
    return prims


def _camera(gi, along_axis):
    cam = gi.camera_spline(3, 11, 64)
    if along_axis:
        cam.hor_angle = cam.vert_angle = 0.0
    return cam


@pytest.mark.parametrize("w,h", SIZES)
@pytest.mark.parametrize("kind", ["room", "few", "many", "degenerate"])
@pytest.mark.parametrize("along_axis", [False, True])
def test_ray_casts_equal_the_oracle(gi, oracle, cuda, w, h, kind, along_axis):
    cam = _camera(gi, along_axis)
    prims = _prims(gi, kind, cam)
    view = gi.view_from_camera(cam, w, h)
    dev, n = gi.prims_to_device(prims)
    new = lambda c: cuda.full((h, w, c), -7.0, dtype=cuda.float32, device="cuda")
    got = {k: new(c) for k, c in (("albedo", 4), ("emissive", 4), ("normal", 4), ("moments", 2), ("ndc", 1))}
    gi.gbuffer(view, dev, n, *got.values())
    shadow = new(1)
    gi.shadow_map(view, dev, n, shadow)
    cuda.cuda.synchronize()
    ref = oracle.gbuffer(view, prims)
    for k, v in got.items():
        np.testing.assert_array_equal(v.cpu().numpy(), ref[k], err_msg=k)
    np.testing.assert_array_equal(shadow.cpu().numpy(), oracle.shadow_map(view, prims))
