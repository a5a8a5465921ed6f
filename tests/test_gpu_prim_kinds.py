"""Primitives whose kind is none of gi_prim_kind are met by no ray, whatever bits their
kind has, as in the fp32 oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [3, -1, 0x100, 0x101, 0x102, 0x7FFFFFFF, -0x80000000])
def test_unknown_kinds_are_not_met(gi, oracle, cuda, kind):
    w, h = 65, 41
    prims = gi.scene_generate(43, 12, 6)
    view = gi.view_from_camera(gi.camera_spline(3, 11, 64), w, h)
    known = [prims[k].kind for k in range(len(prims))]
    for k in (4, 7, 14, len(prims) - 1):  # two boxes and two spheres
        prims[k].kind = kind
    assert {known[4], known[7]} == {gi.GI_PRIM_BOX} and {known[14], known[-1]} == {gi.GI_PRIM_SPHERE}
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
