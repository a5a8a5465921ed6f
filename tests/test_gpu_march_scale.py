"""The march does not depend on the homogeneous scale of the inverse view-projection: the
same matrix times a power of two gives the same bits in every precision (no operation
leaves the normal range at these scales, and powers of two round nothing)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("exponent", [-76, -70, -40, 40, 60])
def test_scaled_matrix_gives_the_same_bits(gi, oracle, cuda, precision, exponent):
    w, h = 97, 66
    prims = gi.scene_generate(77, 6, 2)
    view = gi.view_from_camera(gi.camera_spline(5, 9, 64, prims), w, h)
    light = gi.view_from_camera(gi.scene_light(), 64, 64)
    gb = oracle.gbuffer(view, prims)
    direct = oracle.direct_light(view, light, gb, oracle.shadow_map(light, prims))
    n = gi.mip_level_count(w, h, 10)
    dev = lambda a: cuda.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()
    lb = [dev(a) for a in oracle.blur_pyramid(oracle.mip_chain(direct, n))]
    db = [dev(a) for a in oracle.blur_pyramid(oracle.mip_chain(gb["moments"], n))]

    def march(v):
        out = cuda.full((h, w, 4), -7.0, dtype=cuda.float32, device="cuda")
        gi.march(v, gi.GiMarchParams(6, 24, 4, 0, precision), lb, db, dev(gb["normal"]), dev(gb["ndc"]), out)
        cuda.cuda.synchronize()
        return out.cpu().numpy()

    ref = march(view)
    scaled = gi.GiView.from_buffer_copy(bytes(view))
    for k in range(16):
        scaled.inv_view_proj[k] = view.inv_view_proj[k] * 2.0 ** exponent
    np.testing.assert_array_equal(march(scaled), ref)
