"""The direction split of whole frames (four threads a pixel: the rule's choice for
small frames) against one thread a pixel, bit for bit: the march, and the two-bounce
renderer, whose first bounce records its march and whose second re-lights the record,
at images smaller than a warp's pixels and ragged ones, with directions that do not
divide evenly over the threads."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _inputs(gi, oracle, torch, w, h):
    prims = gi.scene_generate(91, 8, 3)
    view = gi.view_from_camera(gi.camera_spline(4, 7, 64, prims), w, h)
    light = gi.view_from_camera(gi.scene_light(), 64, 64)
    gb = oracle.gbuffer(view, prims)
    direct = oracle.direct_light(view, light, gb, oracle.shadow_map(light, prims))
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()
    return view, [dev(gb[k]) for k in ("albedo", "normal", "moments", "ndc")] + [dev(direct)]


@pytest.mark.parametrize("w,h", [(4, 4), (9, 5), (33, 17), (131, 66), (260, 70)])
@pytest.mark.parametrize("dirs", [4, 5, 11, 32])
@pytest.mark.parametrize("precision", [0, 1, 2])
def test_split_frames_equal_one_thread_a_pixel(gi, oracle, cuda, w, h, dirs, precision):
    view, images = _inputs(gi, oracle, cuda, w, h)
    frames = []
    for rays in (32 * dirs, 32 * ((dirs + 3) // 4)):
        gi.march_set_layout(w, h, dirs, 0, 24, precision, 4, rays)
        r = gi.Renderer(w, h, dirs=dirs, step_cap=24, bounces=2, bilateral=False, precision=precision)
        out = [cuda.full((h, w, 4), -7.0, dtype=cuda.float32, device="cuda") for _ in range(2)]
        r.render(view, *images, *out)
        cuda.cuda.synchronize()
        r.close()
        frames.append(out)
    for a, b in zip(*frames):
        assert cuda.equal(a, b)
