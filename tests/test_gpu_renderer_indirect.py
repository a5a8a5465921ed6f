"""The renderer's optional indirect image: written in place by the frame's last light
stage where it is an image of its own, copied where it overlaps an input or the lit
image (the frame must still read what the caller passed in)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bilateral,radius", [(True, 0), (False, 0), (True, 2), (False, 2)])
@pytest.mark.parametrize("bounces", [1, 2])
@pytest.mark.parametrize("learned", [False, True])
def test_indirect_image_in_place_or_copied(gi, oracle, cuda, bilateral, radius, bounces, learned):
    w, h = 133, 67
    prims = gi.scene_generate(17, 10, 3)
    view = gi.view_from_camera(gi.camera_spline(6, 5, 64, prims), w, h)
    light = gi.view_from_camera(gi.scene_light(), 64, 64)
    gb = oracle.gbuffer(view, prims)
    direct = oracle.direct_light(view, light, gb, oracle.shadow_map(light, prims))
    dev = lambda a: cuda.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()
    images = [dev(gb[k]) for k in ("albedo", "normal", "moments", "ndc")] + [dev(direct)]
    net = gi.Mlp(seed=3) if learned else None

    def frame(place):
        own = [t.clone() for t in images]
        lit = cuda.full((h, w, 4), -7.0, dtype=cuda.float32, device="cuda")
        # "shifted": 16 bytes short of the image, so that it overlaps it in part
        pool = cuda.full((h * w * 4 + 4 * h * w,), -7.0, dtype=cuda.float32, device="cuda")
        ind = {"own": pool[:h * w * 4].view(h, w, 4), "direct": own[4], "albedo": own[0]}.get(place)
        if place == "shifted":
            own[4] = pool[4:4 + h * w * 4].view(h, w, 4)
            own[4].copy_(images[4])
            ind = pool[:h * w * 4].view(h, w, 4)
        r = gi.Renderer(w, h, dirs=6, step_cap=24, bounces=bounces, bilateral=bilateral, denoise_radius=radius)
        if net:
            r.set_learned(net, few_dirs=1, few_step_dirs=16, judge_every=2, threshold=0.25)
        r.render(view, *own, lit, ind)
        cuda.cuda.synchronize()
        r.close()
        return lit, ind.clone()

    lit, ind = frame("own")
    assert float(ind.min()) > -7.0
    for place in ("direct", "albedo", "shifted"):
        l2, i2 = frame(place)
        assert cuda.equal(l2, lit) and cuda.equal(i2, ind), place
