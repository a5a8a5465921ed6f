"""The fast precisions' horizon of a step whose depth is NaN, stated: angle 0, a hit
wherever the horizon is above it (the exact precision takes no hit there).

With NaN depth everywhere, normals that face the eye (initial horizon about pi / 2) and
constant light L, a direction's first step lowers the horizon to 0 and no later one
does.  Its contribution then equals the initial term's, so a direction gives L where
the exact precision, which takes no hit, gives the ambient light: the image is the exact
one times L / ambient, where the samples are clear of the border's fade.  Tolerance:
a term's error in the fast arithmetic is some 1e-6 of it; 1e-4."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

AMBIENT, LIGHT = 0.01, 0.5


def _facing(view, w, h, depth):
    """Unit vectors from the points at window depth `depth` to the eye."""
    inv = np.array(list(view.inv_view_proj), np.float64).reshape(4, 4).T
    eye = (np.array(list(view.inv_view), np.float64).reshape(4, 4).T @ [0, 0, 0, 1])[:3]
    x, y = np.meshgrid((np.arange(w) + 0.5) / w * 2 - 1, (np.arange(h) + 0.5) / h * 2 - 1)
    p = np.stack([x, y, np.full_like(x, depth), np.ones_like(x)], -1) @ inv.T
    d = eye - p[..., :3] / p[..., 3:]
    return d / np.linalg.norm(d, axis=-1, keepdims=True)


@pytest.mark.parametrize("precision", ["fast", "texture"])
@pytest.mark.parametrize("dirs,cap", [(1, 24), (6, 0)])
def test_a_step_of_nan_depth_has_angle_zero(gi, oracle, cuda, precision, dirs, cap):
    w, h = 160, 96
    view = gi.view_from_camera(gi.camera_spline(5, 9, 64, gi.scene_generate(77, 6, 2)), w, h)
    n = gi.mip_level_count(w, h, 10)
    depth = [np.full((h >> k, w >> k, 2), np.nan, np.float32) for k in range(n)]
    light = [np.full((h >> k, w >> k, 4), LIGHT, np.float32) for k in range(n)]
    ndc = np.full((h, w, 1), 0.99, np.float32)
    normal = np.ones((h, w, 4), np.float32)
    normal[..., :3] = _facing(view, w, h, 0.99)
    exact, _ = oracle.march(view, dirs, cap, light, depth, normal, ndc)
    dev = lambda a: cuda.from_numpy(a).cuda()
    out = cuda.full((h, w, 4), -7.0, dtype=cuda.float32, device="cuda")
    p = gi.GiMarchParams(dirs, cap, 4, 0, gi.GI_MARCH_TEXTURE if precision == "texture" else gi.GI_MARCH_FAST)
    gi.march(view, p, [dev(a) for a in light], [dev(a) for a in depth], dev(normal), dev(ndc), out)
    cuda.cuda.synchronize()
    inner = (slice(h // 5, h - h // 5), slice(w // 5, w - w // 5), slice(0, 3))
    ref = exact[inner].astype(np.float64) * (LIGHT / AMBIENT)
    assert ref.min() > 0.0
    np.testing.assert_allclose(out.cpu().numpy()[inner], ref, rtol=1e-4)
