"""The bilateral filter (and the final gather) where its tiles and its exponential can go wrong, against the
fp32 oracle bit for bit (the same operations in the same order): images smaller than a
tile, one row or column past it, odd heights (a thread filters two rows), and depths and
normals whose weights reach every part of the exponential's range: 1, subnormal, 0, and
infinite and NaN exponents."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (5, 3), (2, 9), (32, 16), (33, 17), (31, 15), (70, 34)])
@pytest.mark.parametrize("kind", ["smooth", "range", "special"])
def test_bilateral_equals_the_oracle(gi, oracle, cuda, w, h, kind):
    r = np.random.default_rng(w * 100 + h)
    light = r.uniform(-0.1, 2.0, (h, w, 4)).astype(np.float32)
    normal = r.normal(0.0, 0.3, (h, w, 4)).astype(np.float32)
    moments = r.uniform(0.5, 0.6, (h, w, 2)).astype(np.float32)
    if kind != "smooth":  # exponents to about 130, past the largest that is not 0
        moments[..., 0] = r.uniform(0.0, 12.0, (h, w))
    if kind == "special":
        values = np.array([np.inf, -np.inf, np.nan, 3e38, -0.0, 1e-40], np.float32)
        for a in (moments, normal):
            at = r.random(a.shape) < 0.02
            a[at] = r.choice(values, int(at.sum()))
    dev = lambda a: cuda.from_numpy(a).cuda()
    out = cuda.full((h, w, 4), -7.0, dtype=cuda.float32, device="cuda")
    gi.bilateral(dev(light), dev(moments), dev(normal), out)
    cuda.cuda.synchronize()
    np.testing.assert_array_equal(out.cpu().numpy(), oracle.bilateral(light, moments, normal))


@pytest.mark.parametrize("w,h", [(1, 1), (5, 3), (2, 9), (32, 16), (33, 17), (31, 15), (70, 34)])
def test_final_gather_equals_the_oracle(gi, oracle, cuda, w, h):
    r = np.random.default_rng(w * 100 + h)
    direct, light, albedo = (r.uniform(-0.1, 2.0, (h, w, 4)).astype(np.float32) for _ in range(3))
    dev = lambda a: cuda.from_numpy(a).cuda()
    out = cuda.full((h, w, 4), -7.0, dtype=cuda.float32, device="cuda")
    gi.final_gather(dev(direct), dev(light), dev(albedo), out)
    cuda.cuda.synchronize()
    np.testing.assert_array_equal(out.cpu().numpy(), oracle.final_gather(direct, light, albedo))
