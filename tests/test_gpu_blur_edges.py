"""The blur against the fp32 oracle, bit for bit, at images smaller than a tile, one row
or column past it and ragged ones, for the radius that takes four rows a thread (2, and
the copy, 0) and for others, windows wider than the image among them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (5, 3), (32, 8), (33, 9), (31, 33), (70, 34)])
@pytest.mark.parametrize("channels", [1, 2, 4])
@pytest.mark.parametrize("radius", [0, 1, 2, 3, 9, 64])
def test_blur_equals_the_oracle(gi, oracle, cuda, w, h, channels, radius):
    img = np.random.default_rng(w * 100 + h).uniform(-1.0, 2.0, (h, w, channels)).astype(np.float32)
    src = cuda.from_numpy(img).cuda()
    out = cuda.full((h, w, channels), -7.0, dtype=cuda.float32, device="cuda")
    gi.blur(src, out, radius)
    cuda.cuda.synchronize()
    np.testing.assert_array_equal(out.cpu().numpy(), oracle.blur(img, radius))
