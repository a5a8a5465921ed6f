"""The march at sizes where its tiles, warps and tables can go wrong: images
smaller than a warp's pixels, one row or column past a tile, odd rows in the last
tile, every CTA height, pattern sizes that do not divide the image, a step table
of hundreds of entries, and a single mip level.  The exact precision equals the
fp32 oracle bit for bit (the same operations in the same order); the texture
precision is held to the library's bar for it, 1e-3 relative L1 of the frame
against the oracle's texture-unit march."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(4, 4), (7, 3), (1, 9), (33, 17), (129, 33), (31, 130), (260, 36)]


def _case(gi, oracle, torch, w, h, levels=10):
    prims = gi.scene_generate(77, 6, 2)
    view = gi.view_from_camera(gi.camera_spline(5, 9, 64, prims), w, h)
    light = gi.view_from_camera(gi.scene_light(), 64, 64)
    gb = oracle.gbuffer(view, prims)
    direct = oracle.direct_light(view, light, gb, oracle.shadow_map(light, prims))
    n = gi.mip_level_count(w, h, levels)
    lb = oracle.blur_pyramid(oracle.mip_chain(direct, n))
    db = oracle.blur_pyramid(oracle.mip_chain(gb["moments"], n))
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()
    return view, gb, lb, db, [dev(x) for x in lb], [dev(x) for x in db], dev(gb["normal"]), dev(gb["ndc"])


def _march(gi, torch, c, params):
    view, _, _, _, l, d, nrm, ndc = c
    out = torch.full((view.height, view.width, 4), -7.0, dtype=torch.float32, device="cuda")
    gi.march(view, params, l, d, nrm, ndc, out)
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("w,h", SIZES)
@pytest.mark.parametrize("dirs,cap,pattern", [(1, 0, 4), (5, 7, 4), (8, 0, 3), (16, 64, 1)])
def test_exact_march_equals_oracle_at_edges(gi, oracle, cuda, w, h, dirs, cap, pattern):
    c = _case(gi, oracle, cuda, w, h)
    ref, _ = oracle.march(c[0], dirs, cap, c[2], c[3], c[1]["normal"], c[1]["ndc"], pattern=pattern)
    got = _march(gi, cuda, c, gi.GiMarchParams(dirs, cap, pattern))
    np.testing.assert_array_equal(got, ref)


@pytest.mark.parametrize("w,h", [(33, 17), (260, 36)])
@pytest.mark.parametrize("rows", [2, 4, 8])
def test_every_height_at_edges(gi, oracle, cuda, w, h, rows):
    c = _case(gi, oracle, cuda, w, h)
    for precision in (gi.GI_MARCH_EXACT, gi.GI_MARCH_FAST, gi.GI_MARCH_TEXTURE):
        p = gi.GiMarchParams(3, 41, 4, 0, precision)
        gi.march_set_layout(w, h, 3, 0, 41, precision, 4, 96)
        base = _march(gi, cuda, c, p)
        gi.march_set_layout(w, h, 3, 0, 41, precision, rows, 96)
        np.testing.assert_array_equal(_march(gi, cuda, c, p), base)


@pytest.mark.parametrize("w,h", SIZES)
def test_texture_march_at_edges(gi, oracle, cuda, w, h):
    c = _case(gi, oracle, cuda, w, h)
    ref, _ = oracle.march(c[0], 6, 40, c[2], c[3], c[1]["normal"], c[1]["ndc"],
                          tex=oracle.TEX_DEPTH | oracle.TEX_LIGHT)
    got = _march(gi, cuda, c, gi.GiMarchParams(6, 40, 4, 0, gi.GI_MARCH_TEXTURE))
    assert np.abs(got - ref).sum() <= 1e-3 * np.abs(ref[..., :3]).sum()


@pytest.mark.parametrize("precision", ["exact", "texture"])
def test_long_tables_and_one_level(gi, oracle, cuda, precision):
    """96 directions step without a cap (over a hundred table entries); one mip level."""
    c = _case(gi, oracle, cuda, 70, 50, levels=1)
    tex = precision == "texture"
    ref, steps = oracle.march(c[0], 96, 0, c[2], c[3], c[1]["normal"], c[1]["ndc"],
                              tex=(oracle.TEX_DEPTH | oracle.TEX_LIGHT) if tex else 0)
    assert steps.max() > 96 * 90
    got = _march(gi, cuda, c, gi.GiMarchParams(96, 0, 4, 0, gi.GI_MARCH_TEXTURE if tex else gi.GI_MARCH_EXACT))
    if tex:
        assert np.abs(got - ref).sum() <= 1e-3 * np.abs(ref[..., :3]).sum()
    else:
        np.testing.assert_array_equal(got, ref)
