"""What a program that uses the library has it do, as cases to time.

Every case is one use of the public entry points (legitengine_gb300.gi) over a
seeded procedural room: whole frames through the renderer and the batch, and the
single passes they are made of through their own calls.  The rooms, their
G-buffers and the 64-bit values are evaluated here with plain torch.
"""
import math

import numpy as np
import torch

from legitengine_gb300 import gi
from legitengine_gb300.train_reconstructor import DEFAULT_WEIGHTS

EXACT, FAST, TEXTURE = gi.GI_MARCH_EXACT, gi.GI_MARCH_FAST, gi.GI_MARCH_TEXTURE
PRECISION = {"exact": EXACT, "fast": FAST, "texture": TEXTURE}
PATTERN = 4          # the reference's interleave pattern edge
MIPS = 10            # the reference's requested mip levels
SHADOW = 1024        # shadow map edge
PI_REF = 3.1415      # the shader's pi
AMBIENT = 0.01
BATCH_RES = [(256, 256), (640, 480), (1280, 720), (1920, 1080)]


def listed():
    return [
        # A small view (a probe, a preview, a test): launches and latency count.
        dict(name="frame_small", op="frame", w=256, h=144, dirs=8, cap=32, bounces=2, prec="exact", boxes=16, spheres=0),
        # The frame of a 1080p application: two bounces, taps through the texture units.
        dict(name="frame_1080p", op="frame", w=1920, h=1080, dirs=16, cap=64, bounces=2, prec="texture", boxes=64,
             spheres=16),
        # The same application with the learned reconstructor and its judge.
        dict(name="learned_1080p", op="learned", w=1920, h=1080, dirs=16, cap=64, bounces=2, prec="texture", boxes=64,
             spheres=16),
        # Many views of uneven size in one call (probes, split screen, dataset rendering).
        dict(name="batch_mixed", op="batch", views=6, low=8, high=32, cap=64, prec="texture", boxes=48, spheres=12),
        # The march alone as a renderer of one's own calls it: the 512x512 room in the exact contract,
        dict(name="march_room", op="march", w=512, h=512, dirs=8, cap=32, prec="exact", boxes=16, spheres=0),
        # and a window of an odd size in the fast precision.
        dict(name="march_odd_fast", op="march", w=1283, h=721, dirs=12, cap=40, prec="fast", boxes=64, spheres=16),
        # The interleaved form: deinterleave the G-buffer, march sub-images with the reference's four directions,
        # interleave the result.
        dict(name="interleaved_720p", op="interleaved", w=1280, h=720, dirs=4, cap=0, prec="exact", boxes=64, spheres=16),
        # Mip chains and blur pyramids of the light and of the depth moments.
        dict(name="pyramids_1080p", op="pyramids", w=1920, h=1080, boxes=64, spheres=16),
        # The passes after the march at 4K: bilateral filter and gather.
        dict(name="filters_4k", op="filters", w=3840, h=2160, boxes=64, spheres=16),
        # The passes before it: G-buffer, shadow map and direct light.
        dict(name="inputs_1080p", op="inputs", w=1920, h=1080, boxes=64, spheres=16),
        # The fused reconstruction of a frame whose few-ray light is in hand.
        dict(name="reconstruct_1080p", op="reconstruct", w=1920, h=1080, boxes=64, spheres=16),
        # A training batch of the reconstructor: loss and gradients.
        dict(name="gradients_16k", op="gradients", n=16384, loss="absolute"),
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["frame", "frame", "learned", "batch", "march", "march", "interleaved", "pyramids", "filters",
                     "inputs", "reconstruct", "gradients"])
    boxes = spread(8, 100)
    scene = dict(boxes=boxes, spheres=boxes // 4)
    w, h = spread(200, 1920), spread(120, 1080)
    if op == "frame":
        dirs, bounces = rng.randint(4, 16), rng.randint(1, 2)
        prec = rng.choice(["texture", "texture", "fast", "exact"])
        if prec != "texture":  # no dearer than the largest listed frame
            dirs = min(dirs, 8)
        return dict(op=op, w=w, h=h, dirs=dirs, cap=rng.choice([0, 32, 64]), bounces=bounces, prec=prec, **scene)
    if op == "learned":
        return dict(op=op, w=w, h=h, dirs=rng.randint(8, 24), cap=64, bounces=rng.randint(1, 2),
                    prec=rng.choice(["texture", "texture", "fast"]), **scene)
    if op == "batch":
        return dict(op=op, views=rng.randint(2, 6), low=8, high=rng.randint(8, 24), cap=64,
                    prec=rng.choice(["texture", "texture", "fast"]), **scene)
    if op == "march":
        return dict(op=op, w=w, h=h, dirs=rng.randint(2, 16), cap=rng.choice([0, 32, 64]),
                    prec=rng.choice(["exact", "fast", "texture"]), **scene)
    if op == "interleaved":
        return dict(op=op, w=w // 4 * 4, h=h // 4 * 4, dirs=rng.randint(2, 12), cap=0, prec="exact", **scene)
    if op == "gradients":
        return dict(op=op, n=spread(1000, 65536), loss=rng.choice(["absolute", "squared"]))
    if op in ("pyramids", "filters", "inputs"):
        w, h = spread(200, 3840), spread(120, 2160)
    return dict(op=op, w=w, h=h, **scene)


# ---------------------------------------------------------------------------
# Views, and their G-buffer and direct light in 64 bits.

def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t64(a):
    return torch.as_tensor(np.asarray(list(a), np.float64), device=_dev())


def _scene(case, seed, k=0):
    prims = gi.scene_generate(1000 + 101 * seed + k, case["boxes"], case["spheres"])
    return prims, gi.camera_spline(7 + seed + 13 * k, (11 * seed + 5 * k) % 64, 64, prims)


def _grid(w, h):
    d = _dev()
    x = torch.arange(w, device=d, dtype=torch.float64) + 0.5
    y = torch.arange(h, device=d, dtype=torch.float64) + 0.5
    return (x / w).expand(h, w), (y / h)[:, None].expand(h, w)


def _mul(m, x, y, z, w):
    """Rows of the column-major matrix m times (x, y, z, w)."""
    m = [float(v) for v in m]
    return [m[r] * x + m[4 + r] * y + m[8 + r] * z + m[12 + r] * w for r in range(4)]


def _dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


def _sub(a, b):
    return [a[k] - b[k] for k in range(3)]


def _cross(a, b):
    return [a[1] * b[2] - b[1] * a[2], a[2] * b[0] - b[2] * a[0], a[0] * b[1] - b[0] * a[1]]


def _unit(a):
    r = 1.0 / torch.sqrt(_dot(a, a))
    return [v * r for v in a]


def _unproject(m, sx, sy, z):
    v = _mul(m, sx * 2 - 1, sy * 2 - 1, z, 1.0)
    return [v[k] / v[3] for k in range(3)]


def _cast(view, prims):
    """Nearest hit of the pixels' rays: origin, direction, distance, normal, primitive (-1: none)."""
    sx, sy = _grid(view.width, view.height)
    o = [float(v) for v in view.inv_view[12:15]]
    d = _unit(_sub(_unproject(view.inv_view_proj, sx, sy, 1.0), o))
    best = torch.full_like(sx, math.inf)
    prim = torch.full_like(sx, -1, dtype=torch.int64)
    n = torch.zeros(3, *sx.shape, dtype=torch.float64, device=sx.device)
    iv = [1.0 / v for v in d]
    for i, p in enumerate(prims):
        a, b = [float(v) for v in p.a], [float(v) for v in p.b]
        if p.kind == gi.GI_PRIM_SPHERE:
            oc = [o[k] - a[k] for k in range(3)]
            bb = _dot(oc, d)
            disc = bb * bb - (_dot(oc, oc) - b[0] * b[0])
            t = -bb - torch.sqrt(disc.clamp(min=0))
            near = (disc >= 0) & (t > 0) & (t < best)
            nn = _unit([o[k] + d[k] * t - a[k] for k in range(3)])
        else:
            lo, hi = [], []
            for k in range(3):
                u, v = (a[k] - o[k]) * iv[k], (b[k] - o[k]) * iv[k]
                lo.append(torch.minimum(u, v))
                hi.append(torch.maximum(u, v))
            if p.kind == gi.GI_PRIM_ROOM:
                t, axis = torch.stack(hi).min(0)
                near = (t > 0) & (t < best)
            else:
                t, axis = torch.stack(lo).max(0)
                near = (t <= torch.minimum(torch.minimum(hi[0], hi[1]), hi[2])) & (t > 0) & (t < best)
            nn = [torch.where(axis == k, torch.where(d[k] > 0, -1.0, 1.0), 0.0) for k in range(3)]
        best = torch.where(near, t, best)
        prim[near] = i
        n = torch.where(near, torch.stack(nn), n)
    return o, d, best, n, prim


def _gbuffer(view, prims):
    o, d, t, n, prim = _cast(view, prims)
    miss = prim < 0
    t = torch.where(miss, 0.0, t)
    hit = [o[k] + d[k] * t for k in range(3)]
    dist = torch.sqrt(_dot(_sub(hit, o), _sub(hit, o)))
    q = _mul(view.view_proj, *hit, 1.0)
    colour = lambda f: torch.as_tensor(np.array([list(getattr(p, f)) for p in prims], np.float64) ** 2.2,
                                       device=t.device)[prim.clamp(min=0)] * (~miss)[..., None]
    one = (~miss).to(torch.float64)
    return dict(albedo=colour("albedo"), emissive=colour("emissive"), normal=torch.stack([*n, one], -1),
                moments=torch.stack([dist, dist * dist], -1) * one[..., None],
                ndc=torch.where(miss, 1.0, q[2] / q[3])[..., None])


def _shadow(light, prims):
    o, d, t, _, prim = _cast(light, prims)
    t = torch.where(prim < 0, 0.0, t)
    q = _mul(light.view_proj, *[o[k] + d[k] * t for k in range(3)], 1.0)
    return torch.where(prim < 0, 1.0, q[2] / q[3])[..., None]


def _direct(view, light, g, shadow):
    sx, sy = _grid(view.width, view.height)
    p = _unproject(view.inv_view_proj, sx, sy, g["ndc"][..., 0])
    to = _sub(p, [float(v) for v in light.inv_view[12:15]])
    diffuse = (-_dot(_unit(to), g["normal"].unbind(-1))).clamp(min=0)
    q = _mul(light.view_proj, *p, 1.0)
    u, v, z = q[0] / q[3] * 0.5 + 0.5, q[1] / q[3] * 0.5 + 0.5, q[2] / q[3] - 2e-4
    radius = torch.sqrt((u - 0.5) ** 2 + (v - 0.5) ** 2) * 2
    s = 1 - ((radius - 0.6) / 0.4).clamp(0, 1)
    cone = s * s * (3 - 2 * s) * (_mul(light.view, *p, 1.0)[2] > 0)
    lit = _taps(shadow, u, v, lambda t: (z <= t[..., 0]).to(torch.float64)[..., None])[..., 0]
    li = 5 * cone * lit ** 2.2
    rgb = (diffuse * li)[..., None] * g["albedo"][..., :3] + g["emissive"][..., :3]
    return torch.cat([rgb, torch.ones_like(rgb[..., :1])], -1)


def _taps(img, s, t, f=lambda v: v):
    """Bilinear, clamp-to-edge sample of img [h, w, c] at normalised coordinates; f maps each texel first."""
    h, w = img.shape[:2]
    u, v = (s * w - 0.5).clamp(-1e6, 1e6), (t * h - 0.5).clamp(-1e6, 1e6)
    i, j = u.floor(), v.floor()
    a, b = (u - i)[..., None], (v - j)[..., None]
    i, j = i.long(), j.long()
    i0, i1, j0, j1 = i.clamp(0, w - 1), (i + 1).clamp(0, w - 1), j.clamp(0, h - 1), (j + 1).clamp(0, h - 1)
    return (f(img[j0, i0]) * (1 - a) * (1 - b) + f(img[j0, i1]) * a * (1 - b) +
            f(img[j1, i0]) * (1 - a) * b + f(img[j1, i1]) * a * b)


def _view(case, seed, k=0, size=None):
    prims, cam = _scene(case, seed, k)
    w, h = size or (case["w"], case["h"])
    return prims, gi.view_from_camera(cam, w, h), gi.view_from_camera(gi.scene_light(), SHADOW, SHADOW)


def _images(case, seed, k=0, size=None):
    """The view and its five input images as a program has them: fp32, on the device."""
    prims, view, light = _view(case, seed, k, size)
    g = _gbuffer(view, prims)
    g["direct"] = _direct(view, light, g, _shadow(light, prims))
    return view, {n: g[n].float().contiguous() for n in ("albedo", "normal", "moments", "ndc", "direct")}


# ---------------------------------------------------------------------------
# The GI passes in plain torch (64 bits where the images are).

def _mips(img, levels):
    out = [img]
    for _ in range(1, levels):
        p = out[-1]
        h, w = p.shape[0] // 2 * 2, p.shape[1] // 2 * 2
        out.append((p[0:h:2, 0:w:2] + p[0:h:2, 1:w:2] + p[1:h:2, 0:w:2] + p[1:h:2, 1:w:2]) / 4)
    return out


def _blur(img):
    h, w = img.shape[:2]
    rows = [torch.arange(h, device=img.device).add(d).clamp(0, h - 1) for d in (-2, -1, 0, 1)]
    cols = [torch.arange(w, device=img.device).add(d).clamp(0, w - 1) for d in (-2, -1, 0, 1)]
    v = sum(img[:, c] for c in cols)
    return sum(v[r] for r in rows) / 16


def _pyramid(img, levels):
    m = _mips(img, levels)
    return m, [m[0]] + [_blur(v) for v in m[1:]]


def _levels(w, h):
    return min(MIPS, int(math.log2(min(w, h))) + 1)


def _reverse16(i):
    return int(format(i, "032b")[::-1], 2) / float(0xffffffff)


def _trilinear(flat, base, sizes, s, t, lam):
    """Trilinear samples of a pyramid laid flat; lam: level of detail per sample."""
    lo = lam.floor().long()
    delta = lam - lo
    r = 0
    for lev, wt in ((lo, 1 - delta), ((lo + 1).clamp(max=len(base) - 1), delta)):
        w, h = sizes[lev, 0], sizes[lev, 1]
        u, v = s * w - 0.5, t * h - 0.5
        i, j = u.floor(), v.floor()
        a, b = u - i, v - j
        zero = torch.zeros_like(lev)
        i, j = i.clamp(-1e6, 1e6).long(), j.clamp(-1e6, 1e6).long()
        i0, i1 = torch.maximum(torch.minimum(i, w - 1), zero), torch.maximum(torch.minimum(i + 1, w - 1), zero)
        j0, j1 = torch.maximum(torch.minimum(j, h - 1), zero), torch.maximum(torch.minimum(j + 1, h - 1), zero)
        row0, row1 = base[lev] + j0 * w, base[lev] + j1 * w
        for at, k in ((row0 + i0, (1 - a) * (1 - b)), (row0 + i1, a * (1 - b)), (row1 + i0, (1 - a) * b),
                      (row1 + i1, a * b)):
            k = k * wt
            r = r + flat[at] * (k[..., None] if flat.dim() > 1 else k)
    return r


def _march(view, dirs, cap, step_dirs, light, depth, normal, ndc):
    """The march of SSVGI/indirectLighting.frag in 64 bits."""
    w, h, n_lev = view.width, view.height, len(light)
    d = _dev()
    sizes = torch.tensor([[v.shape[1], v.shape[0]] for v in light], device=d)
    base = torch.tensor(np.cumsum([0] + [v.shape[0] * v.shape[1] for v in light])[:-1], device=d)
    flat_l = torch.cat([v[..., :3].reshape(-1, 3) for v in light]).double()
    flat_d = torch.cat([v[..., 0].reshape(-1) for v in depth]).double()
    sx, sy = _grid(w, h)
    cx, cy = sx * w, sy * h
    pat = (torch.arange(w, device=d) % PATTERN)[None, :] + (torch.arange(h, device=d) % PATTERN)[:, None] * PATTERN
    n_pat = PATTERN * PATTERN
    ang = pat.double() / n_pat
    lin = torch.tensor([_reverse16(i) for i in range(n_pat)], device=d, dtype=torch.float64)[pat]
    cam = [float(v) for v in view.inv_view[12:15]]
    z = ndc[..., 0].double()
    nrm = normal[..., :3].double().unbind(-1)
    cwp = _unproject(view.inv_view_proj, sx, sy, z)
    ed = _unit([cam[k] - cwp[k] for k in range(3)])
    ed_in = [-v for v in ed]
    near, growth = w / 1000.0, 2 * PI_REF / step_dirs
    total = torch.zeros(h, w, 3, device=d, dtype=torch.float64)

    def contribution(qd, qt, lo, hi):
        return qd * (torch.cos(2 * lo) - torch.cos(2 * hi)) + qt * (2 * hi - 2 * lo - torch.sin(2 * hi) + torch.sin(2 * lo))

    for k in range(dirs):
        a = 2 * PI_REF / dirs * (ang + k)
        dx, dy = torch.cos(a), torch.sin(a)
        owp = _unproject(view.inv_view_proj, (cx + dx) / w, (cy + dy) / h, z)
        et = _unit(_sub(_unit(_sub(owp, cam)), ed_in))
        c = _cross(et, ed)
        dnp = _cross([-v for v in c], nrm)
        top = torch.atan2(_dot(dnp, et), _dot(dnp, ed))
        qd, qt = 0.25 * _dot(ed, nrm), 0.25 * _dot(et, nrm)
        light_k = (AMBIENT * contribution(qd, qt, torch.zeros_like(top), top))[..., None].repeat(1, 1, 3)
        path = torch.minimum(torch.maximum(-cx / dx, (w - cx) / dx), torch.maximum(-cy / dy, (h - cy) / dy)).abs()
        steps = (torch.log(path / near) / math.log(growth + 1)).trunc() + 1
        if cap > 0:
            steps = steps.clamp(max=cap)
        for s in range(int(steps.max())):
            off = near * (growth + 1) ** (s + lin) + 1 - near
            px, py = (cx + dx * off) / w, (cy + dy * off) / h
            lam = (torch.log2((growth * (off - 1) * 0.5).clamp(min=0)) - 2).clamp(0, n_lev - 1)
            ray = _unit(_sub(_unproject(view.inv_view_proj, px, py, 1.0), cam))
            dist = _trilinear(flat_d, base, sizes, px, py, lam)
            wd = [cam[q] + ray[q] * dist - cwp[q] for q in range(3)]
            at = torch.atan2(_dot(et, wd), _dot(ed, wd))
            hit = (at < top) & (s < steps)
            edge = lambda v: (v / 0.1).clamp(0, 1)
            hc = contribution(qd, qt, at, top) * edge(1 - px) * edge(px) * edge(1 - py) * edge(py)
            sel = hit.nonzero(as_tuple=True)
            light_k[sel] += (_trilinear(flat_l, base, sizes, px[sel], py[sel], lam[sel]) - AMBIENT) * hc[sel][:, None]
            top = torch.where(hit, at, top)
        total += 2 * light_k / dirs
    return torch.cat([total, torch.ones_like(total[..., :1])], -1)


def _bilateral(ind, moments, normal):
    h, w = ind.shape[:2]
    acc, wsum = 0, 0
    for dy in range(-2, 3):
        r = torch.arange(h, device=ind.device).add(dy).clamp(0, h - 1)
        for dx in range(-2, 3):
            c = torch.arange(w, device=ind.device).add(dx).clamp(0, w - 1)
            q = lambda v: v[r][:, c]
            k = torch.exp(-(q(moments[..., 0]) - moments[..., 0]).abs() * 10.5) * \
                torch.exp(-((q(normal) - normal)[..., :3] ** 2).sum(-1) * 20)
            acc = acc + q(ind)[..., :3] * k[..., None]
            wsum = wsum + k
    out = acc / (wsum + 1e-7)[..., None]
    return torch.cat([out, torch.ones_like(out[..., :1])], -1)


def _net():
    """The shipped reconstructor's weights in 64 bits."""
    flat = np.fromfile(DEFAULT_WEIGHTS, np.float32, offset=16, count=10627).astype(np.float64)
    out, o = [], 0
    for shape in ((32, 64), (64,), (64, 64), (64,), (64, 64), (64,), (64, 3), (3,)):
        out.append(torch.as_tensor(flat[o:o + math.prod(shape)].reshape(shape), device=_dev()))
        o += math.prod(shape)
    return out


def _blend(net, x):
    """The network's softmax blend of the three candidate estimates in the rows x."""
    y = x
    for k in range(3):
        y = torch.relu(y @ net[2 * k] + net[2 * k + 1])
    p = torch.softmax(y @ net[6] + net[7], -1)
    return sum(p[:, k:k + 1] * x[:, c:c + 3] for k, c in enumerate((10, 19, 22)))


def _lum(c):
    return 0.2126 * c[..., 0] + 0.7152 * c[..., 1] + 0.0722 * c[..., 2]


def _reconstruct(g, few, filtered, depth_l2):
    """Features and network of a frame; few: the few-ray light at mip levels 0, 2 and 4."""
    h, w = few[0].shape[:2]
    s, t = _grid(w, h)
    x, y = torch.arange(w, device=s.device), torch.arange(h, device=s.device)
    i2, i4 = _taps(few[1], s, t), _taps(few[2], s, t)
    near = [_lum(few[0][(y + b).clamp(0, h - 1)][:, (x + a).clamp(0, w - 1)])
            for a, b in ((-1, 0), (1, 0), (0, -1), (0, 1), (-1, -1), (1, 1))]
    scale = _lum(i2).abs() + _lum(i4).abs() + 1e-3
    norm = lambda v: (v / scale[..., None]).clamp(-32, 32)
    m = depth_l2[(y // 4).clamp(max=h // 4 - 1)][:, (x // 4).clamp(max=w // 4 - 1)]
    pat = (x % PATTERN)[None, :] + (y % PATTERN)[:, None] * PATTERN
    rev = torch.tensor([_reverse16(i) for i in range(PATTERN * PATTERN)], device=s.device, dtype=torch.float64)[pat]
    rows = torch.cat([
        g["moments"][..., :1], g["normal"][..., :3], g["albedo"][..., :3], norm(few[0][..., :3]),
        norm(filtered[..., :3]), norm(torch.stack(near, -1)), norm(i2[..., :3]), norm(i4[..., :3]),
        torch.sqrt((m[..., 1] - m[..., 0] ** 2).clamp(min=0))[..., None], norm(g["direct"][..., :3]),
        pat[..., None] / float(PATTERN * PATTERN), rev[..., None],
        torch.minimum(torch.minimum(s, 1 - s), torch.minimum(t, 1 - t))[..., None]], -1)
    out = _blend(_net(), rows.reshape(h * w, 32)).reshape(h, w, 3) * scale[..., None]
    return torch.cat([out, torch.ones_like(out[..., :1])], -1)


def _frame(view, img, dirs, cap, bounces, learned=False):
    """A whole frame: lit image and the last bounce's filtered indirect light."""
    g = {k: v.double() for k, v in img.items()}
    n = _levels(view.width, view.height)
    depth = _pyramid(g["moments"], n)[1]
    lit = g["direct"]
    for _ in range(bounces):
        light = _pyramid(lit, n)[1]
        if learned:
            raw = _march(view, 1, cap, 32, light, depth, g["normal"], g["ndc"])
            few = _mips(raw, 5)
            ind = _reconstruct(dict(g, direct=lit), few[0::2], _bilateral(raw, g["moments"], g["normal"]), depth[2])
        else:
            ind = _bilateral(_march(view, dirs, cap, dirs, light, depth, g["normal"], g["ndc"]), g["moments"], g["normal"])
        lit = g["direct"] + ind * g["albedo"]
    return [lit, ind]


# ---------------------------------------------------------------------------
# The cases.

_stream = None


def _frames_stream():
    """The stream a renderer's frames are replayed on (captured graphs need one of their own)."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


def _empty(h, w, c):
    return torch.empty(h, w, c, dtype=torch.float32, device="cuda")


def _few_light(view, g, seed):
    """A noisy few-ray light as the reconstruction meets it: the direct light's coarse mips,
    modulated per pixel (one direction per pixel sees a part of them), dark and bright frames."""
    r = torch.Generator(device=_dev()).manual_seed(seed)
    n = torch.rand(view.height, view.width, 1, generator=r, device=_dev(), dtype=torch.float64)
    s, t = _grid(view.width, view.height)
    soft = _taps(_mips(g["direct"].double(), _levels(view.width, view.height))[4], s, t)
    return torch.cat([(soft * (0.02 + 0.6 * n * n))[..., :3], torch.ones_like(n)], -1).float()


def _batch_views(case, seed):
    """Sizes and directions of a batch's views: every view count has large and small ones."""
    r = np.random.RandomState(len(str(case)) + case["views"])
    sizes = [BATCH_RES[(i + 1) % len(BATCH_RES)] for i in range(case["views"])]
    return [(s, int(r.randint(case["low"], case["high"] + 1))) for s in sizes]


def _rows(case, seed):
    """Feature rows of a training batch (bf16), their targets (rgb, loss weight) and exposure scales."""
    r = torch.Generator(device=_dev()).manual_seed(seed)
    n = case["n"]
    u = lambda c: torch.rand(n, c, generator=r, device=_dev(), dtype=torch.float64)
    g = lambda c: torch.randn(n, c, generator=r, device=_dev(), dtype=torch.float64)
    nrm = g(3)
    light = torch.exp(0.5 * g(1)) * (0.5 + u(3))  # normalised light, about 1
    near = lambda k: (light * torch.exp(k * g(3))).clamp(-32, 32)
    x = torch.cat([0.1 + u(1), nrm / nrm.norm(dim=1, keepdim=True), 0.05 + 0.75 * u(3), near(1.0), near(0.2),
                   near(1.0), near(1.0), near(0.05), near(0.1), 0.1 * u(1) ** 2, near(1.0),
                   torch.floor(16 * u(1)) / 16, u(1), 0.5 * u(1)], 1).to(torch.bfloat16)
    scale = torch.exp(g(1) - 2)
    target = torch.cat([light * scale * torch.exp(0.1 * g(3)), scale / scale.mean()], 1)
    return x.contiguous(), target.float().contiguous(), scale[:, 0].float().contiguous()


def _network():
    net = gi.Mlp(seed=None)
    net.load(DEFAULT_WEIGHTS)
    return net


def prepare(case, seed):
    op = case["op"]
    if op == "gradients":
        x, t, s = _rows(case, seed)
        net = _network()
        net.set_loss(gi.GI_MLP_LOSS_ABSOLUTE if case["loss"] == "absolute" else gi.GI_MLP_LOSS_SQUARED)
        return dict(case=case, net=net, x=x, t=t, s=s)
    if op == "batch":
        specs = []
        for k, ((w, h), dirs) in enumerate(_batch_views(case, seed)):
            view, img = _images(case, seed, k, (w, h))
            specs.append(dict(view=view, march=gi.GiMarchParams(dirs, case["cap"], PATTERN, 0, PRECISION[case["prec"]]),
                              out_lit=_empty(h, w, 4), out_indirect=_empty(h, w, 4), **img))
        return dict(case=case, specs=specs, batch=gi.Batch(specs, tile_rows=0))
    w, h = case["w"], case["h"]
    if op == "inputs":
        prims, view, light = _view(case, seed)
        dev, count = gi.prims_to_device(prims)
        out = dict(albedo=_empty(h, w, 4), emissive=_empty(h, w, 4), normal=_empty(h, w, 4), moments=_empty(h, w, 2),
                   ndc=_empty(h, w, 1), shadow=_empty(SHADOW, SHADOW, 1), direct=_empty(h, w, 4))
        return dict(case=case, view=view, light=light, prims=dev, count=count, out=out)
    view, img = _images(case, seed)
    st = dict(case=case, view=view, lit=_empty(h, w, 4), ind=_empty(h, w, 4), **img)
    n = gi.mip_level_count(w, h, MIPS)
    if op in ("frame", "learned"):
        st["renderer"] = gi.Renderer(w, h, dirs=case["dirs"], step_cap=case["cap"], bounces=case["bounces"],
                                     bilateral=True, precision=PRECISION[case["prec"]])
        if op == "learned":
            st["net"] = _network()
            st["renderer"].set_learned(st["net"], few_dirs=1, few_step_dirs=32, judge_every=64, threshold=0.25)
    elif op in ("march", "interleaved"):
        st["params"] = gi.GiMarchParams(case["dirs"], case["cap"], PATTERN, 0, PRECISION[case["prec"]])
        st["light"] = [v.contiguous() for v in _pyramid(img["direct"], n)[1]]
        st["depth"] = [v.contiguous() for v in _pyramid(img["moments"], n)[1]]
        if op == "interleaved":
            st.update(normal_d=_empty(h, w, 4), ndc_d=_empty(h, w, 1), out_d=_empty(h, w, 4))
    elif op == "pyramids":
        for name, ch in (("direct", 4), ("moments", 2)):
            st[name + "_mips"] = [img[name]] + gi.alloc_pyramid(w, h, ch, n)[1:]
            st[name + "_blur"] = [img[name]] + gi.alloc_pyramid(w, h, ch, n)[1:]
    elif op == "filters":
        st["few"] = _few_light(view, img, seed)
    elif op == "reconstruct":
        st["net"] = _network()
        st["few"] = [v.contiguous() for v in _mips(_few_light(view, img, seed), 5)][0::2]
        st["filtered"] = _bilateral(st["few"][0].double(), img["moments"].double(), img["normal"].double()).float()
        st["depth_l2"] = _pyramid(img["moments"], 3)[1][2].contiguous()
    return st


def run(s):
    op = s["case"]["op"]
    if op in ("frame", "learned"):
        with torch.cuda.stream(_frames_stream()):
            s["renderer"].render(s["view"], s["albedo"], s["normal"], s["moments"], s["ndc"], s["direct"], s["lit"], s["ind"])
        return [s["lit"], s["ind"]]
    if op == "batch":
        with torch.cuda.stream(_frames_stream()):
            s["batch"].render()
        return [[v["out_lit"], v["out_indirect"]] for v in s["specs"]]
    if op == "march":
        gi.march(s["view"], s["params"], s["light"], s["depth"], s["normal"], s["ndc"], s["ind"])
        return s["ind"]
    if op == "interleaved":
        gi.deinterleave(s["normal"], s["normal_d"])
        gi.deinterleave(s["ndc"], s["ndc_d"])
        gi.march(s["view"], s["params"], s["light"], s["depth"], s["normal_d"], s["ndc_d"], s["out_d"], deinterleaved=True)
        gi.interleave(s["out_d"], s["ind"])
        return s["ind"]
    if op == "pyramids":
        out = []
        for name, ch in (("direct", 4), ("moments", 2)):
            gi.build_mips(s[name + "_mips"], ch)
            gi.blur_pyramid(s[name + "_mips"], s[name + "_blur"])
            out.append([s[name + "_mips"][1:], s[name + "_blur"][1:]])
        return out
    if op == "filters":
        gi.bilateral(s["few"], s["moments"], s["normal"], s["ind"])
        gi.final_gather(s["direct"], s["ind"], s["albedo"], s["lit"])
        return [s["ind"], s["lit"]]
    if op == "inputs":
        o = s["out"]
        gi.gbuffer(s["view"], s["prims"], s["count"], o["albedo"], o["emissive"], o["normal"], o["moments"], o["ndc"])
        gi.shadow_map(s["light"], s["prims"], s["count"], o["shadow"])
        gi.direct_light(s["view"], s["light"], o["albedo"], o["emissive"], o["normal"], o["ndc"], o["shadow"], o["direct"])
        return o
    if op == "reconstruct":
        s["net"].reconstruct(s["moments"], s["normal"], s["albedo"], s["direct"], s["few"], s["filtered"], s["depth_l2"],
                             s["ind"])
        return s["ind"]
    loss, grads = s["net"].gradients(s["x"], s["t"], s["s"])
    return [loss, grads]


def _march_work(w, h, dirs, cap, step_dirs):
    """Flops of a march: about 100 a step and 150 a direction, over paths to about 0.4 of the viewport."""
    steps = math.log(max(2.0, 0.4 * max(w, h) * 1000 / w)) / math.log(2 * PI_REF / step_dirs + 1) + 1
    return w * h * dirs * (150 + 100 * (min(steps, cap) if cap else steps))


def work(case):
    op = case["op"]
    if op == "gradients":
        return dict(bytes=case["n"] * 84 + 2 * 4 * 10627, flops=case["n"] * 3 * 20864)
    if op == "batch":
        b = f = 0
        for (w, h), dirs in _batch_views(case, 0):
            b += w * h * (60 + 32)
            f += _march_work(w, h, dirs, case["cap"], dirs) + w * h * 600
        return dict(bytes=b, flops=f)
    px = case["w"] * case["h"]
    if op == "frame":  # five inputs (60 B) and two images out; every bounce marches and filters
        return dict(bytes=px * 92, flops=case["bounces"] * (
            _march_work(case["w"], case["h"], case["dirs"], case["cap"], case["dirs"]) + px * 600))
    if op == "learned":
        return dict(bytes=px * 92, flops=case["bounces"] * (
            _march_work(case["w"], case["h"], 1, case["cap"], 32) + px * (600 + 20864) +
            _march_work(case["w"], case["h"], case["dirs"], case["cap"], case["dirs"]) / 64))
    if op == "march":  # normal, depth, both pyramids, the image
        return dict(bytes=px * (16 + 4 + 32 + 16), flops=_march_work(case["w"], case["h"], case["dirs"], case["cap"],
                                                                     case["dirs"]))
    if op == "interleaved":
        return dict(bytes=px * (16 + 4 + 32 + 16), flops=_march_work(case["w"], case["h"], case["dirs"], case["cap"],
                                                                     case["dirs"]))
    if op == "pyramids":  # level 0 read, a third of it written twice, 4 and 2 channels
        return dict(bytes=px * 24 * (1 + 2 / 3), flops=px * 24 / 4 / 3 * 20)
    if op == "filters":  # light, moments, normal, direct, albedo in; filtered and lit out
        return dict(bytes=px * (16 + 8 + 16 + 16 + 16 + 32), flops=px * 700)
    if op == "inputs":  # six images and the shadow map; a slab test a primitive and ray
        rays = px + SHADOW * SHADOW
        return dict(bytes=px * (16 * 4 + 8 + 4) + SHADOW * SHADOW * 4, flops=rays * (case["boxes"] + case["spheres"]) * 25)
    return dict(bytes=px * (8 + 16 * 4 + 16 * (1 + 1 / 16 + 1 / 256) + 8 / 16 + 16), flops=px * 20864)


def exact(case, seed):
    op = case["op"]
    if op == "gradients":
        x, t, s = _rows(case, seed)
        net = [v.requires_grad_(True) for v in _net()]
        x, t = x.double(), t.double()
        y, w = _blend(net, x), t[:, 3:4]
        e = y - t[:, :3] / s.double()[:, None]
        n = case["n"]
        if case["loss"] == "absolute":
            loss = drive = (w * e.abs()).sum()
        else:  # the gradient clips the error of an output to [-1, 1]
            loss, drive = (w * e * e).sum(), (2 * w * e.detach().clamp(-1, 1) * y).sum()
        grads = torch.autograd.grad(drive, net)
        return [float(loss.detach()) / (3 * n), torch.cat([v.reshape(-1) for v in grads]).cpu().numpy() / n]
    if op == "batch":
        out = []
        for k, (size, dirs) in enumerate(_batch_views(case, seed)):
            view, img = _images(case, seed, k, size)
            out.append(_frame(view, img, dirs, case["cap"], 1))
        return out
    if op == "inputs":
        prims, view, light = _view(case, seed)
        g = _gbuffer(view, prims)
        g["shadow"] = _shadow(light, prims)
        g["direct"] = _direct(view, light, g, g["shadow"])
        return g
    view, img = _images(case, seed)
    n = _levels(case["w"], case["h"])
    if op in ("frame", "learned"):
        return _frame(view, img, case["dirs"], case["cap"], case["bounces"], op == "learned")
    if op in ("march", "interleaved"):
        light, depth = ([v.double() for v in _pyramid(img[k], n)[1]] for k in ("direct", "moments"))
        return _march(view, case["dirs"], case["cap"], case["dirs"], light, depth, img["normal"], img["ndc"])
    if op == "pyramids":
        return [[v[1:] for v in _pyramid(img[k].double(), n)] for k in ("direct", "moments")]
    g = {k: v.double() for k, v in img.items()}
    few = _few_light(view, img, seed)
    if op == "filters":
        ind = _bilateral(few.double(), g["moments"], g["normal"])
        return [ind, g["direct"] + ind * g["albedo"]]
    filtered = _bilateral(few.double(), g["moments"], g["normal"]).float().double()
    return _reconstruct(g, [v.double() for v in _mips(few, 5)][0::2], filtered, _pyramid(img["moments"], 3)[1][2].double())
