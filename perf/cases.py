"""The workloads this framework's speed is judged on, each through its public entry points.

A case is a dict of plain values. ``listed()`` gives the fixed ones, ``draw(rng)`` more of the
same ranges, ``prepare(case, seed)`` what a program holds before the call, ``run(state)`` one
pass, ``work(case)`` the bytes and operations a pass cannot do without, and ``exact(case, seed)``
the pass's outputs in 64 bits from plain torch (the formulas of the photon splat, the refraction
of a height-field plate and the projected Landweber update, none of this package's code).
"""
import math

import torch
import torch.nn.functional as F

from shapefromcaustics_b200 import PDS, BatchedSplat, pds_backward, pds_forward
from shapefromcaustics_b200 import plate as plates
from shapefromcaustics_b200 import scene as scenes
from shapefromcaustics_b200 import synthetic
from shapefromcaustics_b200.caustics import splat_photons
from shapefromcaustics_b200.landweber import LandweberParams, landweber_update, photon_source

DEVICE = "cuda"
MPR = 20           # the largest footprint radius in pixels, the reference's default
FOOTPRINT_PX = 3.0  # initial footprint of the plate's photons in receiver pixels


def listed():
    # amp: the height of the plates' largest bump (mm). The plates that are differentiated have
    # the relief of a reconstruction's first iterations (it starts from a flat plate); the one
    # that is only rendered has the full relief, whose caustics fold.
    return [
        # The drop-in operator pair on the smallest image a test or a preview uses: 2^14
        # photons, where launches and host work are all there is.
        dict(name="pair_16k", kind="pair", n=2 ** 14, c=1, h=128, w=128, s_lo=0.5, s_hi=4.0),
        # The autograd Function on one ordinary simulation: 2^20 photons, 512^2.
        dict(name="autograd_1m", kind="autograd", n=2 ** 20, c=1, h=512, w=512, s_lo=0.5,
             s_hi=4.0),
        # Rendering only (no gradient): three colour channels of an odd-sized image.
        dict(name="render_rgb", kind="render", n=300007, c=3, h=333, w=517, s_lo=0.5, s_hi=4.0),
        # A focused caustic: 2^26 photons on 2048^2, most of them on four thin curves, with
        # footprints from a fraction of a pixel to the radius limit. The largest single call.
        dict(name="caustic_64m", kind="caustic", n=2 ** 26, h=2048, w=2048),
        # 64 simulations of uneven photon counts and image sizes through one plan.
        dict(name="batch_64", kind="batch", sims=64, n_lo=2 ** 16, n_hi=2 ** 22, edges="256,512,1024"),
        # A program with its own tracer: photons given by their receiver-plane differentials,
        # gradients back to the differentials, positions and fluxes.
        dict(name="traced_300k", kind="traced", n=300001, h=400, w=600, s_lo=0.5, s_hi=4.0),
        # One Landweber iteration on a small plate: 256^2 field, 4 photons a texel, 512^2.
        dict(name="landweber_256", kind="landweber", h=256, w=256, per_texel=4, image=512,
             amp=0.01),
        # One Landweber iteration of a full reconstruction: 1024^2 field, 16 simulations of 4
        # photons a texel (2^26 photons), 1024^2 image.
        dict(name="landweber_1024", kind="landweber", h=1024, w=1024, per_texel=64,
             image=1024, amp=0.01),
        # 64 simulations of one 256^2 plate, each with its own light tilt, wavelength, photon
        # count and image size: one batched forward and backward.
        dict(name="plate_batch_64", kind="plate_batch", sims=64, h=256, w=256, n_lo=2 ** 16,
             n_hi=2 ** 22, edges="256,512,1024", amp=0.01),
        # The plate under a point light: photons traced onto the height field, forward and
        # backward.
        dict(name="point_1m", kind="point", n=2 ** 20, h=256, w=256, image=512, amp=0.01),
        # A caustic preview of an odd-sized plate, no gradient (the target's rendering).
        dict(name="preview_200", kind="preview", h=201, w=167, per_texel=2, image=300, amp=0.05),
        # The projected update alone on the largest field (the reconstruction's other half).
        dict(name="update_1024", kind="update", h=1024, w=1024, radius=2, progress=0.6, amp=0.05),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pair", "autograd", "render", "caustic", "batch", "traced", "landweber",
                       "plate_batch", "point", "preview", "update"])
    if kind in ("pair", "autograd", "render", "traced"):
        c = rng.choice([1, 1, 3]) if kind != "traced" else 1
        lo, hi = rng.choice([(0.5, 4.0), (0.5, 8.0), (1.0, 2.0)])
        d = dict(kind=kind, n=_log(rng, 2 ** 12, 2 ** 22), c=c, h=_log(rng, 96, 1200),
                 w=_log(rng, 96, 1200), s_lo=lo, s_hi=hi)
        if kind == "traced":
            del d["c"]
        return d
    if kind == "caustic":
        return dict(kind=kind, n=_log(rng, 2 ** 18, 2 ** 25), h=_log(rng, 400, 2048),
                    w=_log(rng, 400, 2048))
    if kind in ("batch", "plate_batch"):
        d = dict(kind=kind, sims=rng.randint(3, 64), n_lo=_log(rng, 2 ** 12, 2 ** 16),
                 n_hi=_log(rng, 2 ** 17, 2 ** 21),
                 edges=rng.choice(["256,512,1024", "200,333,640", "128,500"]))
        if kind == "plate_batch":
            d["h"], d["w"] = rng.randint(96, 320), rng.randint(96, 320)
            d["amp"] = rng.choice([0.004, 0.007, 0.01])
        return d
    if kind == "point":
        return dict(kind=kind, n=_log(rng, 2 ** 14, 2 ** 22), h=_log(rng, 64, 700),
                    w=_log(rng, 64, 700), image=_log(rng, 128, 1024),
                    amp=rng.choice([0.004, 0.007, 0.01]))
    if kind == "update":
        return dict(kind=kind, h=_log(rng, 64, 2048), w=_log(rng, 64, 2048),
                    radius=rng.choice([1, 2, 2, 3]), progress=rng.choice([0.6, 1.0]),
                    amp=0.05)
    return dict(kind=kind, h=_log(rng, 64, 900), w=_log(rng, 64, 900),
                per_texel=rng.choice([1, 2, 4, 8, 16]), image=_log(rng, 128, 1100),
                amp=0.05 if kind == "preview" else rng.choice([0.004, 0.007, 0.01]))


# ------------------------------------------------------------------ inputs ---------------

def _normal(shape, seed):
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    return torch.randn(shape, generator=g, device=DEVICE)


def _photons(case, seed):
    if case["kind"] == "caustic":
        return synthetic.caustic_curve_photons(case["n"], case["h"], case["w"], seed=seed,
                                               device=DEVICE)
    ph = synthetic.uniform_cluster_photons(case["n"], case["h"], case["w"], seed=seed,
                                           s_range=(case["s_lo"], case["s_hi"]), device=DEVICE)
    c = case.get("c", 1)
    if c > 1:
        g = torch.Generator(device=DEVICE).manual_seed(seed + 1)
        ph = ph[:3] + (torch.randint(0, c, (1, case["n"]), generator=g, device=DEVICE),) + ph[4:]
    return ph


def _scene(h, w, **more):
    texel = 0.1
    return scenes.PlateScene(texel=texel, receiver_distance=50.0,
                             receiver_half=0.5 * max(h, w) * texel * 1.1, **more)


def _field(case, seed):
    return scenes.height_field_bumps(case["h"], case["w"], seed=seed, device=DEVICE,
                                     amp=(0.0, case["amp"]), dtype=torch.float32)


def _batch_specs(case):
    """Photon counts and image shapes of a batch: the case's alone, whatever the seed."""
    edges = tuple(int(v) for v in case["edges"].split(","))
    return synthetic.batch_specs(case["sims"], seed=1000 + case["sims"],
                                 n_range=(case["n_lo"], case["n_hi"]), sizes=edges)


def _plate_sims(case, seed):
    """(photons a texel, image shape, scene) of every simulation of a plate batch."""
    g = torch.Generator().manual_seed(seed + 5)
    sims = []
    for n, shape in _batch_specs(case):
        th, ph, lam = (float(v) for v in torch.rand(3, generator=g, dtype=torch.float64))
        th, ph, lam = math.radians(5.0) * th, 2 * math.pi * ph, 0.45 + 0.2 * lam
        light = (math.sin(th) * math.cos(ph), math.sin(th) * math.sin(ph), -math.cos(th))
        sc = _scene(case["h"], case["w"], ior=float(scenes.fused_silica(lam)), light_dir=light)
        sims.append((max(1, round(n / (case["h"] * case["w"]))), shape, sc))
    return sims


def _params(scene, image):
    return plates.plate_params(scene, FOOTPRINT_PX * 2.0 * scene.receiver_half / image)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("pair", "autograd", "render", "caustic"):
        s["photons"] = _photons(case, seed)
        s["shape"] = [case.get("c", 1), case["h"], case["w"]]
        if kind != "render":
            s["grad"] = _normal(s["shape"], seed + 2)
        if kind in ("autograd", "caustic"):
            for t in s["photons"][:3]:
                t.requires_grad_(True)
    elif kind == "batch":
        specs = _batch_specs(case)
        s["photons"] = synthetic.batch_photons(specs, seed=seed, device=DEVICE)
        s["batch"] = BatchedSplat(specs, MPR, DEVICE)
        s["grad"] = _normal(s["batch"].image_elems, seed + 2)
    elif kind == "traced":
        s.update(_traced(case, seed))
    elif kind in ("landweber", "preview"):
        h, w = case["h"], case["w"]
        sc = _scene(h, w)
        s.update(scene=sc, params=_params(sc, case["image"]), shape=(1, case["image"], case["image"]))
        n = h * w * case["per_texel"]
        s["flux"] = torch.full((n,), 1.0 / n, device=DEVICE)
        s["seed"] = seed
        s["d"] = _field(case, 7 * seed) - 1.0
        if kind == "landweber":
            s["mask"] = torch.ones(h, w, device=DEVICE)
            volume = float(s["d"].sum())
            s["update"] = LandweberParams(tau=1e-4, d1=0.75 * volume, d2=1.25 * volume)
            # the target: another field's caustic, from other photons
            px, py, _ = photon_source(h, w, case["per_texel"], sc.texel, seed + 99, 0, DEVICE)
            with torch.no_grad():
                s["target"] = plates.PlateSplat.apply(_field(case, 7 * seed + 1), px, py, s["flux"],
                                                      s["params"], s["shape"], MPR, False)
            s["scale"] = 1.0 / float((s["target"] ** 2).sum())
    elif kind == "plate_batch":
        sims = _plate_sims(case, seed)
        h, w = case["h"], case["w"]
        counts = [per * h * w for per, _, _ in sims]
        s["field"] = _field(case, 7 * seed)
        s["batch"] = plates.BatchedPlate([(n, shape, _params(sc, shape[1]))
                                          for n, (_, shape, sc) in zip(counts, sims)], MPR, DEVICE)
        parts, offset = [], 0
        for per, _, sc in sims:
            px, py, offset = photon_source(h, w, per, sc.texel, seed, offset, DEVICE)
            parts.append((px, py))
        s["px"], s["py"] = (torch.cat([p[k] for p in parts]) for k in (0, 1))
        s["flux"] = torch.cat([torch.full((n,), 1.0 / n, device=DEVICE) for n in counts])
        s["target"] = s["batch"].forward(_field(case, 7 * seed + 1), s["px"], s["py"], s["flux"])
    elif kind == "point":
        h, w = case["h"], case["w"]
        sc = _scene(h, w)
        hx, hy = 0.5 * (w - 2) * sc.texel, 0.5 * (h - 2) * sc.texel
        s["light"] = plates.point_light((0.0, 0.0, 400.0), (-hx, -hy, hx, hy), 1.0, 4.0, 1.0)
        s["light_photons"] = plates.point_light_source(s["light"], case["n"], DEVICE, seed=seed)[:4]
        s.update(scene=sc, params=_params(sc, case["image"]), shape=(1, case["image"], case["image"]))
        s["field"] = _field(case, 7 * seed)
        s["grad"] = _normal(s["shape"], seed + 2)
    elif kind == "update":
        h, w = case["h"], case["w"]
        full = _field(case, 7 * seed) - 1.0
        volume = float(full.sum())
        s["d"] = case["progress"] * full
        s["grad"] = _normal((h, w), seed + 2)
        s["mask"] = (_normal((h, w), seed + 3) > -2.0).float()
        s["update"] = LandweberParams(tau=1e-4, d1=0.75 * volume, d2=1.25 * volume,
                                      radius=case["radius"])
    return s


def _traced(case, seed):
    """Photons as a tracer gives them: receiver-plane differentials, normals, fluxes."""
    E, X, M, C, _ = _photons(case, seed)
    inv = torch.linalg.inv(M[:, :2].permute(2, 0, 1).double())  # D / 2 of Mp D = 2
    D = torch.zeros((2, 3, case["n"]), dtype=torch.float64, device=DEVICE)
    D[:, :2] = 2.0 * inv.permute(2, 1, 0)
    n = torch.zeros((3, case["n"]), device=DEVICE)
    n[2] = 1.0
    Du, Dv = D[0].float().contiguous(), D[1].float().contiguous()
    s = {"Du": Du, "Dv": Dv, "flux": (E * 1e-6).contiguous(), "xy": X}
    for t in s.values():
        t.requires_grad_(True)
    s.update(normal=n, channel=C[0].contiguous(), shape=(1, case["h"], case["w"]),
             grad=_normal((1, case["h"], case["w"]), seed + 2))
    return s


# ------------------------------------------------------------------ one pass -------------

def run(s):
    kind = s["case"]["kind"]
    if kind == "pair":
        return pds_forward(*s["photons"], s["shape"], MPR) + pds_backward(s["grad"], *s["photons"], MPR)
    if kind == "render":
        return pds_forward(*s["photons"], s["shape"], MPR)
    if kind in ("autograd", "caustic"):
        img = PDS.apply(*s["photons"], s["shape"], MPR)
        return [img.detach(), *torch.autograd.grad(img, s["photons"][:3], s["grad"])]
    if kind == "batch":
        s["batch"].plan(*s["photons"])
        return [s["batch"].forward(), *s["batch"].backward(s["grad"])]
    if kind == "traced":
        img = splat_photons(s["Du"], s["Dv"], s["normal"], s["flux"], s["xy"], s["channel"],
                            s["shape"], MPR)
        return [img.detach(), *torch.autograd.grad(img, [s[k] for k in ("Du", "Dv", "flux", "xy")],
                                                   s["grad"])]
    if kind == "landweber":
        c, sc = s["case"], s["scene"]
        px, py, _ = photon_source(c["h"], c["w"], c["per_texel"], sc.texel, s["seed"], 0, DEVICE)
        field = (1.0 + s["d"]).requires_grad_(True)
        img = plates.PlateSplat.apply(field, px, py, s["flux"], s["params"], s["shape"], MPR, True)
        diff = img - s["target"]
        (0.5 * s["scale"] * (diff * diff).sum()).backward()
        d = landweber_update(s["d"].clone(), field.grad, s["mask"], s["update"])
        return [img.detach(), field.grad, d]
    if kind == "preview":
        c, sc = s["case"], s["scene"]
        px, py, _ = photon_source(c["h"], c["w"], c["per_texel"], sc.texel, s["seed"], 0, DEVICE)
        with torch.no_grad():
            return [plates.PlateSplat.apply(1.0 + s["d"], px, py, s["flux"], s["params"],
                                            s["shape"], MPR, False)]
    if kind == "plate_batch":
        b, photons = s["batch"], (s["px"], s["py"], s["flux"])
        img = b.forward(s["field"], *photons)
        return [img, b.backward(s["field"], *photons, img - s["target"])]
    if kind == "point":
        field = s["field"].detach().requires_grad_(True)
        img = plates.PointPlateSplat.apply(field, *s["light_photons"], s["light"], s["params"],
                                           s["shape"], MPR)
        return [img.detach(), *torch.autograd.grad(img, [field], s["grad"])]
    return landweber_update(s["d"].clone(), s["grad"], s["mask"], s["update"])


# ------------------------------------------------------------------ what it must do ------

# Operations of one pixel inside the splat's support (forward 22, backward 55) and of one
# photon's refraction (the chain about 400, its reverse sweep with the chain about 1200; the
# traced hit adds about 300 to each).
FWD_PX, BWD_PX, CHAIN, CHAIN_BWD, TRACE = 22, 55, 400, 1200, 300


def _support(case):
    """Mean pixels of a photon's support: pi s1 s2 with both axes log-uniform."""
    lo, hi = (0.25, 16.0) if case["kind"] == "caustic" else (case.get("s_lo", 0.5), case.get("s_hi", 4.0))
    return math.pi * ((hi - lo) / math.log(hi / lo)) ** 2


def work(case):
    kind = case["kind"]
    if kind in ("pair", "autograd", "caustic", "render", "batch", "traced"):
        if kind == "batch":
            specs = _batch_specs(case)
            n, image = sum(k for k, _ in specs), sum(h * w for _, (_, h, w) in specs)
        else:
            n, image = case["n"], case.get("c", 1) * case["h"] * case["w"]
        per_in, per_out = (56, 36) if kind == "traced" else (40, 36)
        if kind == "render":
            return {"bytes": per_in * n + 4 * image, "flops": FWD_PX * _support(case) * n}
        return {"bytes": (per_in + per_out) * n + 8 * image,
                "flops": (FWD_PX + BWD_PX) * _support(case) * n}
    if kind == "update":
        return {"bytes": 16 * case["h"] * case["w"],
                "flops": (10 + (2 * case["radius"] + 1) ** 2) * case["h"] * case["w"]}
    texels = case["h"] * case["w"]
    px = math.pi * (FOOTPRINT_PX / 2) ** 2  # the photons' support at the initial footprint
    if kind == "plate_batch":
        sims = _plate_sims(case, 0)
        n, image = sum(per * texels for per, _, _ in sims), sum(s[1] * s[2] for _, s, _ in sims)
        return {"bytes": 12 * n + 12 * image + 8 * texels,
                "flops": n * (CHAIN + CHAIN_BWD + px * (FWD_PX + BWD_PX))}
    image = case["image"] ** 2
    if kind == "point":
        return {"bytes": 40 * case["n"] + 8 * image + 8 * texels,
                "flops": case["n"] * (CHAIN + CHAIN_BWD + 2 * TRACE + px * (FWD_PX + BWD_PX))}
    n = texels * case["per_texel"]
    if kind == "preview":
        return {"bytes": 4 * n + 4 * image + 4 * texels, "flops": n * (CHAIN + px * FWD_PX)}
    return {"bytes": 4 * n + 8 * image + 16 * texels,
            "flops": n * (CHAIN + CHAIN_BWD + px * (FWD_PX + BWD_PX))}


# ------------------------------------------------------------------ in 64 bits -----------

def _boxes(E, X, M, C, R, shape, mpr):
    """The photons' footprint boxes in blocks: (photon indices [n, 1], pixel index [n, k] into
    the flat image, offset dx, dy [n, k], inside [n, k])."""
    c, h, w = shape
    rx = torch.ceil(R * 0.5 * w).clamp(max=mpr)
    ry = torch.ceil(R * 0.5 * h).clamp(max=mpr)
    cx = torch.trunc((0.5 * X[0] + 0.5) * w).long()
    cy = torch.trunc((0.5 * X[1] + 0.5) * h).long()
    ok = (C >= 0) & (C < c) & (rx >= 0) & (ry >= 0) & torch.isfinite(X[0] + X[1])
    big = torch.where(ok, torch.maximum(rx, ry), torch.full_like(rx, -1.0)).long()
    order = torch.argsort(big)
    counts = torch.bincount(big + 1, minlength=mpr + 2).tolist()
    at = counts[0]
    for r, count in enumerate(counts[1:]):
        k = torch.arange(-r, r + 1, device=R.device)
        ky, kx = (t.reshape(1, -1) for t in torch.meshgrid(k, k, indexing="ij"))
        step = max(1, 2 ** 24 // kx.numel())
        for b in range(at, at + count, step):
            i = order[b:min(b + step, at + count)][:, None]
            px, py = cx[i] + kx, cy[i] + ky
            inside = ((kx.abs() <= rx[i]) & (ky.abs() <= ry[i]) & (px >= 0) & (px < w) &
                      (py >= 0) & (py < h) & ((2.0 * kx / w) ** 2 + (2.0 * ky / h) ** 2 <= 1.0))
            pixel = (C[i] * h + py) * w + px
            yield (i, torch.where(inside, pixel, torch.zeros_like(pixel)),
                   2.0 * px / w - 1.0 - X[0][i], 2.0 * py / h - 1.0 - X[1][i], inside)
        at += count


def _splat64(photons, shape, mpr, grad=None):
    """Image of the photons, or with ``grad`` (grad_Ep, grad_xp, grad_Mp), in 64 bits."""
    E, X, M, C, R = photons
    E, X, M, R = (t.detach().double() for t in (E, X, M, R))
    C = C.reshape(-1)
    out = torch.zeros(math.prod(shape), dtype=torch.float64, device=E.device)
    gE, gX, gM = torch.zeros_like(E), torch.zeros_like(X), torch.zeros_like(M)
    flat = grad.detach().double().reshape(-1) if grad is not None else None
    for i, pixel, dx, dy, inside in _boxes(E, X, M, C, R, shape, mpr):
        m00, m01, m10, m11 = M[0, 0][i], M[0, 1][i], M[1, 0][i], M[1, 1][i]
        u, v = m00 * dx + m01 * dy, m10 * dx + m11 * dy
        t = 1.0 - (u * u + v * v)
        inside = inside & (t > 0)
        if flat is None:
            val = 3.0 / math.pi * t * t * E[i]
            out.index_add_(0, pixel[inside], val[inside])
            continue
        tg = torch.where(inside, t, torch.zeros_like(t)) * flat[pixel]
        p = i[:, 0]
        gE[p] = 3.0 / math.pi * (t * tg).sum(1)
        a = -12.0 / math.pi * E[i] * tg
        au, av = a * u, a * v
        su, sv = au.sum(1), av.sum(1)
        gX[0, p] = -(m00[:, 0] * su + m10[:, 0] * sv)
        gX[1, p] = -(m01[:, 0] * su + m11[:, 0] * sv)
        gM[0, 0, p], gM[0, 1, p] = (au * dx).sum(1), (au * dy).sum(1)
        gM[1, 0, p], gM[1, 1, p] = (av * dx).sum(1), (av * dy).sum(1)
    return out.reshape(shape) if flat is None else (gE, gX, gM)


def _dot(a, b):
    return (a * b).sum(0)


def _bilinear(field, fx, fy):
    """Bilinear sample of [C, H, W] at texel coordinates, and its two slopes."""
    c, h, w = field.shape
    fx, fy = fx.clamp(0, w - 1), fy.clamp(0, h - 1)
    x0, y0 = fx.detach().floor().clamp(max=w - 2).long(), fy.detach().floor().clamp(max=h - 2).long()
    ax, ay = fx - x0, fy - y0
    flat = field.reshape(c, -1)
    a, b = flat[:, y0 * w + x0], flat[:, y0 * w + x0 + 1]
    e, f = flat[:, (y0 + 1) * w + x0], flat[:, (y0 + 1) * w + x0 + 1]
    top, bot = a + (b - a) * ax, e + (f - e) * ax
    return top + (bot - top) * ay, (b - a) * (1 - ay) + (f - e) * ay, bot - top


def _onto(D, Dd, t, n, d):
    """Differential D with direction differential Dd carried along d by t onto a plane."""
    nd = _dot(n, d)
    return D - _dot(n, D) / nd * d + t * (Dd - _dot(n, Dd) / nd * d)


def _bend(d, n, eta, pairs):
    """Snell's refraction of d at a normal facing it, with its differentials (Igehy 1999)."""
    cos = _dot(d, n)
    root = torch.sqrt(1 - eta * eta * (1 - cos * cos))
    mu = eta * cos + root
    dmu = eta + eta * eta * cos / root
    return eta * d - mu * n, [eta * Dd - mu * dn - dmu * (_dot(Dd, n) + _dot(d, dn)) * n
                              for Dd, dn in pairs]


def _plate64(h, p, px, py, d, hz, Ds):
    """Receiver position [2, n] and differentials [3, n] in receiver units of photons hitting
    the field ``h`` at (px, py, hz) along d; Ds: (positional, direction differential, length)
    pairs up to the hit."""
    rows, cols = h.shape
    fx, fy = px / p["texel"] + (cols - 1) / 2.0, py / p["texel"] + (rows - 1) / 2.0
    k = torch.tensor([[[-1., 0, 1], [-2, 0, 2], [-1, 0, 1]], [[-1, -2, -1], [0, 0, 0], [1, 2, 1]]],
                     dtype=h.dtype, device=h.device)[:, None] * (-1.0 / (8.0 * p["texel"]))
    g = F.conv2d(F.pad(h[None, None], (1, 1, 1, 1), mode="replicate"), k)[0]
    N, Nx, Ny = _bilinear(torch.cat((g, torch.ones_like(h)[None])), fx, fy)
    if hz is None:
        hz = _bilinear(h[None], fx, fy)[0][0]
    length2 = _dot(N, N)
    n = N / length2.sqrt()
    up = torch.zeros_like(n)
    up[2] = 1.0
    on, pairs = [], []
    for D, Dd, t in Ds:
        D1 = _onto(D, Dd, t, n, d)
        dN = (Nx * D1[0] + Ny * D1[1]) / p["texel"]
        on.append(D1)
        pairs.append((Dd, (length2 * dN - _dot(N, dN) * N) / length2 ** 1.5))
    t1, D1d = _bend(d, n, 1.0 / p["ior"], pairs)
    s1 = -hz / t1[2]
    D2 = [_onto(D, Dd, s1, up, t1) for D, Dd in zip(on, D1d)]
    t2, D2d = _bend(t1, up, p["ior"], [(Dd, torch.zeros_like(Dd)) for Dd in D1d])
    s2 = -p["distance"] / t2[2]
    D3 = [_onto(D, Dd, s2, up, t2) / p["half"] for D, Dd in zip(D2, D2d)]
    x = torch.stack((px + s1 * t1[0] + s2 * t2[0], py + s1 * t1[1] + s2 * t2[1])) / p["half"]
    return x, D3[0], D3[1]


def _basis64(Du, Dv, n, flux):
    """Splat inputs (Ep, Mp, radius) of receiver-plane differentials."""
    a = torch.linalg.cross(Dv, n, dim=0)
    M = 2.0 / _dot(Du, a) * torch.stack((a, torch.linalg.cross(n, Du, dim=0)))
    area = torch.linalg.cross(Du, Dv, dim=0).norm(dim=0)
    return 4.0 * flux / area, M, 0.5 * torch.maximum(Du.norm(dim=0), Dv.norm(dim=0))


def _collimated64(h, params, px, py, flux):
    """Splat inputs (Ep, xp, Mp, radius) of collimated photons on the plate."""
    p = dict(texel=params.texel, ior=params.ior, distance=params.receiver_distance,
             half=params.receiver_half)
    d = torch.tensor(list(params.light_dir), dtype=h.dtype, device=h.device)[:, None].expand(3, px.numel())
    zero = torch.zeros_like(d)
    Du, Dv = torch.zeros_like(d), torch.zeros_like(d)
    Du[0], Dv[1] = params.du0, params.du0
    x, Du, Dv = _plate64(h, p, px, py, d, None, [(Du, zero, 0.0), (Dv, zero, 0.0)])
    Ep, M, r = _basis64(Du, Dv, _up(Du), flux)
    return Ep, x, M, r


def _up(D):
    n = torch.zeros_like(D)
    n[2] = 1.0
    return n


def _traced64(h, params, light, direction, dtheta, dphi, flux):
    """Splat inputs of a point light's photons, traced onto the field's bilinear surface."""
    p = dict(texel=params.texel, ior=params.ior, distance=params.receiver_distance,
             half=params.receiver_half)
    rows, cols = h.shape
    o = torch.tensor(list(light.position), dtype=h.dtype, device=h.device)[:, None]
    t = (o[2] - light.plane_z) / (-direction[2])
    for _ in range(8):
        q = o + t * direction
        v, vx, vy = _bilinear(h[None], q[0] / p["texel"] + (cols - 1) / 2.0,
                              q[1] / p["texel"] + (rows - 1) / 2.0)
        slope = direction[2] - (vx[0] * direction[0] + vy[0] * direction[1]) / p["texel"]
        t = t - (q[2] - v[0]) / slope
    q = o + t * direction
    zero = torch.zeros_like(direction)
    x, Du, Dv = _plate64(h, p, q[0], q[1], direction, q[2], [(zero, dtheta, t), (zero, dphi, t)])
    Ep, M, r = _basis64(Du, Dv, _up(Du), flux)
    return Ep, x, M, r


CHUNK = 2 ** 21


def _chunks(chain, h, photons, grads=None):
    """Splat inputs of all photons (``grads`` None), or the height gradient for the gradients
    (Ep, xp, Mp) of them, chunk by chunk."""
    n = photons[0].shape[-1]
    parts, gh = [], torch.zeros_like(h)
    for b in range(0, n, CHUNK):
        ph = [t[..., b:b + CHUNK].double() for t in photons]
        if grads is None:
            with torch.no_grad():
                parts.append(chain(h, *ph))
        else:
            hv = h.detach().requires_grad_(True)
            gh += torch.autograd.grad(chain(hv, *ph)[:3], hv, [g[..., b:b + CHUNK] for g in grads])[0]
    return gh if grads is not None else [torch.cat([p[k] for p in parts], dim=-1) for k in range(4)]


def _splat_chain64(chain, h, photons, shape, grad_of):
    """(image, height gradient) through a chain; ``grad_of(image)`` the image's gradient, None:
    no gradient wanted."""
    E, X, M, R = _chunks(chain, h, photons)
    ph = (E, X, M, torch.zeros(E.numel(), dtype=torch.int64, device=h.device), R)
    img = _splat64(ph, shape, MPR)
    if grad_of is None:
        return img, None
    grads = _splat64(ph, shape, MPR, grad_of(img))
    return img, _chunks(chain, h, photons, grads)


def _update64(d, g, mask, p):
    x = d - p.tau * g
    x = mask * (torch.relu(x.abs() - p.tau * p.alpha) * x.sign()).clamp(p.lower, p.upper)
    v = float(x.sum())
    mean = F.avg_pool2d(x[None, None], 2 * p.radius + 1, stride=1, padding=p.radius)[0, 0]
    if v <= p.d1:
        return x + mask * mean * math.sin(v / p.d1 * math.pi) * p.gamma
    if v >= p.d2:
        return x - mask * mean * math.sin((v / p.d2 - 1) * math.pi) * p.gamma
    return x


def exact(case, seed):
    kind = case["kind"]
    s = prepare(case, seed)
    if kind in ("pair", "autograd", "caustic", "render"):
        shape = tuple(s["shape"])
        img = _splat64(s["photons"], shape, MPR)
        return [img] if kind == "render" else [img, *_splat64(s["photons"], shape, MPR, s["grad"])]
    if kind == "batch":
        imgs, grads, at, pixel = [], [], 0, 0
        for n, shape in _batch_specs(case):
            ph = tuple(t[..., at:at + n] for t in s["photons"])
            size = math.prod(shape)
            imgs.append(_splat64(ph, shape, MPR).reshape(-1))
            grads.append(_splat64(ph, shape, MPR, s["grad"][pixel:pixel + size]))
            at, pixel = at + n, pixel + size
        return [torch.cat(imgs), *(torch.cat([g[k] for g in grads], dim=-1) for k in range(3))]
    if kind == "traced":
        Du, Dv, flux = (s[k].detach().double().requires_grad_(True) for k in ("Du", "Dv", "flux"))
        E, M, R = _basis64(Du, Dv, s["normal"].double(), flux)
        ph = (E, s["xy"], M, s["channel"], R)
        gE, gX, gM = _splat64(ph, s["shape"], MPR, s["grad"])
        return [_splat64(ph, s["shape"], MPR),
                *torch.autograd.grad([E, M], [Du, Dv, flux], [gE, gM]), gX]
    if kind in ("landweber", "preview"):
        # the photons' entry points are drawn by the device source, whose float32 values are
        # the pass's inputs
        px, py, _ = photon_source(case["h"], case["w"], case["per_texel"], s["scene"].texel, seed,
                                  0, DEVICE)
        field = (1.0 + s["d"]).double()

        def chain(h, px, py, flux):
            return _collimated64(h, s["params"], px, py, flux)
        photons = (px, py, s["flux"])
        if kind == "preview":
            return [_splat_chain64(chain, field, photons, s["shape"], None)[0]]
        target = s["target"].double()
        img, g = _splat_chain64(chain, field, photons, s["shape"], lambda i: s["scale"] * (i - target))
        return [img, g, _update64(s["d"].double(), g, s["mask"].double(), s["update"])]
    if kind == "plate_batch":
        field, at, pixel = s["field"].double(), 0, 0
        imgs, gh = [], torch.zeros_like(field)
        for per, shape, sc in _plate_sims(case, seed):
            n, size = per * case["h"] * case["w"], math.prod(shape)
            par = _params(sc, shape[1])
            target = s["target"][pixel:pixel + size].double().reshape(shape)
            img, g = _splat_chain64(lambda h, *ph, par=par: _collimated64(h, par, *ph), field,
                                    [s[k][at:at + n] for k in ("px", "py", "flux")], shape,
                                    lambda i, target=target: i - target)
            imgs.append(img.reshape(-1))
            gh += g
            at, pixel = at + n, pixel + size
        return [torch.cat(imgs), gh]
    if kind == "point":
        return list(_splat_chain64(lambda h, *ph: _traced64(h, s["params"], s["light"], *ph),
                                   s["field"].double(), s["light_photons"], s["shape"],
                                   lambda i: s["grad"].double()))
    return _update64(s["d"].double(), s["grad"].double(), s["mask"].double(), s["update"])
