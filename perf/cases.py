"""The work this library is used for, as cases that can be timed and compared.

A single-particle project runs the same few calls over and over:

* reconstruction (``Reconstructor``): a micrograph's worth of particles, a
  project's batch or the last iteration's half maps are inserted and the map
  is finished; the box, the interpolation, the CTF action, the resolution
  limit and the point group change with the project;
* pose search (``Matcher``): particles against a panel of central sections at
  trial origins, over the whole panel or around proposed poses, then grid
  refinement of the best pose with its defocus;
* the learned proposer (``Proposer``): poses of a batch of images, and the
  loss and gradient of a training batch;
* real-space back-projection (``BackProjector``).

Particle images are noisy, CTF-modulated projections of a phantom of Gaussian
blobs with random views, shifts and defoci, as ``bsoft_b200.synth`` makes them
(on the GPU here, so that they are quick to make).
"""
import math

import numpy as np
import torch

from bsoft_b200.backproj import BackProjector, BackprojPlan
from bsoft_b200.cnn import Proposer
from bsoft_b200.match import Matcher, ctf_record
from bsoft_b200.plan import ReconPlan
from bsoft_b200.recon import Reconstructor

VOLT, CS, AMP = 200000.0, 2.7e7, 0.07       # 200 kV, 2.7 mm, 7% amplitude contrast
PIXEL = 1.5                                 # angstrom per pixel
TRIAL = [(dx, dy) for dy in range(-2, 3) for dx in range(-2, 3)]    # 25 trial origins, +-2 pixels
CHANNELS, HIDDEN = (32, 64, 64, 128, 128, 128), 1024                # the proposer's default network


def listed():
    return [
        # the smallest call: one sparse micrograph of small particles, host
        # arrays in and out; launches, copies and set-up count most here
        {"name": "recon-64-few", "kind": "recon", "box": 64, "images": 60, "interp": 2, "ctf": 1, "maps": 1,
         "res": 0.0, "wiener": 0.0, "sym": "C1", "host": True},
        # a small project at low resolution: 2,000 boxes of 64 pixels into two
        # half maps and their FSC
        {"name": "recon-64-halves", "kind": "recon", "box": 64, "images": 2000, "interp": 2, "ctf": 1, "maps": 2,
         "res": 0.0, "wiener": 0.0, "sym": "C1", "host": False},
        # breconstruct's default interpolation (nearest) on a box that is no
        # power of two, with a resolution limit (the taper) and the CTF applied
        {"name": "recon-100-nearest", "kind": "recon", "box": 100, "images": 500, "interp": 0, "ctf": 2, "maps": 1,
         "res": 8.3, "wiener": 0.0, "sym": "C1", "host": False},
        # a dimer: D2 symmetry inserted, CTF corrected with a Wiener constant
        {"name": "recon-128-d2", "kind": "recon", "box": 128, "images": 400, "interp": 2, "ctf": 4, "maps": 1,
         "res": 0.0, "wiener": 0.2, "sym": "D2", "host": False},
        # the ordinary large job: a batch of 2,000 boxes of 256 pixels, trilinear
        # with CTF flip, into one map
        {"name": "recon-256", "kind": "recon", "box": 256, "images": 2000, "interp": 2, "ctf": 1, "maps": 1,
         "res": 0.0, "wiener": 0.0, "sym": "C1", "host": False},
        # the largest: boxes of 384 pixels (transform 1024) into two half maps,
        # both finished, and their FSC
        {"name": "recon-384-halves", "kind": "recon", "box": 384, "images": 500, "interp": 2, "ctf": 1, "maps": 2,
         "res": 0.0, "wiener": 0.0, "sym": "C1", "host": False},
        # exhaustive pose search of a batch over a 6 degree panel
        {"name": "search-128", "kind": "search", "box": 128, "images": 256, "step": 6.0},
        # search within 10 degrees of proposed poses, over the same panel
        {"name": "local-128", "kind": "local", "box": 128, "images": 512, "step": 6.0},
        # brefine's grid refinement with the defocus search
        {"name": "refine-128", "kind": "refine", "box": 128, "images": 24},
        # the proposer's poses for a search batch
        {"name": "predict-128", "kind": "predict", "box": 128, "images": 2048},
        # one training batch's loss and gradient
        {"name": "gradient-128", "kind": "gradient", "box": 128, "images": 256},
        # real-space back-projection (bbackproj) of one micrograph's particles
        {"name": "backproject-128", "kind": "backproject", "box": 128, "images": 200, "maps": 1, "res": 6.0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["recon"] * 6 + ["search", "local", "refine", "predict", "gradient", "backproject"])
    if kind == "recon":
        # even edges that are products of 2, 3, 5 and 7, as the map transform takes them
        edges = [e for e in range(48, 386, 2) if _smooth(e)]
        box = rng.choice(edges)
        ft = _pow2(2 * box)
        most = int(3.2e8 / (ft * ft))       # as many pixels as the largest listed case at most
        sym = rng.choice(["C1"] * 5 + ["C3", "D2"])
        images = _log(rng, 40, min(2500, most // (1 if sym == "C1" else 4)))
        ctf = rng.choice([0, 1, 1, 1, 2, 4])
        return {"kind": kind, "box": box, "images": images, "interp": rng.choice([2, 2, 2, 2, 1, 0]), "ctf": ctf,
                "maps": rng.choice([1, 1, 2]), "res": rng.choice([0.0, 0.0, 0.0, 5.9, 8.3]),
                "wiener": 0.2 if ctf == 4 else 0.0, "sym": sym, "host": rng.random() < 0.25}
    if kind in ("search", "local"):
        return {"kind": kind, "box": rng.choice([64, 128, 128]), "images": _log(rng, 16, 256),
                "step": round(rng.uniform(6.0, 12.0), 1)}
    if kind == "refine":
        return {"kind": kind, "box": rng.choice([64, 128]), "images": _log(rng, 2, 24)}
    if kind == "predict":
        return {"kind": kind, "box": rng.choice([64, 128, 128]), "images": _log(rng, 1, 2048)}
    if kind == "gradient":
        return {"kind": kind, "box": rng.choice([64, 128, 128]), "images": _log(rng, 8, 256)}
    return {"kind": kind, "box": rng.choice([60, 64, 90, 96, 100, 128]), "images": _log(rng, 20, 200),
            "maps": rng.choice([1, 2]), "res": round(rng.uniform(4.5, 12.0), 1)}


def _smooth(n):
    for p in (2, 3, 5, 7):
        while n % p == 0:
            n //= p
    return n == 1


def _pow2(n):
    p = 1
    while p < n:
        p *= 2
    return p


# ---- inputs ----------------------------------------------------------------

def _rotations(rng, n):
    """Uniform random rotation matrices (n, 3, 3)."""
    q = rng.normal(size=(n, 4))
    w, x, y, z = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
    return np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                     2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                     2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], axis=1).reshape(n, 3, 3)


def _views(rng, n):
    """Random views (x, y, z, angle) and their matrices, as View::matrix gives them."""
    v = rng.normal(size=(n, 3))
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    return np.concatenate([v, rng.uniform(-math.pi, math.pi, (n, 1))], axis=1)


def _ctf(rng, n, lo=8000.0, hi=35000.0):
    """Aberration weights (n, 7) of random defoci (angstrom) and astigmatism."""
    wl = 6.62607015e-34 * 1e10 / math.sqrt(2 * 9.1093837e-31 * 1.602176634e-19 * VOLT
                                           * (1 + 1.602176634e-19 * VOLT / (2 * 9.1093837e-31 * 299792458.0 ** 2)))
    defocus, dev, ang = rng.uniform(lo, hi, n), rng.uniform(0, 1000.0, n), rng.uniform(-math.pi, math.pi, n)
    c = np.zeros((n, 7))
    c[:, 0] = -math.asin(AMP)
    c[:, 1] = -math.pi * wl * defocus
    c[:, 2] = -math.pi * wl * dev * np.cos(2 * ang)
    c[:, 3] = -math.pi * wl * dev * np.sin(2 * ang)
    c[:, 4] = math.pi / 2 * wl ** 3 * CS
    return c


def _chi(c, sx, sy):
    """The even aberration of weights c (n, 7) at frequencies sx, sy."""
    c = c.reshape(c.shape[0], 7, *([1] * sx.dim())).unbind(1)
    s2 = sx * sx + sy * sy
    return c[0] + c[1] * s2 + c[2] * (sx * sx - sy * sy) + c[3] * (2 * sx * sy) + c[4] * s2 * s2


def _phantom(rng, box, blobs=60):
    d = rng.normal(size=(blobs, 3))
    d *= (0.35 * box * rng.uniform(0, 1, blobs) ** (1 / 3) / np.linalg.norm(d, axis=1))[:, None]
    return d, rng.uniform(1.5, 3.0, blobs) * max(1.0, box / 128), rng.uniform(0.5, 1.0, blobs)


def _volume(ph, box):
    c, s, a = (torch.from_numpy(t).cuda() for t in ph)
    g = torch.arange(box, dtype=torch.float64, device="cuda") - box // 2
    e = [torch.exp(-(g[:, None] - c[None, :, i]) ** 2 / (2 * s * s)) for i in range(3)]
    return torch.einsum("zk,yk,xk->zyx", e[2] * a, e[1], e[0]).float().contiguous()


def _images(rng, ph, mats, origins, ctf, box, snr):
    """Projections of the phantom with CTF and white noise, (n, box, box) float32 on the GPU."""
    n = len(mats)
    out = torch.empty((n, box, box), dtype=torch.float32, device="cuda")
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(rng.integers(1 << 40)))
    c, s, a = (torch.from_numpy(t).cuda().float() for t in ph)
    f = torch.fft.fftfreq(box, PIXEL, dtype=torch.float64, device="cuda")
    sy, sx = torch.meshgrid(f, f, indexing="ij")
    x = torch.arange(box, dtype=torch.float32, device="cuda")
    for i in range(0, n, 250):
        m = torch.from_numpy(mats[i:i + 250]).cuda().float()
        o = torch.from_numpy(origins[i:i + 250]).cuda().float()
        p = [torch.exp(-(x[None, :, None] - (c @ m[:, :, j, None]).reshape(len(m), 1, -1) - o[:, j, None, None]) ** 2
                       / (2 * s * s)) for j in (0, 1)]
        im = torch.bmm(p[1] * (a * s * math.sqrt(2 * math.pi)), p[0].transpose(1, 2))
        if ctf is not None:
            w = torch.sin(_chi(torch.from_numpy(ctf[i:i + 250]).cuda(), sx, sy)).float()
            im = torch.fft.ifft2(torch.fft.fft2(im) * w).real
        noise = torch.randn(im.shape, generator=gen, device="cuda")
        out[i:i + 250] = im + noise * (im.std(dim=(1, 2), keepdim=True) / math.sqrt(snr))
    return out


def _recon_inputs(case, seed):
    rng = np.random.default_rng([seed, case["box"], case["images"]])
    n, P = case["box"], case["images"]
    mats = _rotations(rng, P)
    origins = n // 2 + rng.uniform(-2, 2, (P, 2))
    ctf = _ctf(rng, P)
    imgs = _images(rng, _phantom(rng, n), mats, origins, ctf if case["ctf"] else None, n, 0.05)
    ft = _pow2(2 * n)
    rec = np.zeros((P, 32))                    # the C ABI's particle record
    rec[:, 0:2] = origins
    rec[:, 4:13] = mats.reshape(P, 9)
    rec[:, 13] = PIXEL
    rec[:, 14] = 1.0
    rec[:, 15] = 1.0
    rec[:, 16:23] = ctf
    rec[:, 23] = np.arange(P) % 2
    hi = max(case["res"], 2 * PIXEL / math.sqrt(3.0))
    plan = ReconPlan(n=n, ft=ft, map=n, map_sampling=PIXEL, hi_res=hi, interp=case["interp"], ctf_action=case["ctf"],
                     wiener=case["wiener"], params=rec, nmaps=case["maps"], symmetry=case["sym"], resolution=PIXEL)
    return plan, imgs


def _match_inputs(case, seed):
    n, P = case["box"], case["images"]
    rng = np.random.default_rng([seed, n, P])
    ph = _phantom(rng, n)
    from bsoft_b200.geometry import views_to_matrices
    views = _views(rng, P)
    mats = views_to_matrices(views)
    shift = rng.uniform(-2, 2, (P, 2))
    ctf = _ctf(rng, P, 10000.0, 30000.0)
    imgs = _images(rng, ph, mats, n // 2 + shift, ctf, n, 0.1)
    m = Matcher(n=n, map=n, map_sampling=PIXEL, pixel=PIXEL, hi_res=3.75)
    m.set_reference(_volume(ph, n), (n // 2,) * 3)
    recs = np.stack([ctf_record(VOLT, c) for c in ctf])
    return rng, m, imgs, recs, views, mats, shift


def _panel(step):
    from bsoft_b200.geometry import asymmetric_unit_views_c, quaternion_to_matrix, search_views, view_to_quaternion
    dirs = asymmetric_unit_views_c(1, math.radians(step), math.radians(step))
    psi = int(360 / step)
    # the matrix of (direction, angle + psi) is the direction's matrix times the
    # in-plane rotation by psi
    d = np.stack([quaternion_to_matrix(view_to_quaternion(v)) for v in search_views(dirs, 1)])
    a = 2 * math.pi * np.arange(psi) / psi
    z = np.zeros((psi, 3, 3))
    z[:, 0, 0] = z[:, 1, 1] = np.cos(a)
    z[:, 1, 0] = np.sin(a)
    z[:, 0, 1] = -np.sin(a)
    z[:, 2, 2] = 1
    return np.einsum("dij,pjk->dpik", d, z).reshape(-1, 3, 3)


def _network(rng, box):
    """Parameters in the library's order: six convolutions and two dense
    layers, weight then bias each, as a trained net's are distributed."""
    side, cin, parts = box // 64, 1, []
    for c in CHANNELS:
        parts += [rng.normal(size=(c, 9 * cin)) * math.sqrt(2 / (9 * cin)), rng.normal(size=c) * 0.02]
        cin = c
    k = side * side * cin
    parts += [rng.normal(size=(HIDDEN, k)) * math.sqrt(2 / k), rng.normal(size=HIDDEN) * 0.02]
    parts += [rng.normal(size=(8, HIDDEN)) * math.sqrt(1 / HIDDEN), rng.normal(size=8) * 0.02]
    return [p.astype(np.float32) for p in parts]


def _net_inputs(case, seed):
    n, P = case["box"], case["images"]
    rng = np.random.default_rng([seed, n, P])
    mats = _rotations(rng, P)
    shift = rng.uniform(-2, 2, (P, 2))
    imgs = _images(rng, _phantom(rng, n), mats, n // 2 + shift, _ctf(rng, P, 10000.0, 30000.0), n, 0.1)
    targets = np.concatenate([mats.reshape(P, 9), shift], axis=1).astype(np.float32)
    return imgs, targets, _network(rng, n)


def _backproject_inputs(case, seed):
    n, P = case["box"], case["images"]
    rng = np.random.default_rng([seed, n, P])
    mats = _rotations(rng, P)
    origins = n // 2 + rng.uniform(-2, 2, (P, 2))
    imgs = _images(rng, _phantom(rng, n), mats, origins, None, n, 0.1)
    rec = np.zeros((P, 16))                    # the C ABI's back-projection record
    rec[:, 0:2] = origins
    rec[:, 2:11] = mats.reshape(P, 9)
    rec[:, 11] = 1.0
    rec[:, 12] = np.arange(P) % 2 if case["maps"] == 2 else 0
    rec[:, 13] = PIXEL
    plan = BackprojPlan(n=n, map=n, map_sampling=PIXEL, pixel=PIXEL, resolution=case["res"], records=rec,
                        nmaps=case["maps"])
    return plan, imgs


def prepare(case, seed):
    kind = case["kind"]
    if kind == "recon":
        plan, imgs = _recon_inputs(case, seed)
        if case["host"]:
            imgs = imgs.cpu().numpy()
        s = dict(plan=plan, imgs=imgs, rec=Reconstructor(plan))
        if not case["host"]:
            n = plan.map
            s["out"] = [torch.empty((n, n, n), dtype=torch.float32, device="cuda") for _ in range(plan.nmaps)]
    elif kind in ("search", "local", "refine"):
        rng, m, imgs, recs, views, mats, shift = _match_inputs(case, seed)
        n, P = case["box"], case["images"]
        s = dict(m=m, imgs=imgs, recs=recs)
        s["origins"] = n // 2 + np.array(TRIAL, dtype=np.float64)
        if kind != "refine":
            m.set_panel(_panel(case["step"]))
        if kind == "local":
            # proposals a few degrees and a fraction of a pixel off
            ax = rng.normal(size=(P, 3))
            ax *= (np.radians(rng.uniform(0, 8, P)) / np.linalg.norm(ax, axis=1))[:, None]
            z = np.zeros(P)
            K = np.stack([z, -ax[:, 2], ax[:, 1], ax[:, 2], z, -ax[:, 0], -ax[:, 1], ax[:, 0], z],
                         axis=1).reshape(P, 3, 3)
            u, _, vt = np.linalg.svd((np.eye(3) + K) @ mats)
            prop = np.concatenate([(u @ vt).reshape(P, 9), shift + rng.normal(size=(P, 2)) * 0.5], axis=1)
            s["proposals"] = torch.from_numpy(prop.astype(np.float32)).cuda()
        if kind == "refine":
            m.set_c_curve_weights()
            v = views.copy()
            v[:, :3] += rng.normal(size=(P, 3)) * math.radians(1.2)
            v[:, :3] /= np.linalg.norm(v[:, :3], axis=1, keepdims=True)
            v[:, 3] += rng.normal(size=P) * math.radians(1.2)
            start = n // 2 + np.rint(shift)
            s["start"] = np.column_stack([np.arange(P), v, start])
    elif kind in ("predict", "gradient"):
        imgs, targets, net = _net_inputs(case, seed)
        p = Proposer(box=case["box"], batch=256, channels=CHANNELS, hidden=HIDDEN)
        p.set_params(np.concatenate([t.ravel() for t in net]))
        s = dict(net=p, imgs=imgs, targets=targets)
        if kind == "predict":
            s["out"] = torch.empty((case["images"], 11), dtype=torch.float32, device="cuda")
        else:
            s["imgs"] = imgs.cpu().numpy()     # loss_grad takes host arrays
    else:
        plan, imgs = _backproject_inputs(case, seed)
        s = dict(plan=plan, imgs=imgs, bp=BackProjector(plan))
    s["kind"] = kind
    torch.cuda.synchronize()
    return s


# ---- one pass --------------------------------------------------------------

def run(s):
    kind = s["kind"]
    if kind == "recon":
        rec, plan = s["rec"], s["plan"]
        rec.reset()
        rec.insert(s["imgs"], plan.params)
        which = [0] if plan.nmaps == 1 else [1, 2]
        maps = [rec.finish(i, out=s["out"][k] if "out" in s else None) for k, i in enumerate(which)]
        return {"maps": maps, "fsc": rec.fsc()} if plan.nmaps == 2 else {"maps": maps}
    if kind in ("search", "local"):
        m = s["m"]
        m.set_images(s["imgs"], s["recs"])
        r = m.search(s["origins"]) if kind == "search" else m.search_local(s["proposals"], s["origins"])
        return {"section": r[:, :, 0].astype(np.int64), "origin": r[:, :, 1].astype(np.int64), "scores": r[:, :, 2:]}
    if kind == "refine":
        m = s["m"]
        m.set_images(s["imgs"], s["recs"])
        # 2 to 0.5 degrees, 0.4 to 0.1 pixel, defocus +-5 x 100 angstrom
        return m.refine(s["start"], math.radians(2.0), math.radians(0.5), 0.4, 0.1, 100.0)
    if kind == "predict":
        return s["net"].predict(s["imgs"], out=s["out"])
    if kind == "gradient":
        loss, grad = s["net"].loss_grad(s["imgs"], s["targets"])
        return {"loss": np.float32(loss), "grad": grad}
    bp, plan = s["bp"], s["plan"]
    bp.reset()
    bp.add(s["imgs"], plan.records)
    return [bp.finish(i) for i in ([0] if plan.nmaps == 1 else [1, 2])]


# ---- what one pass cannot do without ---------------------------------------

def work(case):
    n, P = case["box"], case["images"]
    kind = case["kind"]
    if kind == "recon":
        ft, nsym = _pow2(2 * n), {"C1": 1, "C3": 3, "D2": 4}[case["sym"]]
        # a 2-D transform of each image, one half plane of pixels (the other
        # is its conjugate) spread over 8 (1) voxels, the 3-D transform
        lit = ft * ft / 2 * min(1.0, math.pi * (PIXEL / case["res"]) ** 2 if case["res"] else 1.0)
        flops = P * 5 * ft * ft * math.log2(ft) + P * nsym * lit * (8 * 8 if case["interp"] == 2 else 8)
        return {"bytes": 4.0 * P * n * n + 256.0 * P + 4.0 * n ** 3 * case["maps"],
                "flops": flops + case["maps"] * 15 * n ** 3 * math.log2(n)}
    if kind in ("search", "local", "refine"):
        rad = n * PIXEL / 3.75                     # shells up to the resolution limit
        half = math.pi / 2 * rad * rad             # pixels of the half plane
        dirs = 4 * math.pi / math.radians(case.get("step", 6.0)) ** 2
        sections = dirs * 360 / case.get("step", 6.0)
        if kind == "search":
            return {"bytes": 4.0 * P * n * n + 4 * half * sections + 40.0 * 8 * P,
                    "flops": 4 * half * sections * P * len(TRIAL)}
        if kind == "local":
            near = sections * (math.radians(10) ** 3 / 6) / math.pi     # share of the rotations within 10 degrees
            return {"bytes": 4.0 * P * n * n + min(1, P * near / sections) * 4 * half * sections + 40.0 * 8 * P,
                    "flops": 4 * half * near * P * 9}
        # about 300 views a particle, 512 taps a pixel, and some 9,400 scored
        # hypotheses a particle
        return {"bytes": 4.0 * P * n * n + 8.0 * (2.2 * rad) ** 3, "flops": P * half * (300 * 512 * 4 + 9400 * 20.0)}
    if kind in ("predict", "gradient"):
        macs, side, cin, params = 0, n, 1, 0
        for c in CHANNELS:
            side //= 2
            macs += side * side * c * 9 * cin
            params += 9 * cin * c + c
            cin = c
        macs += side * side * cin * HIDDEN + HIDDEN * 8
        params += side * side * cin * HIDDEN + HIDDEN * 9 + 8
        if kind == "predict":
            return {"bytes": P * (4.0 * n * n + 44) + 4.0 * params, "flops": 2.0 * P * macs}
        return {"bytes": P * (4.0 * n * n + 44) + 8.0 * params, "flops": 6.0 * P * macs}
    return {"bytes": 4.0 * P * n * n + 4.0 * n ** 3 * case["maps"],
            "flops": P * 20.0 * n * n * math.log2(n) + 30.0 * P * n ** 3}


# ---- the same results in 64 bits -------------------------------------------

def _exact_map(v, w, n, sinc):
    f = torch.where(w > 1e-30, v / w.clamp_min(1e-30), torch.zeros_like(v)).reshape(n, n, n)
    g = torch.arange(n, device="cuda")
    odd = (g[:, None, None] + g[None, :, None] + g[None, None, :]) % 2
    r = torch.fft.ifftn(f * (1 - 2 * odd)).real * math.sqrt(n ** 3)
    if sinc:
        d = (g.double() - n // 2) / n
        a = math.pi * torch.sqrt(d[:, None, None] ** 2 + d[None, :, None] ** 2 + d[None, None, :] ** 2)
        r = torch.where(a > 0, (a / torch.sin(a)) ** 2 * r, r)
    return r, f


def _operators(sym):
    c, s = math.cos(2 * math.pi / 3), math.sin(2 * math.pi / 3)
    if sym == "C3":
        rot = torch.tensor([[c, -s, 0], [s, c, 0], [0, 0, 1]], dtype=torch.float64, device="cuda")
        return [torch.eye(3, dtype=torch.float64, device="cuda"), rot, rot @ rot]
    diag = [(1, 1, 1)] + ([(-1, -1, 1), (1, -1, -1), (-1, 1, -1)] if sym == "D2" else [])
    return [torch.diag(torch.tensor(d, dtype=torch.float64, device="cuda")) for d in diag]


def _exact_recon(case, seed):
    plan, imgs = _recon_inputs(case, seed)
    n, ft, P, dev = plan.n, plan.ft, case["images"], "cuda"
    par = torch.from_numpy(plan.params).cuda()
    k = torch.fft.fftfreq(ft, 1.0 / ft, dtype=torch.float64, device=dev)
    ky, kx = torch.meshgrid(k, k, indexing="ij")
    x = torch.arange(n, dtype=torch.float64, device=dev) / (n // 2)
    outside = (x[:, None] ** 2 + x[None, :] ** 2) > 1          # the circle about the file origin, (0, 0)
    inv, scale = 1 / (ft * PIXEL), n / ft
    lim = plan.hi_res
    s2 = (kx * kx + ky * ky) * inv * inv
    taper = torch.sqrt(((1 / lim ** 2 - s2) * n * PIXEL).clamp(0, 1))
    keep = (s2 <= 1 / lim ** 2).flatten()
    hk = torch.stack([kx.flatten()[keep], ky.flatten()[keep]])
    pw = (taper / ((ft / n) ** 2 * 0.6)).flatten()[keep]
    ops = _operators(case["sym"])
    nm = plan.nmaps
    v = torch.zeros((nm, n ** 3, 2), dtype=torch.float64, device=dev)
    w = torch.zeros((nm, n ** 3), dtype=torch.float64, device=dev)
    for i in range(P):
        im = imgs[i].double()
        big = torch.full((ft, ft), float(im[outside].mean()), dtype=torch.float64, device=dev)
        big[:n, :n] = im
        f = torch.fft.fft2(big) / ft
        f = f * torch.polar(torch.ones_like(kx), 2 * math.pi / ft * (kx * par[i, 0] + ky * par[i, 1]))
        if case["ctf"]:
            c = torch.sin(_chi(par[i:i + 1, 16:23], kx * inv, ky * inv)[0])
            if case["ctf"] == 1:
                c = torch.where(c < 0, -1.0, 1.0).double()
            elif plan.wiener:
                c = (plan.wiener + 1) * c / (c * c + plan.wiener)
            f = f * c * (s2 <= 1 / plan.hi_res ** 2)
        f = torch.view_as_real(f.flatten()[keep])
        half = int(plan.params[i, 23]) if nm == 2 else 0
        for o in ops:
            m = (o @ par[i, 4:13].reshape(3, 3))[:, :2] @ hk * scale
            if case["interp"] == 2:
                b = torch.floor(m)
                r = m - b
                corners = [(dx, dy, dz) for dz in (0, 1) for dy in (0, 1) for dx in (0, 1)]
            else:
                b = torch.floor(m + 0.5)
                r = m - b
                corners = [(0, 0, 0)]
            b = b.long()
            for c in corners:
                if case["interp"] == 2:
                    t = pw
                    for a in range(3):
                        t = t * (r[a] if c[a] else 1 - r[a])
                else:
                    t = pw * (1 - r.norm(dim=0)).clamp_min(0) if case["interp"] == 1 else pw
                j = (b[0] + c[0]) % n + n * ((b[1] + c[1]) % n + n * ((b[2] + c[2]) % n))
                v[half].index_add_(0, j, f * t[:, None])
                w[half].index_add_(0, j, t)
    got = [_exact_map(torch.view_as_complex(v[h]), w[h], n, case["interp"] == 2) for h in range(nm)]
    if nm == 1:
        return {"maps": [got[0][0]]}
    # the half maps' FSC: each voxel split linearly between its two shells
    rmax = int(n * PIXEL / plan.hi_res)
    g = torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device=dev)
    g = torch.where(g == -n // 2, -g, g)
    rad = torch.sqrt(g[:, None, None] ** 2 + g[None, :, None] ** 2 + g[None, None, :] ** 2).flatten()
    lo = rad.long()
    a, b = got[0][1].flatten(), got[1][1].flatten()
    sums = torch.zeros((3, 2 * n), dtype=torch.float64, device=dev)
    ok = lo < rmax
    for q, t in enumerate(((a * b.conj()).real, a.abs() ** 2, b.abs() ** 2)):
        sums[q].index_add_(0, lo[ok], (t * (1 - (rad - lo)))[ok])
        sums[q].index_add_(0, lo[ok] + 1, (t * (rad - lo))[ok])
    fsc = torch.nan_to_num(sums[0] / torch.sqrt(sums[1] * sums[2]), 0.0, 0.0, 0.0)
    fsc[0] = 1
    fsc[rmax:] = 0
    return {"maps": [got[0][0], got[1][0]], "fsc": fsc[:n // 2].cpu().numpy()}


def _exact_net(case, seed):
    imgs, targets, net = _net_inputs(case, seed)
    w = [torch.from_numpy(t).cuda().bfloat16().double().requires_grad_(case["kind"] == "gradient") for t in net]
    res, total = [], 0.0
    for i in range(0, len(imgs), 256):
        x = imgs[i:i + 256].double()
        x = (x - x.mean(dim=(1, 2), keepdim=True)) / x.std(dim=(1, 2), keepdim=True, unbiased=False)
        x, cin = x[:, None], 1
        for k, c in enumerate(CHANNELS):
            ker = w[2 * k].reshape(c, 3, 3, cin).permute(0, 3, 1, 2)
            u = torch.nn.functional.unfold(x, 3, padding=1, stride=2)      # (n, cin * 9, pixels)
            y = ker.reshape(c, -1) @ u + w[2 * k + 1][:, None]
            side = x.shape[-1] // 2
            x, cin = torch.relu(y).reshape(len(x), c, side, side), c
        x = x.permute(0, 2, 3, 1).reshape(len(x), -1)
        o = torch.relu(x @ w[12].T + w[13]) @ w[14].T + w[15]
        b1 = o[:, :3] / (o[:, :3].norm(dim=1, keepdim=True) + 1e-12)
        b2 = o[:, 3:6] - (b1 * o[:, 3:6]).sum(1, keepdim=True) * b1
        b2 = b2 / (b2.norm(dim=1, keepdim=True) + 1e-12)
        R = torch.stack([b1, b2, torch.linalg.cross(b1, b2)], dim=2)
        if case["kind"] == "predict":
            res.append(torch.cat([R.reshape(-1, 9), o[:, 6:8]], dim=1))
            continue
        t = torch.from_numpy(targets[i:i + 256]).cuda().double()
        loss = (((R.reshape(-1, 9) - t[:, :9]) ** 2).sum() + 0.05 * ((o[:, 6:8] - t[:, 9:]) ** 2).sum()) / len(imgs)
        loss.backward()
        total += float(loss.detach())
    if case["kind"] == "predict":
        return torch.cat(res)
    return {"loss": np.float64(total), "grad": torch.cat([t.grad.flatten() for t in w]).cpu().numpy()}


def _exact_backproject(case, seed):
    plan, imgs = _backproject_inputs(case, seed)
    n, dev = plan.n, "cuda"
    k = torch.arange(n, dtype=torch.float64, device=dev)
    s = torch.where(k > n // 2, n - k, k) / (n * PIXEL)
    s2 = s[:, None] ** 2 + s[None, :] ** 2
    ramp = torch.where(s2 > 1 / max(case["res"], math.sqrt(2) * PIXEL) ** 2, 0.0, torch.sqrt(s2))
    g = k - n // 2
    maps = torch.zeros((case["maps"], n, n, n), dtype=torch.float64, device=dev)
    for i in range(case["images"]):
        r = plan.records[i]
        f = torch.fft.ifft2(torch.fft.fft2(imgs[i].double()) * ramp).real
        f = (f - f.mean()) / f.std(unbiased=False)
        ell = ((k[None, :] - r[0]) / (n // 2)) ** 2 + ((k[:, None] - r[1]) / (n // 2)) ** 2
        fill = f[ell > 1].mean()
        m = r[2:11].reshape(3, 3)
        X, Y = (m[0, c] * g[None, None, :] + m[1, c] * g[None, :, None] + m[2, c] * g[:, None, None] + r[c]
                for c in (0, 1))
        inside = (X >= 0) & (X < n) & (Y >= 0) & (Y < n)
        ix, iy = X.clamp(0, n - 1).long(), Y.clamp(0, n - 1).long()
        fx, fy = X - ix, Y - iy
        # the reference's sample weights flip once per visited sample: at the
        # last column the second row gets the unflipped one
        last_x, last_y = ix == n - 1, iy == n - 1
        jx, jy = (ix + 1).clamp_max(n - 1), (iy + 1).clamp_max(n - 1)
        zero = torch.zeros_like(fx)
        ws = [(1 - fx) * (1 - fy), torch.where(last_x, zero, fx * (1 - fy)),
              torch.where(last_y, zero, torch.where(last_x, fx, 1 - fx) * fy),
              torch.where(last_x | last_y, zero, fx * fy)]
        val = ws[0] * f[iy, ix] + ws[1] * f[iy, jx] + ws[2] * f[jy, ix] + ws[3] * f[jy, jx]
        tot = ws[0] + ws[1] + ws[2] + ws[3]
        val = torch.where(tot != 0, val / torch.where(tot != 0, tot, torch.ones_like(tot)), fill)
        maps[int(r[12])] += torch.where(inside, val, fill)
    return [m.cpu().numpy() for m in maps]


def exact(case, seed):
    """What run() returns, from plain torch in 64 bits.  The searches and the
    refinement choose among hypotheses by scores that the library defines
    (BF16 correlations, brefine's decisions); restating them in plain torch
    takes minutes, so they have none."""
    kind = case["kind"]
    if kind == "recon":
        return _exact_recon(case, seed)
    if kind in ("predict", "gradient"):
        return _exact_net(case, seed)
    if kind == "backproject":
        return _exact_backproject(case, seed)
    return None
