"""The work a McSART program has this engine do, as timed cases.

A case is one call (or the fixed run of calls a program makes for one view)
through the public entry points of ``mcsart_b200``:

  view     one SART view of a static volume through the launchers, as
           host_AUMISART's loop body makes it (src/AUMISART.cu:42-63)
  motion   one view of the DVF-update pass through the launchers
           (src/AUMISART.cu:236-288), norms included
  warp     a volume deformed to a breathing phase and back, the displacement
           and its inverse, and a 16-bit exact-weight warp
  views    every view of one volume projected in one call (simulating a scan)
  pair     the projector and its exact adjoint (a gradient step)
  loop     host_AUMISART's loop on device-resident buffers
  batch    several uneven reconstructions at once
  host     the MATLAB gateway's call: host arrays in, host arrays out

Sizes are those of ``mcsart_b200.synthetic`` and of the tests, and odd ones in
the same range.  Geometry, phantom, breathing amplitudes and field strengths
follow ``mcsart_b200.synthetic``; the inputs are made on the GPU (ellipsoid
line integrals for the measured projections), so that a case is quick to set up.
"""
import math

import numpy as np
import torch

import mcsart_b200 as m
from mcsart_b200 import gateway, synthetic

DEV = "cuda"


# ------------------------------------------------------------------ the cases
def _case(name, kind, nx, ny, nz, na, nb, vox, pitch, views=1, **kw):
    return dict(name=name, kind=kind, nx=nx, ny=ny, nz=nz, na=na, nb=nb, vox=vox, pitch=pitch,
                views=views, **kw)


def listed():
    return [
        # the smallest calls: a program stepping through a 64^3 scan view by view
        _case("view_64", "view", 64, 64, 64, 128, 96, 2.0, 1.6),
        # the same at the clinical size, whose volume is twice the L2
        _case("view_512", "view", 512, 512, 256, 1024, 768, 0.5, 0.388),
        # a DVF-update view, non-square slices and odd sizes everywhere
        _case("motion_view_odd", "motion", 201, 173, 97, 301, 211, 1.5, 1.25),
        # deforming the 256x256x160 volume
        _case("warp_256", "warp", 256, 256, 160, 8, 8, 1.0, 0.776),
        # simulating a scan of the 256x256x160 volume
        _case("views_256", "views", 256, 256, 160, 512, 384, 1.0, 0.776, 32),
        # forward and adjoint of one view
        _case("pair_256", "pair", 256, 256, 160, 512, 384, 1.0, 0.776),
        # static SART, the smallest whole reconstruction: latency and launches count
        _case("static_64", "loop", 64, 64, 64, 128, 96, 2.0, 1.6, 60, motion=False, ops="11111",
              storage=0, interp=0, fp_sum=0, geom64=0, subset=1),
        # an outer iteration (image pass, DVF pass) of a motion-compensated scan
        _case("motion_128", "loop", 128, 128, 96, 256, 192, 2.0, 1.2, 360, motion=True, ops="10",
              storage=0, interp=0, fp_sum=0, geom64=0, subset=1),
        # the same at the benchmark workload's size
        _case("motion_256", "loop", 256, 256, 160, 512, 384, 1.0, 0.776, 660, motion=True,
              ops="10", storage=0, interp=0, fp_sum=0, geom64=0, subset=1),
        # image passes in the most exact mode: Kahan sums, FP64 geometry, exact warp weights
        _case("precise_128", "loop", 128, 128, 96, 256, 192, 2.0, 1.2, 24, motion=True, ops="1",
              storage=0, interp=1, fp_sum=2, geom64=1, subset=1),
        # the uneven batch, ordered subsets, 16-bit storage
        _case("batch_8", "batch", 256, 256, 128, 512, 384, 1.0, 1.238, 60, problems=8, ops="10",
              storage=1, interp=0, fp_sum=0, geom64=0, subset=10),
        # the gateway's call with host arrays, a short motion-compensated scan
        _case("host_128", "host", 128, 128, 96, 256, 192, 2.0, 1.2, 120, motion=True, ops="10"),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["view", "motion", "warp", "views", "pair", "loop", "loop", "batch", "host"])
    top = {"view": 384, "motion": 320, "warp": 288, "views": 256, "pair": 288, "loop": 256,
           "batch": 160, "host": 144}[kind]
    nx = _logint(rng, 48, top)
    square = kind in ("batch", "loop") or rng.random() < 0.5
    ny = nx if square else max(40, min(top, nx + rng.randint(-24, 24)))
    nz = max(24, int(nx * rng.uniform(0.45, 1.0)))
    na = max(48, int(nx * rng.uniform(1.4, 2.1)))
    nb = max(40, int(na * rng.uniform(0.6, 0.8)))
    vox = round(256.0 / nx, 4)
    # the detector covers the slice magnified by 1.5, with a margin
    pitch = round(1.5 * 1.1 * nx * vox / na, 4)
    c = _case("", kind, nx, ny, nz, na, nb, vox, pitch)
    del c["name"]
    if kind == "views":
        c["views"] = rng.randint(2, 32)
    if kind in ("loop", "host"):
        c["views"] = rng.randint(11, 97)
        c["motion"] = rng.random() < 0.7
        c["ops"] = rng.choice(["1", "10", "101"]) if c["motion"] else rng.choice(["1", "11", "10"])
    if kind == "loop":
        c.update(storage=rng.choice([0, 0, 1, 2]), interp=rng.choice([0, 0, 1]), fp_sum=0,
                 geom64=0, subset=rng.choice([1, 1, 1, 4, 7]))
        if rng.random() < 0.3:
            c.update(fp_sum=rng.choice([1, 2]), geom64=rng.choice([0, 1]), subset=1, ops="1")
    if kind == "batch":
        c.update(views=rng.randint(11, 47), problems=rng.randint(2, 5), ops="10",
                 storage=rng.choice([0, 1, 2]), interp=0, fp_sum=0, geom64=0,
                 subset=rng.choice([1, 5, 10]))
    return c


# ------------------------------------------------------------------ the inputs
def _geo(c):
    f = np.float32
    return dict(nx=c["nx"], ny=c["ny"], nz=c["nz"], na=c["na"], nb=c["nb"],
                SO=float(f(synthetic.SAD_MM / c["vox"])), SD=float(f(synthetic.SDD_MM / c["vox"])),
                da=float(f(c["pitch"] / c["vox"])), db=float(f(c["pitch"] / c["vox"])),
                ai=float(-(f(c["na"]) / f(2) - f(0.5))), bi=float(-(f(c["nb"]) / f(2) - f(0.5))),
                dx=1.0)


def _args(g):
    return (g["SO"], g["SD"], g["da"], g["na"], g["ai"], g["db"], g["nb"], g["bi"], g["nx"],
            g["ny"], g["nz"])


class _Phantom:
    """Ten ellipsoids and a lesion, in voxels: as synthetic.phantom, rotated about z."""

    def __init__(self, g, seed):
        rng = np.random.default_rng(seed)
        s = g["nx"] / 256.0
        self.c = rng.uniform(-50, 50, (11, 3)) * s * np.array([1, 1, g["nz"] / g["nx"] * 1.4])
        self.r = rng.uniform(8, 40, (11, 3)) * s
        self.r[10] = rng.uniform(6, 12, 3) * s
        self.th = rng.uniform(0, math.pi, 11)
        self.mu = rng.uniform(0, 0.04, 11)
        self.mu[10] = 0.06
        self.g = g

    def volume(self):
        g = self.g
        x = torch.arange(g["nx"], device=DEV) + 0.5 - g["nx"] / 2
        y = (torch.arange(g["ny"], device=DEV) + 0.5 - g["ny"] / 2)[:, None]
        z = (torch.arange(g["nz"], device=DEV) + 0.5 - g["nz"] / 2)[:, None, None]
        v = torch.zeros((g["nz"], g["ny"], g["nx"]), device=DEV)
        for c, r, th, mu in zip(self.c, self.r, self.th, self.mu):
            ct, st = math.cos(th), math.sin(th)
            p, q = (x - c[0]) * ct + (y - c[1]) * st, (y - c[1]) * ct - (x - c[0]) * st
            v += mu * (((p / r[0]) ** 2 + (q / r[1]) ** 2 + ((z - c[2]) / r[2]) ** 2) <= 1).float()
        return v

    def projections(self, angles, shift_z):
        """Line integrals in the projector's units (slabs of the driving axis)."""
        g = self.g
        out = torch.zeros((len(angles), g["nb"], g["na"]), device=DEV)
        ya = (torch.arange(g["na"], device=DEV) + g["ai"]) * g["da"]
        zb = ((torch.arange(g["nb"], device=DEV) + g["bi"]) * g["db"])[:, None]
        for v, (a, dz) in enumerate(zip(angles, shift_z)):
            ca, sa = math.cos(a), math.sin(a)
            sx, sy = -g["SO"] * ca, -g["SO"] * sa
            x20 = g["SD"] - g["SO"]
            ex, ey = x20 * ca - ya * sa - sx, ya * ca + x20 * sa - sy
            drive = torch.maximum(ex.abs(), ey.abs())
            for c, r, th, mu in zip(self.c, self.r, self.th, self.mu):
                ct, st = math.cos(th), math.sin(th)
                o = ((sx - c[0]) * ct + (sy - c[1]) * st, (sy - c[1]) * ct - (sx - c[0]) * st,
                     -(c[2] + dz))
                o0, o1, o2 = (o[i] / r[i] for i in range(3))
                d0, d1, d2 = (ex * ct + ey * st) / r[0], (ey * ct - ex * st) / r[1], zb / r[2]
                aa = d0 * d0 + d1 * d1 + d2 * d2
                bb = d0 * o0 + d1 * o1 + d2 * o2
                disc = bb * bb - aa * (o0 * o0 + o1 * o1 + o2 * o2 - 1)
                out[v] += mu * (2 * disc.clamp_min(0).sqrt() / aa) * drive
        return out


def _fields(c, g, vols, flows, seed):
    """Six smooth fields whose largest displacement over the scan is 10 mm (z), 3 mm (x, y)."""
    gen = torch.Generator(device="cpu").manual_seed(seed)
    low = torch.randn((1, 6, g["nz"] // 8 + 2, g["ny"] // 8 + 2, g["nx"] // 8 + 2), generator=gen)
    f = torch.nn.functional.interpolate(low.to(DEV), size=(g["nz"], g["ny"], g["nx"]),
                                        mode="trilinear", align_corners=True)[0]
    da, db = float(np.abs(vols - vols[0]).max()), float(np.abs(flows - flows[0]).max())
    for k in range(3):
        peak = (f[k].abs() * da + f[3 + k].abs() * db).max().item()
        s = (10.0 if k == 2 else 3.0) / c["vox"] / max(peak, 1e-6)
        f[k] *= s
        f[3 + k] *= s
    return f.contiguous()


def _scan(c, seed, motion):
    g = _geo(c)
    nv = c["views"]
    rng = np.random.default_rng(seed + 3)
    start = float(rng.uniform(0, 2 * math.pi))
    angles = (start + np.linspace(0, 2 * np.pi, nv, endpoint=False)).astype(np.float32)
    vols, flows = synthetic.breathing(max(nv, 16), seed)
    vols, flows = vols[:nv].copy(), flows[:nv].copy()
    if not motion:
        vols, flows = np.zeros(nv, np.float32), np.zeros(nv, np.float32)
    ph = _Phantom(g, seed)
    shift = (vols - vols[0]) * (5.0 / c["vox"] / 16.0)
    return g, ph, angles, vols, flows, ph.projections(angles, shift)


STORAGE = {0: torch.float32, 1: torch.bfloat16, 2: torch.float16}


def _context():
    return m.Context(0, stream=torch.cuda.current_stream())


def _loop_state(c, seed):
    g, _, angles, vols, flows, proj = _scan(c, seed, c["motion"])
    dt = STORAGE[c["storage"]]
    shape = (g["nz"], g["ny"], g["nx"])
    f0 = _fields(c, g, vols, flows, seed + 1).to(dt) if c["motion"] else None
    return dict(geo=g, n_views=c["views"], lambda_=1.0, angles=angles, volumes=vols, flows=flows,
                img=torch.zeros(shape, device=DEV), proj=proj.to(dt),
                fields=None if f0 is None else f0.clone(),
                resid=torch.zeros_like(proj), norm=torch.zeros(len(c["ops"]) * c["views"],
                                                               device=DEV)), f0


def _options(c):
    return m.default_options(storage=c["storage"], interp=c["interp"], fp_sum=c["fp_sum"],
                             geom64=c["geom64"], subset=c["subset"])


def _batch_cases(c):
    """The problems of a batch: the named size first, the others cut down from it."""
    rng = np.random.default_rng(11)
    out = []
    for i in range(c["problems"]):
        s = 1.0 if i == 0 else float(rng.uniform(0.4, 0.9))
        nx = max(32, int(c["nx"] * s) // 8 * 8 + (3 if i == 2 else 0))
        q = dict(c, nx=nx, ny=nx, nz=max(24, int(c["nz"] * s)), na=max(48, int(c["na"] * s)),
                 nb=max(40, int(c["nb"] * s)), vox=round(c["vox"] / s, 4), motion=True)
        q["pitch"] = round(1.5 * 1.1 * nx * q["vox"] / q["na"], 4)
        out.append(q)
    return out


def prepare(case, seed):
    c = case
    kind = c["kind"]
    ctx = _context()
    s = dict(case=c, ctx=ctx)
    if kind == "loop":
        s["q"], s["f0"] = _loop_state(c, seed)
        s["opt"], s["op"] = _options(c), np.array([int(o) for o in c["ops"]], np.int32)
        return s
    if kind == "batch":
        both = [_loop_state(q, seed + 100 * i) for i, q in enumerate(_batch_cases(c))]
        for q, _ in both:
            q["resid"] = None
        s["qs"], s["f0s"] = [b[0] for b in both], [b[1] for b in both]
        s["opt"], s["op"] = _options(c), np.array([int(o) for o in c["ops"]], np.int32)
        return s
    if kind == "host":
        g, _, angles, vols, flows, proj = _scan(c, seed, c["motion"])
        it = dict(n_iter=len(c["ops"]), op_iter=np.array([int(o) for o in c["ops"]], np.int32),
                  n_views=c["views"], outIter=1, volumes=vols, flows=flows, angles=angles,
                  err_weights=np.ones(c["views"], np.float32))
        it["lambda"] = 1.0
        if c["motion"]:
            f = _fields(c, g, vols, flows, seed + 1).cpu().numpy()
            it.update(zip(("alpha_x", "alpha_y", "alpha_z", "beta_x", "beta_y", "beta_z"), f))
        para = dict(g, ai=0.0, bi=0.0)  # the gateway shifts the detector offsets itself
        s.update(img=np.zeros((g["nz"], g["ny"], g["nx"]), np.float32), proj=proj.cpu().numpy(),
                 geo=para, it=it)
        return s
    g, ph, angles, vols, flows, proj = _scan(dict(c, views=max(2, c["views"])), seed, True)
    s.update(geo=g, args=_args(g), angles=angles[:c["views"]], angle=float(angles[1]),
             img=ph.volume(), meas=proj[1].contiguous())
    shape, det = tuple(s["img"].shape), (g["nb"], g["na"])

    def vol(n):
        return [torch.zeros(shape, device=DEV) for _ in range(n)]

    if kind in ("view", "motion"):
        # the current estimate: the phantom blurred, as some iterations leave it
        s["img"] = torch.nn.functional.avg_pool3d(s["img"][None], 5, 1, 2)[0].contiguous()
    if kind == "view":
        s["x"], s["tmp"], s["den"], s["ones"] = vol(4)
        s["resid"], s["fp"] = (torch.zeros(det, device=DEV) for _ in range(2))
    if kind == "motion":
        s["f0"] = _fields(c, g, vols, flows, seed + 1)
        s["f"] = [f.clone() for f in s["f0"]]
        s["tmp"], s["aux"] = vol(2)
        s["resid"], s["fp"] = (torch.zeros(det, device=DEV) for _ in range(2))
        s["vd"], s["fd"] = float(vols[1] - vols[0]), float(flows[1] - flows[0])
    if kind == "warp":
        # two breathing phases apart, as in the scan: amplitude and flow differences
        vv, ff = synthetic.breathing(16, seed)
        s["v"], s["w"] = float(vv[9] - vv[0]), float(ff[9] - ff[0])
        s["f6"] = _fields(c, g, vv, ff, seed + 1)
        s["f"] = list(s["f6"])
        s["f16"] = s["f6"].to(torch.bfloat16)
        s["out"], s["back"] = vol(2)
        s["o16"] = torch.zeros(shape, device=DEV, dtype=torch.bfloat16)
        s["disp"], s["inv"] = vol(3), vol(3)
    if kind == "views":
        s["out"] = torch.zeros((c["views"],) + det, device=DEV)
    if kind == "pair":
        s["fp"], s["bp"] = torch.zeros(det, device=DEV), torch.zeros(shape, device=DEV)
    return s


# ---------------------------------------------------------------------- a pass
def run(state):
    s = state
    c, ctx = s["case"], s["ctx"]
    kind = c["kind"]
    if kind == "loop":
        q = s["q"]
        q["img"].zero_()
        if s["f0"] is not None:
            q["fields"].copy_(s["f0"])
        ctx.aumisart_device(n_iter=len(s["op"]), op_iter=s["op"], options=s["opt"], **q)
        return dict(img=q["img"], resid=q["resid"], norm=q["norm"],
                    **({} if s["f0"] is None else {"fields": q["fields"]}))
    if kind == "batch":
        for q, f0 in zip(s["qs"], s["f0s"]):
            q["img"].zero_()
            q["fields"].copy_(f0)
        ctx.batch_run(s["qs"], n_iter=len(s["op"]), op_iter=s["op"], options=s["opt"])
        return [dict(img=q["img"], norm=q["norm"], fields=q["fields"]) for q in s["qs"]]
    if kind == "host":
        return gateway.entry_AUMISART(s["img"], s["proj"], s["geo"], s["it"], ctx)
    g, args, a = s["geo"], s["args"], s["angle"]
    n3, n2 = (g["nx"], g["ny"], g["nz"]), (g["na"], g["nb"], 1)
    if kind == "view":
        x, resid = s["x"], s["resid"]
        x.copy_(s["img"])
        resid.copy_(s["meas"])
        ctx.host_projection(s["fp"], x, a, *args)
        ctx.host_add(resid, s["fp"], *n2, -1.0)
        ctx.host_backprojection(s["tmp"], resid, a, *args)
        ctx.host_initial(s["ones"], *n3, 1.0)
        ctx.host_projection(s["fp"], s["ones"], a, *args)
        ctx.host_backprojection(s["den"], s["fp"], a, *args)
        ctx.host_division(s["tmp"], s["den"], *n3)
        ctx.host_add(x, s["tmp"], *n3, 1.0)
        return dict(img=x, resid=resid, ones=s["fp"])
    if kind == "motion":
        img, f, resid, aux, tmp = s["img"], s["f"], s["resid"], s["aux"], s["tmp"]
        vd, fd = s["vd"], s["fd"]
        for k in range(6):
            f[k].copy_(s["f0"][k])
        # gradient axis 1 pairs with alpha_y / beta_y, axis 2 with alpha_x / beta_x
        pairs = ((1, vd, 1), (0, vd, 2), (2, vd, 3), (4, fd, 1), (3, fd, 2), (5, fd, 3))
        resid.copy_(s["meas"])
        ctx.host_projection(s["fp"], img, a, *args)
        ctx.host_add(resid, s["fp"], *n2, -1.0)
        ctx.host_initial(aux, *n3, 0.0)
        for k, w, ind in pairs:
            ctx.host_add2(aux, f[k], *n3, img, w, ind)
        ctx.host_projection(s["fp"], aux, a, *args)
        ctx.host_add(resid, s["fp"], *n2, 1.0)
        nb = ctx.snrm2(resid.numel(), s["meas"])
        nr = ctx.snrm2(resid.numel(), resid)
        ctx.host_backprojection(tmp, resid, a, *args)
        ctx.host_initial2(aux, *n3, img, -vd, -fd)
        ctx.host_projection(s["fp"], aux, a, *args)
        ctx.host_backprojection(aux, s["fp"], a, *args)
        ctx.host_division(tmp, aux, *n3)
        for k, w, ind in pairs:
            ctx.host_add2(f[k], tmp, *n3, img, -w, ind)
        return dict(resid=resid, fp=s["fp"], den=aux, fields=f, norms=[nb, nr])
    if kind == "warp":
        v, w = s["v"], s["w"]
        ctx.host_deform(s["out"], s["img"], *n3, v, w, *s["f"])
        ctx.host_deform(s["back"], s["out"], *n3, -v, -w, *s["f"])
        ctx.deform_ex(s["o16"], s["img"], *n3, v, w, s["f16"], interp=m.INTERP_EXACT)
        ctx.kernel_forwardDVF(*s["disp"], *s["f"], v, w, *n3)
        out = dict(out=s["out"], back=s["back"], o16=s["o16"], disp=s["disp"])
        if g["nx"] == g["ny"]:
            ctx.invert_dvf(*s["inv"], *s["f"], v, w, *n3, 8)
            out["inv"] = s["inv"]
        return out
    if kind == "views":
        ctx.projection_views(s["out"], s["img"], s["angles"], *args)
        return s["out"]
    ctx.host_projection(s["fp"], s["img"], a, *args)
    ctx.host_backprojection_adjoint(s["bp"], s["meas"], a, *args)
    return dict(fp=s["fp"], bp=s["bp"])


# ------------------------------------------------- what a pass cannot do without
def _view_flops(c):
    """Multiply-adds of one projection and one backprojection of a view: a ray
    meets about (1 + cell width)^2 voxels per slab, a voxel (1 + its width on
    the detector)^2 cells, at most the whole volume's shadow."""
    w = c["pitch"] / c["vox"] / 1.5
    rays = c["na"] * c["nb"] * min(1.0, (c["nx"] / (c["na"] * w)) * (c["nz"] / (c["nb"] * w)))
    fp = rays * max(c["nx"], c["ny"]) * (1 + w) ** 2
    bp = c["nx"] * c["ny"] * c["nz"] * (1 + 1 / w) ** 2
    return fp, bp


def work(case):
    c = case
    V, P, kind = c["nx"] * c["ny"] * c["nz"], c["na"] * c["nb"], c["kind"]
    fp, bp = _view_flops(c)
    if kind == "batch":
        w = [work(dict(q, kind="loop")) for q in _batch_cases(c)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    if kind == "view":  # volume and measurement in; volume, residual and ones-projection out
        return {"bytes": 4 * (2 * V + 3 * P), "flops": 4 * fp + 4 * bp}
    if kind == "motion":  # volume and fields in; fields, denominator, residual out
        return {"bytes": 4 * (14 * V + 3 * P), "flops": 6 * fp + 4 * bp + 40 * V}
    if kind == "warp":  # two warps, a 16-bit one, the displacement and its inverse
        n = (8 + 8) * 4 + 4 + 14 + 9 * 4 + (9 * 4 if c["nx"] == c["ny"] else 0)
        return {"bytes": n * V, "flops": (3 * 30 + 9 + (8 * 60 if c["nx"] == c["ny"] else 0)) * V}
    if kind == "views":
        return {"bytes": 4 * (V + c["views"] * P), "flops": 2 * fp * c["views"]}
    if kind == "pair":
        return {"bytes": 4 * (2 * V + 2 * P), "flops": 4 * fp}
    # loops: views follow one another, so every view reads and writes the
    # volume, and with motion reads the six fields for each warp (image pass)
    # or reads and writes them (DVF pass)
    es = 4 if kind == "host" or c["storage"] == 0 else 2
    flops = nbytes = 0.0
    for o in c["ops"]:
        if o == "1":
            per = 8 * V + (es + 4) * P + (12 * es * V if c["motion"] else 0)
            nbytes += c["views"] * per
            flops += c["views"] * (4 * fp + 4 * bp + (70 * V if c["motion"] else 2 * V))
        else:
            n = c["views"] - 1 if c["motion"] else (c["views"] + 8) // 10
            nbytes += n * (4 * V + es * P + 12 * es * V)
            flops += n * (6 * fp + 4 * bp + 40 * V)
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------ the same in 64 bits
def _axis(lo, hi, n, k):
    """Index floor(lo) + k, its overlap with [lo, hi] over hi - lo, and whether it is inside."""
    i = torch.floor(lo) + k
    w = (torch.minimum(i + 1, hi) - torch.maximum(i, lo)) / (hi - lo)
    ok = (i <= torch.floor(hi)) & (i >= 0) & (i <= n - 1)
    return i.clamp(0, n - 1).long(), torch.where(ok, w, torch.zeros_like(w))


def _fp64(img, angle, g):
    """src/cu_projection.cu:15-145 in 64 bits: img [nz, ny, nx] -> [nb, na]."""
    img = img.double()
    f8 = dict(dtype=torch.float64, device=DEV)
    a = float(np.float32(angle))
    ca, sa = math.cos(a), math.sin(a)
    x1, y1, x20 = -g["SO"] * ca, -g["SO"] * sa, g["SD"] - g["SO"]
    y20 = (torch.arange(g["na"], **f8) + g["ai"]) * g["da"]
    z2 = (torch.arange(g["nb"], **f8) + g["bi"]) * g["db"]
    x21, y21 = x20 * ca - y20 * sa - x1, y20 * ca + x20 * sa - y1
    xd = x21.abs() > y21.abs()
    out = torch.zeros((g["nb"], g["na"]), **f8)
    for drive in (True, False):
        cols = torch.nonzero(xd == drive).flatten()
        if not len(cols):
            continue
        hs, hc = g["da"] / 2 * sa, g["da"] / 2 * ca
        xl, xr = x21[cols] - hs, x21[cols] + hs
        yl, yr = y21[cols] - hc, y21[cols] + hc
        if drive:
            nd, nu, num, den, main, u0, src = g["nx"], g["ny"], (yl, yr), (xl, xr), x21[cols], y1, x1
        else:
            nd, nu, num, den, main, u0, src = g["ny"], g["nx"], (xl, xr), (yl, yr), y21[cols], x1, y1
        rat = torch.stack([n / d for n in num for d in den])          # [4, cols]
        rz = torch.stack([(z2[:, None] + e) / main for e in (-g["db"] / 2, g["db"] / 2)])
        step = max(1, min(nd, (8 << 20) // (g["nb"] * len(cols))))
        acc = torch.zeros((g["nb"], len(cols)), **f8)
        for d0 in range(0, nd, step):
            d = torch.arange(d0, min(nd, d0 + step), device=DEV)
            dc = d.double() + 0.5 - nd / 2 - src
            cu = rat[:, None, :] * dc[:, None] + u0 + nu // 2           # [4, slabs, cols]
            ulo, uhi = cu.amin(0), cu.amax(0)
            cz = rz[:, None] * dc[:, None, None] + g["nz"] // 2         # [2, slabs, nb, cols]
            zlo, zhi = cz.amin(0), cz.amax(0)
            ku = int((torch.floor(uhi) - torch.floor(ulo)).max()) + 1
            kz = int((torch.floor(zhi) - torch.floor(zlo)).max()) + 1
            for i in range(ku):
                u, wu = _axis(ulo, uhi, nu, i)
                at = (u * g["nx"] + d[:, None]) if drive else (d[:, None] * g["nx"] + u)
                for j in range(kz):
                    z, wz = _axis(zlo, zhi, g["nz"], j)
                    v = img.reshape(-1)[z * (g["nx"] * g["ny"]) + at[:, None, :]]
                    acc += (v * wu[:, None, :] * wz).sum(0)
        out[:, cols] = acc
    return out


def _bp64(proj, angle, g):
    """src/cu_backprojection.cu:49-170 in 64 bits: proj [nb, na] -> [nz, ny, nx]."""
    f8 = dict(dtype=torch.float64, device=DEV)
    proj = proj.double()
    a = float(np.float32(angle))
    ca, sa = math.cos(a), math.sin(a)
    xc = torch.arange(g["nx"], **f8) - g["nx"] // 2 + 0.5
    yc = (torch.arange(g["ny"], **f8) - g["ny"] // 2 + 0.5)[:, None]
    zc = (torch.arange(g["nz"], **f8) - g["nz"] // 2 + 0.5)[:, None, None]
    t, u = xc * ca + yc * sa, yc * ca - xc * sa
    rl, rr, r0 = (g["SD"] / (t + e + g["SO"]) for e in (-0.5, 0.5, 0.0))
    e = torch.stack([rl * (u - 0.5), rl * (u + 0.5), rr * (u + 0.5), rr * (u - 0.5), r0 * u])
    amax, amin = (v / g["da"] - g["ai"] + 0.5 for v in (e.amax(0), e.amin(0)))
    out = torch.zeros((g["nz"], g["ny"], g["nx"]), **f8)
    step = max(1, (16 << 20) // (g["nx"] * g["ny"]))
    for z0 in range(0, g["nz"], step):
        zz = zc[z0:z0 + step]
        e = torch.stack([rl * zz, rr * zz, r0 * (zz + 0.5), r0 * (zz - 0.5)])
        bmax, bmin = (v / g["db"] - g["bi"] + 0.5 for v in (e.amax(0), e.amin(0)))
        ia0, ib0 = torch.floor(amin).clamp_min(0), torch.floor(bmin).clamp_min(0)
        alim, blim = amax.clamp_max(g["na"]), bmax.clamp_max(g["nb"])
        ka = int((torch.ceil(alim) - ia0).max())
        kb = int((torch.ceil(blim) - ib0).max())
        acc = out[z0:z0 + step]
        for i in range(max(0, ka)):
            ia = ia0 + i
            wa = torch.minimum(ia + 1, amax) - torch.maximum(ia, amin)
            wa = torch.where(ia < alim, wa, torch.zeros_like(wa))
            for j in range(max(0, kb)):
                ib = ib0 + j
                wb = torch.minimum(ib + 1, bmax) - torch.maximum(ib, bmin)
                wb = torch.where(ib < blim, wb, torch.zeros_like(wb))
                at = ib.clamp(0, g["nb"] - 1).long() * g["na"] + ia.clamp(0, g["na"] - 1).long()
                acc += wa * wb * proj.reshape(-1)[at]
    return out


def _adjoint64(proj, angle, g):
    """The transpose of _fp64: proj [nb, na] -> [nz, ny, nx]."""
    x = torch.zeros((g["nz"], g["ny"], g["nx"]), dtype=torch.float64, device=DEV,
                    requires_grad=True)
    # _fp64 is linear in the volume, so its gradient is the transpose
    _fp64(x, angle, g).backward(proj.double())
    return x.grad


def _transposed(shape):
    """The warp's in-slice index: memory position r of a slice stands for (r // ny, r % ny)."""
    nz, ny, nx = shape
    r = torch.arange(nx * ny, device=DEV)
    return (r // ny).view(ny, nx), (r % ny).view(ny, nx)


def _sample64(vol, x, y, z):
    """Trilinear sample at voxel coordinates (clamped at the edges)."""
    nz, ny, nx = vol.shape
    vol, out = vol.reshape(-1), 0.0
    x0, y0, z0 = torch.floor(x), torch.floor(y), torch.floor(z)
    for k in range(8):
        i, j, l = x0 + (k & 1), y0 + ((k >> 1) & 1), z0 + (k >> 2)
        w = ((1 - (x - i).abs()) * (1 - (y - j).abs()) * (1 - (z - l).abs()))
        at = (l.clamp(0, nz - 1).long() * ny + j.clamp(0, ny - 1).long()) * nx + i.clamp(0, nx - 1).long()
        out = out + w * vol[at]
    return out


def _warp64(vol, mx, my, mz):
    """src/cu_deform.cu:79-90 with exact weights: out[q] = vol(iy + my, ix + mx, iz + mz)."""
    ix, iy = _transposed(vol.shape)
    iz = torch.arange(vol.shape[0], device=DEV)[:, None, None]
    return _sample64(vol.double(), iy + my, ix + mx, iz + mz)


def _disp64(f, v, w):
    f = [x.double() for x in f]
    return [f[k] * v + f[3 + k] * w for k in range(3)]


def _invert64(disp, n_iter):
    mx, my, mz = disp
    nz, ny, nx = mx.shape
    X = torch.arange(nx, device=DEV).double()
    Y = torch.arange(ny, device=DEV).double()[:, None]
    Z = torch.arange(nz, device=DEV).double()[:, None, None]
    n = [torch.zeros_like(mx) for _ in range(3)]
    for _ in range(n_iter):
        p = (X + n[0], Y + n[1], Z + n[2])
        n = [-_sample64(d, *p) for d in (my, mx, mz)]
    return [n[1], n[0], n[2]]


def _ratio64(num, den):
    q = num / den
    return torch.where(torch.isfinite(q), q, torch.zeros_like(q))


def _image_views64(q, opt, ops):
    """Image passes, one view at a time, in 64 bits."""
    g, img = q["geo"], torch.zeros(q["img"].shape, dtype=torch.float64, device=DEV)
    proj, fields = q["proj"].double(), q["fields"]
    ones = torch.ones_like(img)
    resid, norm = torch.zeros_like(proj), torch.zeros((len(ops), len(proj)), dtype=torch.float64)
    for it in range(len(ops)):
        for v in range(q["n_views"]):
            a = q["angles"][v]
            x = img
            if fields is not None:
                dv, df = (float(t[v] - t[0]) for t in (q["volumes"], q["flows"]))
                x = _warp64(img, *_disp64(fields, dv, df))
            resid[v] = proj[v] - _fp64(x, a, g)
            r = _ratio64(_bp64(resid[v], a, g), _bp64(_fp64(ones, a, g), a, g))
            if fields is not None:
                r = _warp64(r, *_disp64(fields, -dv, -df))
            img = img + r
            norm[it, v] = resid[v].norm() / proj[v].norm()
    return dict(img=img, resid=resid, norm=norm.flatten())


def exact(case, seed):
    c = case
    kind = c["kind"]
    if kind == "batch":
        return None  # the DVF pass divides by a signed sum: no 64-bit value to compare with
    if kind in ("loop", "host"):
        size = c["nx"] * c["ny"] * c["nz"] * c["views"] * len(c["ops"])
        if "0" in c["ops"] or c.get("subset", 1) != 1 or size > 1.3e8 or c.get("storage", 0):
            return None
    s = prepare(case, seed)
    if kind == "host":
        q, f0 = _loop_state(dict(c, storage=0), seed)
        o = _image_views64(q, None, c["ops"])
        ax = torch.zeros_like(q["img"]) if f0 is None else f0[0].double()
        return o["img"], o["norm"].reshape(-1, 1), ax, o["resid"]
    if kind == "loop":
        o = _image_views64(s["q"], s["opt"], c["ops"])
        if s["f0"] is not None:
            o["fields"] = s["f0"].double()
        return o
    g, a = s["geo"], s["angle"]
    if kind == "view":
        x = s["img"].double()
        resid = s["meas"].double() - _fp64(x, a, g)
        ones = _fp64(torch.ones_like(x), a, g)
        return dict(img=x + _ratio64(_bp64(resid, a, g), _bp64(ones, a, g)), resid=resid, ones=ones)
    if kind == "motion":
        img, f = s["img"].double(), s["f0"].double()
        d = [torch.zeros_like(img) for _ in range(3)]
        d[0][:, :, :-1] = img[:, :, 1:] - img[:, :, :-1]
        d[1][:, :-1] = img[:, 1:] - img[:, :-1]
        d[2][:-1] = img[1:] - img[:-1]
        nz, ny, nx = img.shape

        def turned(t):  # the field at the transposed in-slice index iy + ix*ny
            return t.reshape(nz, nx, ny).transpose(1, 2)

        aux = sum(turned(f[k]) * w * d[i] for k, w, i in (
            (1, s["vd"], 0), (0, s["vd"], 1), (2, s["vd"], 2), (4, s["fd"], 0), (3, s["fd"], 1),
            (5, s["fd"], 2)))
        resid = s["meas"].double() - _fp64(img, a, g) + _fp64(aux, a, g)
        fp = _fp64((d[0] + d[1] + d[2]) * (-s["vd"] - s["fd"]), a, g)
        # the field update divides by the signed den: no 64-bit value to compare with
        return dict(resid=resid, fp=fp, den=_bp64(fp, a, g), fields=None,
                    norms=[float(s["meas"].double().norm()), float(resid.norm())])
    if kind == "warp":
        disp, dn = _disp64(s["f"], s["v"], s["w"]), _disp64(s["f"], -s["v"], -s["w"])
        out = _warp64(s["img"], *disp)
        r = dict(out=out, back=_warp64(out, *dn),
                 o16=_warp64(s["img"], *_disp64(s["f16"], s["v"], s["w"])), disp=disp)
        if g["nx"] == g["ny"]:
            r["inv"] = _invert64(disp, 8)
        return r
    if kind == "views":
        return torch.stack([_fp64(s["img"], v, g) for v in s["angles"]])
    return dict(fp=_fp64(s["img"], a, g), bp=_adjoint64(s["meas"], a, g))
