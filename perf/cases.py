"""Workloads of the far-field stage, timed through its public entry points.

Each case is one call (or one step) that a program built on this package makes:
a single outbeam's amplitude on the tracer's inner path, one orientation's
amplitude grids in either precision, their Mueller matrices, an orientation
average from host or device arrays, and one gradient step of an inverse
problem.  `listed` holds the sizes of the package's own configurations and
tests; `draw` gives others of the same ranges, odd ones among them.

The FP32 form's results are single-precision numbers carried in
double-precision arrays; a program that asked for FP32 keeps them as float32,
and so do the cases that use it (into arrays of its own, kept from call to
call).  FP64 results stay as they are.

`exact` evaluates the same sums in 64 bits with plain torch: the facets'
aperture integrals from their closed form, the second divided difference of
e^{ix} at the vertex phases, which has no singular directions.
"""
import math
from fractions import Fraction

import numpy as np
import torch

import abt_b200
from abt_b200 import autograd as _ag
from abt_b200.diff import BatchGraph, diff_batch_dev

LAM = 0.532
FAR = 1.0e6                                # distance of the far-field points
PI_REF = float(np.float32(math.pi))        # the reference's pi, a single-precision literal
C_KY = float(np.float32(0.999999))         # its clamp of the aperture's y component
C_FWD = float(np.float32(0.999))           # its limit for the forward scattering plane
_NPAR = 18


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # the tracer's memory-saving loop: one outbeam per call, host arrays in and out
        dict(name="diffraction_one", kind="diffraction", mesh=14, beams=1, corners=3, ntheta=181,
             nphi=180, fast=False),
        # one orientation of the plain method (column of a few micrometres), reference arithmetic
        dict(name="diff_main_fp64", kind="main", prec="fp64", mesh=21, beams=1700, corners=3,
             ntheta=181, nphi=180, fast=False),
        # polygonal facets, an odd grid and the field-of-view test, reference arithmetic
        dict(name="diff_main_fp64_fast", kind="main", prec="fp64", mesh=11, beams=900, corners=8,
             ntheta=301, nphi=97, fast=True),
        # the same orientation as diff_main_fp64 in the FP32 form
        dict(name="diff_main_fp32", kind="main", prec="fp32", mesh=21, beams=1700, corners=3,
             ntheta=181, nphi=180, fast=False),
        # an orientation's amplitude grids to Mueller matrices and cross sections
        dict(name="finalise", kind="finalise", ntheta=361, nphi=180, scaling=False),
        # a short orientation average in the reference's arithmetic, energies rescaled
        dict(name="average_fp64", kind="average", prec="fp64", norient=4, mesh=16, beams=700,
             corners=3, ntheta=181, nphi=90, fast=False, scaling=True),
        # the orientation average: rough particle, lists as long as the tracer's (about 3,300)
        dict(name="average_fp32", kind="average", prec="fp32", norient=24, mesh=18, beams=2650,
             corners=3, ntheta=361, nphi=180, fast=False, scaling=False),
        # the same with the field-of-view test, polygons, an odd grid and rescaled energies
        dict(name="average_fp32_fast", kind="average", prec="fp32", norient=16, mesh=16,
             beams=3001, corners=6, ntheta=359, nphi=181, fast=True, scaling=True),
        # a small orientation replayed as a graph: lists already on the device, launches count
        dict(name="replay_small", kind="replay", norient=1, mesh=8, beams=400, ntheta=91, nphi=72,
             fast=False),
        # many small orientations of a coarse particle in one device call
        dict(name="device_many", kind="device", norient=256, mesh=6, beams=150, ntheta=91, nphi=72,
             fast=False),
        # the precision study: 200,000 facets on a fine grid, lists on the device
        dict(name="device_study", kind="device", norient=1, mesh=0, beams=200000, ntheta=721,
             nphi=360, fast=False),
        # one gradient step on a rough plate of 20,000 triangles: loss, vertex and field gradients
        dict(name="gradient_plate", kind="gradient", mesh=72, beams=20600, ntheta=181, nphi=90,
             fast=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["diffraction", "main", "main", "main", "finalise", "average", "average",
                       "replay", "device", "device", "gradient"])
    ntheta, nphi = _log(rng, 61, 721), _log(rng, 48, 360)
    fast = rng.random() < 0.3
    if kind == "diffraction":
        while ntheta * nphi > 65536:
            ntheta, nphi = _log(rng, 61, 721), _log(rng, 48, 360)
        return dict(kind=kind, mesh=rng.randint(4, 40), beams=1, corners=rng.randint(3, 8),
                    ntheta=ntheta, nphi=nphi, fast=fast)
    if kind == "finalise":
        return dict(kind=kind, ntheta=ntheta, nphi=nphi, scaling=rng.random() < 0.4)
    if kind == "gradient":
        ntheta, nphi = _log(rng, 61, 181), _log(rng, 36, 120)
        return dict(kind=kind, mesh=rng.randint(8, 60), beams=_log(rng, 200, 12000),
                    ntheta=ntheta, nphi=nphi, fast=False)
    prec = rng.choice(["fp64", "fp32"]) if kind in ("main", "average") else "fp32"
    # facet-bins of one pass: the largest listed case has 5.2e10
    most = 1.5e9 if prec == "fp64" else 8e9
    norient = 1 if kind in ("main", "replay") else _log(rng, 2, 200)
    mesh = rng.randint(4, 24)
    beams = _log(rng, 40, 20000)
    while norient * (beams + 2 * mesh * mesh) * ntheta * nphi > most:
        beams = max(20, beams // 2)
        norient = max(1, norient // 2)
        ntheta = max(61, int(ntheta * 0.8))
        mesh = max(4, mesh - 2)
    c = dict(kind=kind, norient=norient, mesh=mesh, beams=beams, ntheta=ntheta, nphi=nphi, fast=fast)
    if kind in ("main", "average"):
        c.update(prec=prec, corners=rng.choice([3, 3, 3, rng.randint(4, 8)]))
    if kind == "average":
        c.update(scaling=rng.random() < 0.4)
    return c


# ------------------------------------------------------------------ the inputs

def _angles(case):
    return (np.arange(case["ntheta"]) * (180.0 / (case["ntheta"] - 1)) * PI_REF / 180.0,
            np.arange(case["nphi"]) * (360.0 / case["nphi"]) * PI_REF / 180.0)


def _unit(v):
    return v / np.linalg.norm(v, axis=-1, keepdims=True)


def _perp(rng, p):
    r = rng.normal(size=p.shape)
    return _unit(r - (r * p).sum(-1, keepdims=True) * p)


def _rotation(rng):
    q, r = np.linalg.qr(rng.normal(size=(3, 3)))
    q = q * np.sign(np.diag(r))
    return q if np.linalg.det(q) > 0 else -q


def _plate(rng, n, half=8.0, thick=4.0, rough=0.05):
    """A rough square plate: two sheets of n x n cells, two triangles a cell, outward faces."""
    s = np.linspace(-half, half, n + 1)
    gx, gy = np.meshgrid(s, s, indexing="ij")
    idx = np.arange((n + 1) ** 2).reshape(n + 1, n + 1)
    a, b, c, d = (x.ravel() for x in (idx[:-1, :-1], idx[1:, :-1], idx[1:, 1:], idx[:-1, 1:]))
    up = np.concatenate([np.stack([a, b, c], 1), np.stack([a, c, d], 1)])
    verts = np.concatenate([np.stack([gx.ravel(), gy.ravel(),
                                      z + rng.normal(0, rough, gx.size)], 1)
                            for z in (thick / 2, -thick / 2)])
    return verts, np.concatenate([up, up[:, ::-1] + (n + 1) ** 2])


def _polygons(rng, n, corners, box=8.0):
    """n flat polygons of 3 .. corners vertices (every face its own vertices)."""
    nv = rng.integers(3, corners + 1, size=n)
    off = np.concatenate([[0], np.cumsum(nv)]).astype(np.int64)
    nrm = _unit(rng.normal(size=(n, 3)))
    e1 = _perp(rng, nrm)
    e2 = np.cross(nrm, e1)
    face = np.repeat(np.arange(n), nv)
    k = np.arange(off[-1]) - off[face]
    ang = 2 * np.pi * (k + rng.uniform(0, 0.6, size=len(k))) / nv[face]
    rad = rng.uniform(0.3, 1.2, size=n)[face]
    centre = rng.uniform(-box, box, size=(n, 3))
    verts = centre[face] + rad[:, None] * (np.cos(ang)[:, None] * e1[face]
                                           + np.sin(ang)[:, None] * e2[face])
    return verts, off


def _records(rng, m, prop, fi, sigma):
    ob = np.zeros(m, dtype=abt_b200.OUTBEAM_DTYPE)
    z = 0.13 * np.exp(rng.normal(-1.0, sigma, size=(m, 4)) + 2j * np.pi * rng.uniform(size=(m, 4)))
    ob["ampl"][:, 0::2], ob["ampl"][:, 1::2] = z.real, z.imag
    ob["prop_out"], ob["vk7"] = prop, _perp(rng, prop)
    ob["fov"] = rng.uniform(0.3, 0.8, size=m)
    ob["fi"] = fi + 1
    return ob


def _lit(verts, off, vi):
    """External diffraction: the half of the faces turned most to the incidence (0,0,-1) emits the
    incident field with its path phase, rotated into the face's own plane."""
    first = vi[off[:-1, None] + np.arange(3)] - 1
    tri = verts[first]
    nrm = np.cross(tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0])
    area = 0.5 * np.linalg.norm(nrm, axis=1)
    nrm = _unit(nrm)
    lit = np.sort(np.argsort(-nrm[:, 2], kind="stable")[:len(nrm) // 2])
    inc = np.array([0.0, 0.0, -1.0])
    ext = np.zeros(len(lit), dtype=abt_b200.OUTBEAM_DTYPE)
    vk = _unit(np.cross(nrm[lit], inc) + 1e-9 * np.array([1.0, 0.0, 0.0]))
    c, s = vk[:, 0], -vk[:, 1]
    ph = np.exp(1j * (2 * PI_REF / LAM) * (verts[:, 2].max() - tri[lit, :, 2].mean(1)))
    z = np.stack([c * ph, s * ph, -s * ph, c * ph], 1)
    ext["ampl"][:, 0::2], ext["ampl"][:, 1::2] = z.real, z.imag
    ext["prop_out"], ext["vk7"], ext["fov"], ext["fi"] = inc, vk, PI_REF / 2, lit + 1
    return nrm, ext, float((area[lit] * np.maximum(nrm[lit, 2], 0.0)).sum())


def _study(rng, n):
    """The precision study's list: n triangles (edges 0.3-1.5 um) in a 100 um cube, 100 a beam."""
    e1 = _unit(rng.normal(size=(n, 3)))
    e2 = _perp(rng, e1)
    ang = np.sort(rng.uniform(0, 2 * np.pi, size=(n, 3)), axis=1) + np.array([0.0, 0.5, 1.0])
    rad = rng.uniform(0.2, 0.85, size=(n, 1))
    tri = (rng.uniform(0, 100, size=(n, 1, 3)) + (rad * np.cos(ang))[..., None] * e1[:, None]
           + (rad * np.sin(ang))[..., None] * e2[:, None])
    b = -(-n // 100)
    prop = _unit(rng.normal(size=(b, 3)))
    one = _records(rng, b, prop, np.zeros(b, np.int64), 1.5)
    ob = one[np.arange(n) // 100]
    ob["fi"] = np.arange(1, n + 1)
    return dict(off=np.arange(0, 3 * n + 1, 3, dtype=np.int64),
                vi=np.arange(1, 3 * n + 1, dtype=np.int64), verts=[tri.reshape(-1, 3)], beams=[ob],
                exts=[ob[:0]], pin=_params([1.0]))


def _params(cross):
    p = np.zeros(len(cross), dtype=abt_b200.PARAMS_DTYPE)
    for i, g in enumerate(cross):
        p[i] = abt_b200.params(abs=0.02 * g, geo_cross_sec=g, beam_energy_out=0.9 * g,
                               ext_energy_out=1.1 * g)
    return p


def _lists(case, seed):
    """Faces, and per orientation the rotated vertices and the two outbeam lists."""
    rng = np.random.default_rng([seed, 77])
    if case["mesh"] == 0:
        return _study(rng, case["beams"])
    if case.get("corners", 3) == 3:
        v0, f = _plate(rng, case["mesh"])
        off = np.arange(0, 3 * len(f) + 1, 3, dtype=np.int64)
        vi = (f.ravel() + 1).astype(np.int64)
    else:
        v0, off = _polygons(rng, 4 * case["mesh"] ** 2, case["corners"])
        vi = np.arange(1, len(v0) + 1, dtype=np.int64)
    verts, beams, exts, cross = [], [], [], []
    for _ in range(case.get("norient", 1)):
        V = v0 @ _rotation(rng).T
        nrm, ext, g = _lit(V, off, vi)
        # lists of uneven length from orientation to orientation
        m = case["beams"] if case.get("norient", 1) == 1 else int(case["beams"] * rng.uniform(0.6, 1.4)) + 1
        fi = np.sort(rng.integers(0, len(off) - 1, size=m))
        d = _unit(rng.normal(size=(m, 3)))
        d *= np.where((d * nrm[fi]).sum(1) < 0, -1.0, 1.0)[:, None]
        verts.append(V)
        beams.append(_records(rng, m, d, fi, 0.8))
        exts.append(ext)
        cross.append(max(g, 1.0))
    return dict(off=off, vi=vi, verts=verts, beams=beams, exts=exts, pin=_params(cross))


def _grids(case, seed):
    """Amplitude grids as an orientation gives them: a forward peak over a speckle background."""
    rng = np.random.default_rng([seed, 78])
    theta, _ = _angles(case)
    shape = (case["nphi"], case["ntheta"], 2, 2)
    fall = (1.0 / (0.02 + theta ** 2))[None, :, None, None]
    out = []
    for scale in (0.1, 1.0):
        z = rng.normal(size=shape) + 1j * rng.normal(size=shape)
        out.append(np.asfortranarray(scale * fall * (z + 2.0 * np.eye(2))))
    return out


def _device(a):
    a = np.ascontiguousarray(a)
    return torch.from_numpy(a.view(np.uint8).reshape(-1).copy()).cuda()


def prepare(case, seed):
    theta, phi = _angles(case)
    ctx = abt_b200.Context(0)
    s = dict(kind=case["kind"], ctx=ctx, theta=theta, phi=phi, fast=case.get("fast", False),
             scaling=case.get("scaling", False), prec=case.get("prec", "fp64"))
    if case["kind"] == "finalise":
        s["grids"], s["pin"] = _grids(case, seed), _params([300.0])[0]
        return s
    L = _lists(case, seed)
    s["geo"] = dict(verts=L["verts"][0], face_off=L["off"], face_vi=L["vi"])
    s["L"] = L
    nphi, nt = len(phi), len(theta)
    if case["kind"] in ("main", "diffraction"):
        # the program's geometry as the library wants it (Fortran order), ready to be passed
        s["geo"]["verts"] = np.asfortranarray(L["verts"][0])
        if s["prec"] == "fp32":
            s["keep"] = [np.zeros((nphi, nt, 2, 2), np.complex64, order="F") for _ in range(2)]
    elif case["kind"] == "average":
        L["verts"] = [np.asfortranarray(v) for v in L["verts"]]
        pin = [torch.zeros(16 * nphi * nt, dtype=torch.float64).pin_memory(),
               torch.zeros(16 * nt, dtype=torch.float64).pin_memory()]
        s["pinned"] = pin
        s["out"] = (pin[0].numpy().reshape((nphi, nt, 16), order="F"),
                    pin[1].numpy().reshape((nt, 16), order="F"))
        if s["prec"] == "fp32":
            s["keep"] = [np.zeros_like(o, dtype=np.float32) for o in s["out"]]
    elif case["kind"] in ("device", "replay"):
        n = len(L["beams"])
        boff = np.concatenate([[0], np.cumsum([len(b) for b in L["beams"]])]).astype(np.int64)
        eoff = np.concatenate([[0], np.cumsum([len(e) for e in L["exts"]])]).astype(np.int64)
        d = dict(beam=_device(np.concatenate(L["beams"])), vi=torch.from_numpy(L["vi"]).cuda(),
                 ext=_device(np.concatenate(L["exts"] + [np.zeros(1, abt_b200.OUTBEAM_DTYPE)])),
                 verts=torch.from_numpy(np.concatenate([v.ravel(order="F") for v in L["verts"]])).cuda(),
                 pin=_device(L["pin"]),
                 mu=torch.zeros((16, nt, nphi), dtype=torch.float64, device="cuda"),
                 m1=torch.zeros((16, nt), dtype=torch.float64, device="cuda"),
                 pav=torch.zeros(_NPAR, dtype=torch.float64, device="cuda"),
                 per=torch.zeros((n, _NPAR), dtype=torch.float64, device="cuda"))
        s["d"] = d
        s["args"] = (n, d["beam"], boff, d["ext"], eoff, d["verts"], len(L["verts"][0]), L["off"],
                     d["vi"], theta, phi, LAM, d["pin"], d["mu"], d["m1"], d["pav"], d["per"], s["fast"])
        if case["kind"] == "replay":
            s["graph"] = BatchGraph(ctx, torch.cuda.current_stream().cuda_stream, *s["args"])
    elif case["kind"] == "gradient":
        rng = np.random.default_rng([seed, 79])
        s["verts"] = torch.from_numpy(np.ascontiguousarray(L["verts"][0]))
        s["ba"] = torch.from_numpy(L["beams"][0]["ampl"].copy())
        s["ea"] = torch.from_numpy(L["exts"][0]["ampl"].copy())
        s["target"] = _target(case, rng)
    return s


def _target(case, rng):
    """A smooth target pattern (M11 with a forward peak, -M12/M11 of a few per cent)."""
    theta, _ = _angles(case)
    t11 = np.repeat((1e3 / (0.02 + theta ** 2))[None], case["nphi"], 0)
    t11 = t11 * np.exp(0.2 * rng.normal(size=t11.shape))
    return torch.from_numpy(t11), torch.from_numpy(0.05 * t11 * np.sin(theta)[None])


# ------------------------------------------------------------------ one pass

def run(s):
    L, ctx = s.get("L"), s["ctx"]
    if s["kind"] == "diffraction":
        return ctx.diffraction(L["beams"][0], s["geo"], s["theta"], s["phi"], LAM, is_fast_diff=s["fast"])
    if s["kind"] == "main":
        r = ctx.diff_main(L["beams"][0], L["exts"][0], s["geo"], s["theta"], s["phi"], LAM,
                          is_fast_diff=s["fast"], precision=s["prec"])
        if s["prec"] == "fp64":
            return r
        for k, a in zip(s["keep"], r):
            np.copyto(k, a, casting="same_kind")
        return s["keep"]
    if s["kind"] == "finalise":
        mu, m1, p = ctx.finalise(s["grids"][0], s["grids"][1], s["theta"], s["phi"], LAM, s["pin"],
                                 scaling=s["scaling"])
        return mu, m1, np.atleast_1d(p).view(np.float64)
    if s["kind"] == "average":
        mu, m1, pav, per = ctx.diff_batch(L["beams"], L["exts"], L["verts"], s["geo"], s["theta"],
                                          s["phi"], LAM, L["pin"], is_fast_diff=s["fast"],
                                          scaling=s["scaling"], precision=s["prec"], out=s["out"])
        p = np.concatenate([np.atleast_1d(pav), per]).view(np.float64).reshape(-1, _NPAR)
        if s["prec"] == "fp64":
            return mu, m1, p
        for k, a in zip(s["keep"], (mu, m1)):
            np.copyto(k, a, casting="same_kind")
        return s["keep"][0], s["keep"][1], p.astype(np.float32)
    if s["kind"] in ("device", "replay"):
        st, d = torch.cuda.current_stream().cuda_stream, s["d"]
        if s["kind"] == "replay":
            s["graph"].launch(st)
        else:
            diff_batch_dev(ctx, st, *s["args"])
        return d["mu"].float(), d["m1"].float(), d["pav"].float(), d["per"].float()
    # gradient: forward, loss against the target, gradients of vertices and fields
    v, ba, ea = (x.clone().requires_grad_(True) for x in (s["verts"], s["ba"], s["ea"]))
    afb, afe = _ag.far_field(ctx, v, ba, ea, L["beams"][0], L["exts"][0], s["geo"], s["theta"],
                             s["phi"], LAM, is_fast_diff=s["fast"])
    m11, m12 = _ag.mueller11_12(afb, afe, LAM)
    loss = _ag.mueller_loss(m11, m12, s["target"][0], s["target"][1], s["theta"])
    loss.backward()
    return loss.detach().float(), v.grad.float(), ba.grad.float(), ea.grad.float()


# ------------------------------------------------------------------ what a pass cannot do without

def _count(case, seed=0):
    """(triangle records, faces, vertices, orientations), on average over the draws of the lists."""
    n = case.get("norient", 1)
    if case["mesh"] == 0:
        return case["beams"], case["beams"], 3 * case["beams"], 1
    c = case.get("corners", 3)
    tri = 1.0 if c == 3 else (3 + c) / 2 - 2
    faces = 4 * case["mesh"] ** 2
    ext = 0 if case["kind"] == "diffraction" else faces / 2
    return n * (case["beams"] + ext) * tri, faces, (2 * (case["mesh"] + 1) ** 2 if c == 3
                                                    else faces * (3 + c) / 2), n


def work(case):
    """170 operations a triangle and bin (phase, divided difference, polarisation, 2 x 2 complex
    sum), about 2.6 times that with the backward pass; 100 a bin for the Mueller matrix.  The
    field-of-view test leaves the bins within fov of a beam, half of them for external diffraction."""
    nb = case["ntheta"] * case["nphi"]
    if case["kind"] == "finalise":
        return dict(bytes=nb * (128 + 128) + case["ntheta"] * 128, flops=140.0 * nb)
    rec, faces, nverts, n = _count(case)
    share = 0.2 if case.get("fast") else 1.0
    grid = {"diffraction": 64, "main": 128, "gradient": 128}.get(case["kind"], 128)
    return dict(bytes=128.0 * rec + 24.0 * nverts * n + 32.0 * faces + grid * nb,
                flops=(620.0 if case["kind"] == "gradient" else 170.0) * rec * nb * share)


# ------------------------------------------------------------------ the same in 64 bits

_K = 2.0 * PI_REF / LAM


def _two_pi():
    # 2 pi to 50 digits
    return Fraction(628318530717958647692528676655900576839433879875021, 10 ** 50)


def _second_difference(t):
    """The second divided difference of e^{ix} at t[0], t[1], t[2] without cancellation."""
    lo = torch.minimum(torch.minimum(t[0], t[1]), t[2])
    hi = torch.maximum(torch.maximum(t[0], t[1]), t[2])
    mid = t[0] + t[1] + t[2] - lo - hi
    D = hi - lo
    small = D < 2e-3
    h1, h2 = (mid - lo) / 2, (hi - mid) / 2
    q = 1.0 / torch.where(small, torch.ones_like(D), D)
    a = torch.sinc(h2 / math.pi) * torch.exp(1j * (mid + hi) / 2)
    b = torch.sinc(h1 / math.pi) * torch.exp(1j * (lo + mid) / 2)
    m = (t[0] + t[1] + t[2]) / 3
    p2 = sum((x - m) ** 2 for x in t)
    p3 = sum((x - m) ** 3 for x in t)
    near = torch.exp(1j * m) * torch.complex(p2 / 48 - 0.5, p3 / 360)
    return torch.where(small, near, 1j * (a - b) * q)


def _cross(a, b):
    return (a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0])


def _dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


def _sum_facets(V, faces, fan, amp, prop, vk7, cosfov, dirs, theta_row, out_phi, fast):
    """sum over records of area integral x polarisation x amplitude, [2, 2, bins]; `faces` (F, c)
    vertex indices padded with -1, `fan` the record's triangle."""
    there = (faces >= 0).to(V.dtype)[..., None]
    P = V[faces.clamp(min=0)]
    com = (P * there).sum(1) / there.sum(1)
    tri = torch.stack([V[faces.gather(1, (fan + q if q else 0 * fan)[:, None])[:, 0]] for q in range(3)], 1)
    a1, b1 = P[:, 0] - com, P[:, 1] - com
    z = -torch.linalg.cross(a1, b1)
    z = z / z.norm(dim=1, keepdim=True)
    x = prop - (prop * z).sum(1, keepdim=True) * z
    x = x / x.norm(dim=1, keepdim=True)
    y = torch.linalg.cross(z, x)
    par = torch.linalg.cross(vk7, prop)
    par = (par * z).sum(1) / par.norm(dim=1)
    sign = torch.where(par > float(np.float32(1e-4)), -1.0, 1.0)
    col = [c[:, None] for c in com.unbind(1)]
    row = [d[None] for d in dirs]

    def seen(u):
        w = [FAR * u[i] - col[i] for i in range(3)]
        r = torch.sqrt(_dot(w, w))
        return [wi / r for wi in w], r

    kl, r = seen(row)
    uc = _dot(row, col)
    way = _K * (_dot(col, col) - 2 * FAR * uc) / (r + FAR)
    ax = [[v[:, i:i + 1] for i in range(3)] for v in (x, y, z)]
    k = [_dot(a, kl) for a in ax]
    Kx, Kz = (prop * x).sum(1, keepdim=True), (prop * z).sum(1, keepdim=True)
    rel = tri - com[:, None]
    t = []
    for q in range(3):
        vx, vy = (rel[:, q] * x).sum(1, keepdim=True), (rel[:, q] * y).sum(1, keepdim=True)
        t.append(way + _K * ((Kx - k[0]) * vx - k[1] * vy))
    area = 0.5 * (torch.linalg.cross(tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]) * z).sum(1)
    g = _second_difference(t) * (2j * area * sign / LAM)[:, None]
    ky = k[1].clamp(-C_KY, C_KY)
    sq = torch.sqrt(1 - ky * ky)
    m = (-k[0] * ky / sq, sq, -ky * k[2] / sq)
    d = 0.5 * (-Kz * sq - k[2] / sq)
    e = 0.5 * (-k[0] * ky / sq)
    inc = [-a[2] for a in ax]
    kc = (k[0], ky, k[2])
    other, _ = seen([o[None] for o in theta_row])
    bend = [_dot(a, other) for a in ax]
    fwd = _dot(inc, kc).abs() >= C_FWD
    h = _cross(inc, [torch.where(fwd, o, c) for o, c in zip(bend, kc)])
    hn = torch.sqrt(_dot(h, h))
    ev = _cross(kc, m)
    en = torch.sqrt(_dot(ev, ev))
    p, rr = _dot(h, m) / hn, _dot(h, ev) / (hn * en)
    A, B = p * d + rr * e, p * e - rr * d
    if fast:
        g = torch.where(_dot([prop[:, i:i + 1] for i in range(3)], kl) < cosfov[:, None],
                        torch.zeros_like(g), g)
    gA, gB = (g * A).transpose(0, 1), (g * B).transpose(0, 1)
    top = gA @ amp[:, 0] + gB @ amp[:, 1]
    low = gA @ amp[:, 1] - gB @ amp[:, 0]
    s, c = out_phi
    S = torch.stack([top, low], 0)          # (a, bins, b)
    T0 = -S[..., 0] * s + S[..., 1] * c
    T1 = -S[..., 0] * c - S[..., 1] * s
    return torch.stack([T0, T1], 1)          # (a, b, bins)


def _tensors(L, obs, ext, dev):
    """Per record of a list: padded faces, fan position and the outbeam it belongs to."""
    off, vi = L["off"], L["vi"]
    nv = (off[1:] - off[:-1])[obs["fi"] - 1]
    who = np.repeat(np.arange(len(obs)), nv - 2)
    fan = np.concatenate([np.arange(n - 2) for n in nv]) if len(nv) and nv.max() > 3 else np.zeros(len(who), int)
    width = int(nv.max()) if len(nv) else 3
    pos = off[obs["fi"] - 1][:, None] + np.arange(width)
    faces = np.where(np.arange(width) < nv[:, None], vi[np.minimum(pos, len(vi) - 1)] - 1, -1)
    fov = np.full(len(obs), PI_REF / 2) if ext else obs["fov"]
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    return dict(faces=to(faces[who]), fan=to(fan), who=to(who), prop=to(obs["prop_out"][who]),
                vk7=to(obs["vk7"][who]), cosfov=to(np.cos(fov)[who]))


def _dirs(case, dev):
    theta, phi = _angles(case)
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    st, ct = np.sin(theta)[:, None], np.cos(theta)[:, None]
    cp, sp = np.cos(phi)[None], np.sin(phi)[None]
    grid = [to((w * np.ones((len(theta), len(phi)))).ravel()) for w in (st * cp, st * sp, -ct)]
    i = int(np.argmax(theta > PI_REF / 180))
    same = [to((w * np.ones((len(theta), len(phi)))).ravel())
            for w in (st[i] * cp, st[i] * sp, -ct[i])]
    turn = tuple(to((w * np.ones((len(theta), 1))).ravel()) for w in (sp, cp))
    return grid, same, turn


def _amp(a):
    """(n, 8) re/im of (1,1),(2,1),(1,2),(2,2) to (n, 2, 2) complex."""
    z = torch.complex(a[:, 0::2], a[:, 1::2])
    return torch.stack([torch.stack([z[:, 0], z[:, 2]], 1), torch.stack([z[:, 1], z[:, 3]], 1)], 1)


def _chunks(n, nb, size):
    step = max(1, int(size // nb))
    return [slice(i, min(n, i + step)) for i in range(0, n, step)]


def _orientation(case, L, o, grid, dev, obs_of=("beams", "exts")):
    V = torch.from_numpy(np.ascontiguousarray(L["verts"][o])).to(dev)
    out = []
    for name in obs_of:
        obs = L[name][o]
        S = torch.zeros((2, 2, len(grid[0][0])), dtype=torch.complex128, device=dev)
        if len(obs):
            R = _tensors(L, obs, name == "exts", dev)
            amp = _amp(torch.from_numpy(np.ascontiguousarray(obs["ampl"])).to(dev))
            for c in _chunks(len(R["who"]), S.shape[-1], 1.2e7):
                S += _sum_facets(V, R["faces"][c], R["fan"][c], amp[R["who"][c]], R["prop"][c],
                                 R["vk7"][c], R["cosfov"][c], grid[0], grid[1], grid[2],
                                 case.get("fast", False))
        out.append(S)
    return out


def _far_phase():
    turns = Fraction(_K) * Fraction(FAR)
    return float(turns - (turns // _two_pi()) * _two_pi())


def _layout(S, case):
    """(2, 2, bins) to the grids' (nphi, ntheta, 2, 2)."""
    return S.reshape(2, 2, case["ntheta"], case["nphi"]).permute(3, 2, 0, 1)


def _simpson(x):
    """Weights of the piecewise quadratic rule on any spacing: pairs of intervals, and for an even
    number of points the last interval from the last three points."""
    n, w = len(x), np.zeros(len(x), dtype=np.longdouble)

    def panel(i, lo, hi):
        p = x[i:i + 3].astype(np.longdouble)
        mid = p[1]
        a, b, u = lo - mid, hi - mid, p - mid
        m0, m1, m2 = b - a, (b * b - a * a) / 2, (b ** 3 - a ** 3) / 3
        for q in range(3):
            r, s = u[(q + 1) % 3], u[(q + 2) % 3]
            w[i + q] += (m2 - (r + s) * m1 + r * s * m0) / ((u[q] - r) * (u[q] - s))

    for i in range(0, n - 2, 2):
        panel(i, x[i].astype(np.longdouble), x[i + 2].astype(np.longdouble))
    if n % 2 == 0:
        panel(n - 3, x[n - 2].astype(np.longdouble), x[n - 1].astype(np.longdouble))
    return w.astype(np.float64)


def _mueller(a):
    """The 16 Mueller elements of (nphi, ntheta, 2, 2) amplitudes."""
    s11, s12, s21, s22 = a[..., 0, 0], a[..., 0, 1], a[..., 1, 0], a[..., 1, 1]
    p11, p12, p21, p22 = (s.abs() ** 2 for s in (s11, s12, s21, s22))
    re = lambda u, v: (u * v.conj()).real  # noqa: E731
    im = lambda u, v: (u * v.conj()).imag  # noqa: E731
    return torch.stack([
        (p11 + p12 + p21 + p22) / 2, (p11 - p12 + p21 - p22) / 2, re(s11, s12) + re(s22, s21),
        im(s11, s12) - im(s22, s21), (p11 + p12 - p21 - p22) / 2, (p11 - p12 - p21 + p22) / 2,
        re(s11, s12) - re(s22, s21), im(s11, s12) + im(s22, s21), re(s11, s21) + re(s22, s12),
        re(s11, s21) - re(s22, s12), re(s11, s22) + re(s12, s21), im(s11, s22) + im(s21, s12),
        im(s21, s11) + im(s22, s12), im(s21, s11) - im(s22, s12), im(s22, s11) - im(s12, s21),
        re(s22, s11) - re(s12, s21)], -1)


def _finalise(case, gb, ge, pin, scaling):
    """(mueller, mueller_1d, the 18 parameters) of one orientation's grids (cuda tensors)."""
    theta, phi = _angles(case)
    dev = gb.device
    wp, wt = (torch.from_numpy(_simpson(x)).to(dev) for x in (phi, theta))
    st, ct = torch.from_numpy(np.sin(theta)).to(dev), torch.from_numpy(np.cos(theta)).to(dev)
    gb, ge = gb * _K, ge * _K

    def total(a):
        m = (a.abs() ** 2).sum((-1, -2)) / 2
        row = torch.einsum("i,ij->j", wp, m) * st / _K ** 2
        return float((row * wt).sum()), float((row * ct * wt).sum())

    if scaling:
        gb = gb / math.sqrt(total(gb)[0] / float(pin["beam_energy_out"]))
        ge = ge / math.sqrt(total(ge)[0] / float(pin["ext_energy_out"]))
    mu = _mueller(gb + ge)
    m1 = torch.einsum("i,ije->je", wp, mu)
    (sc, sg), (sb, bg), (se, eg) = total(gb + ge), total(gb), total(ge)
    g, ab = float(pin["geo_cross_sec"]), float(pin["abs"])
    back = float(mu[0, int(np.argmin(np.abs(theta - 2 * PI_REF))), 0]) * 4 * PI_REF / _K ** 2
    par = [ab, sc, ab + sc, sc / (ab + sc), sg / sc, ab / g, sc / g, (ab + sc) / g, g, back,
           float(pin["beam_energy_out"]), float(pin["ext_energy_out"]), sb, se, bg / sb, eg / se,
           sb / g, se / g]
    return mu, m1, np.array(par)


def exact(case, seed):
    dev = "cuda"
    if case["kind"] == "finalise":
        a, b = (torch.from_numpy(np.ascontiguousarray(g)).to(dev) for g in _grids(case, seed))
        mu, m1, p = _finalise(case, a, b, _params([300.0])[0], case["scaling"])
        return mu.cpu().numpy(), m1.cpu().numpy(), p
    rec, _, _, n = _count(case)
    nb = case["ntheta"] * case["nphi"]
    if rec * nb > (7e8 if case["kind"] == "gradient" else 1.2e10):
        return None
    L, grid = _lists(case, seed), _dirs(case, dev)
    if case["kind"] in ("diffraction", "main"):
        turn = complex(math.cos(_far_phase()), math.sin(_far_phase()))
        got = [(_layout(S, case) * turn).cpu().numpy()
               for S in _orientation(case, L, 0, grid, dev,
                                     ("beams",) if case["kind"] == "diffraction" else ("beams", "exts"))]
        return got[0] if case["kind"] == "diffraction" else got
    if case["kind"] == "gradient":
        return _exact_gradient(case, seed, L, grid, dev)
    mu, m1, per = 0.0, 0.0, []
    for o in range(n):
        gb, ge = (_layout(S, case) for S in _orientation(case, L, o, grid, dev))
        if not len(L["exts"][o]):
            return None    # ratios of the empty part have no value
        u, v, p = _finalise(case, gb, ge, L["pin"][o], case.get("scaling", False))
        mu, m1 = mu + u / n, m1 + v / n
        per.append(p)
    per = np.array(per)
    avg = per.mean(0)
    avg[10:12] = 0.0        # the two energies are not averaged
    if case["kind"] == "average":
        return mu.cpu().numpy(), m1.cpu().numpy(), np.concatenate([avg[None], per])
    return mu.permute(2, 1, 0).contiguous(), m1.transpose(0, 1).contiguous(), avg, per


def _exact_gradient(case, seed, L, grid, dev):
    rng = np.random.default_rng([seed, 79])
    t11, t12 = (t.to(dev) for t in _target(case, rng))
    theta = torch.from_numpy(_angles(case)[0]).to(dev)
    turn = complex(math.cos(_far_phase()), math.sin(_far_phase()))
    S = [s.clone() for s in _orientation(case, L, 0, grid, dev)]
    total = (S[0] + S[1]).requires_grad_(True)
    p = ((_layout(total * turn, case) * _K).abs() ** 2)
    m11 = 0.5 * (p[..., 0, 0] + p[..., 0, 1] + p[..., 1, 0] + p[..., 1, 1])
    m12 = 0.5 * (p[..., 0, 0] - p[..., 0, 1] + p[..., 1, 0] - p[..., 1, 1])
    w = torch.sin(theta)[None].expand_as(m11)
    loss = (w / w.sum() * ((torch.log(m11) - torch.log(t11)) ** 2
                           + (-m12 / m11 + t12 / t11) ** 2)).sum()
    loss.backward()
    V = torch.from_numpy(np.ascontiguousarray(L["verts"][0])).to(dev).requires_grad_(True)
    grads = []
    for name in ("beams", "exts"):
        obs = L[name][0]
        a = torch.from_numpy(np.ascontiguousarray(obs["ampl"])).to(dev).requires_grad_(True)
        R = _tensors(L, obs, name == "exts", dev)
        for c in _chunks(len(R["who"]), S[0].shape[-1], 3e6):
            part = _sum_facets(V, R["faces"][c], R["fan"][c], _amp(a)[R["who"][c]], R["prop"][c],
                               R["vk7"][c], R["cosfov"][c], grid[0], grid[1], grid[2], False)
            part.backward(total.grad)
        grads.append(a.grad)
    return loss.detach(), V.grad, grads[0], grads[1]
