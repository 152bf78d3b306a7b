"""Performance cases: the calls that programs make of bpm_gb300, over the range of sizes, modes
and data types in use.

Each case is a dict of plain values whose "kind" names the public entry point:
  march    bpm_3d, one field through one volume
  batch    bpm_3d_batched, many illuminations through one shared volume
  adjoint  propagate_exit with its backward pass, one step of a reconstruction
  psf      psf, the vectorial focus field on a volume
  plane    focus_field_debye_plane, one plane of the focus field
  points   focus_field_debye_at, the focus field at free points
`exact` restates each in 64-bit torch and numpy (the evanescent cut, the grid coordinates and
the end weights of the quadrature keep their defined float32 recipes, which decide which terms
enter the result).
"""
import math

import numpy as np
import torch

import bpm_gb300
from bpm_gb300.adjoint import propagate_exit

LAM, N0, UNITS = .5, 1.33, (.1, .1, .1)
KINDS = ("march", "batch", "adjoint", "psf", "plane", "points")


# ----------------------------------------------------------------------------------------
# cases
# ----------------------------------------------------------------------------------------

def march(nx, ny, nz, mode="weighted", dn="f32", out="intensity", absorb=0, scatter=False, **kw):
    """mode: mean_mode; dn: "f32", "f16" (store_dn_as_half) or "c64"; out: "field",
    "intensity" (volumes) or "last" (the exit plane alone); scatter: return_scattering and
    return_g."""
    return dict(kind="march", nx=nx, ny=ny, nz=nz, mode=mode, dn=dn, out=out, absorb=absorb, scatter=scatter, **kw)


def batch(fields, nx, ny, nz, mode="weighted", out="intensity", **kw):
    return dict(kind="batch", fields=fields, nx=nx, ny=ny, nz=nz, mode=mode, dn="f32", out=out, **kw)


def adjoint(fields, nx, ny, nz, ckpt, **kw):
    return dict(kind="adjoint", fields=fields, nx=nx, ny=ny, nz=nz, ckpt=ckpt, **kw)


def psf(nx, ny, nz, steps, na_in=0., na_out=1.1, field=False, **kw):
    return dict(kind="psf", nx=nx, ny=ny, nz=nz, steps=steps, na_in=na_in, na_out=na_out, field=field, **kw)


def listed():
    return [
        # the smallest march in use: a quick look through a small phantom, default options,
        # the complex field volume back
        march(64, 64, 64, out="field", name="march_64"),
        # an ordinary single march: the 128^3 sphere phantom, default weighted mode
        march(128, 128, 128, name="march_128"),
        # an absorbing sample (complex index) under a focused beam
        march(256, 256, 256, mode="ignore", dn="c64", name="march_256_absorbing"),
        # a long rectangular sample stored as half, absorbing border, scattering analysis
        march(512, 256, 100, dn="f16", out="field", absorb=16, scatter=True, name="march_512x256_scatter"),
        # the largest single field: a whole camera frame
        march(1024, 1024, 128, name="march_1024"),
        # a few illuminations of a small sample whose exit planes alone matter
        batch(12, 128, 128, 96, mode="simple", out="last", name="batch_128_exit"),
        # many illumination angles through one large sample, intensity volumes
        batch(32, 512, 512, 128, name="batch_512"),
        # one step of a tomographic reconstruction: forward march, loss, gradient
        adjoint(16, 256, 256, 128, 16, name="adjoint_256"),
        # the focus of a water-dipping objective on a large volume, finely integrated
        psf(256, 256, 256, 512, name="psf_256"),
        # a small annular (Bessel-like) focus with its vector components, default steps
        psf(64, 64, 48, 200, na_in=.4, na_out=.8, field=True, name="psf_64_annulus"),
        # one plane of a focus, as an input field or a quick view
        dict(kind="plane", nx=128, ny=128, steps=200, z=1., na=.6, name="plane_128"),
        # the focus field at the positions of a few thousand emitters
        dict(kind="points", n=4000, steps=200, na=.8, name="points_4000"),
    ]


def draw(rng):
    """One more case of the ranges above (rng: random.Random)."""
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def pow2(lo, hi):
        return 1 << rng.randint(lo, hi)

    kind = rng.choice(KINDS)
    if kind == "march":
        mode = rng.choice(["weighted", "weighted", "simple", "ignore"])
        dn = rng.choice(["f32", "f32", "f16"] + (["c64"] if mode == "ignore" else []))
        return march(pow2(5, 10), pow2(5, 10), log(16, 128), mode=mode, dn=dn,
                     out=rng.choice(["field", "intensity", "intensity", "last"]),
                     absorb=rng.choice([0, 0, 10, 16]), scatter=rng.random() < .25)
    if kind == "batch":
        return batch(log(2, 32), pow2(6, 9), pow2(6, 9), log(16, 128), mode=rng.choice(["weighted", "simple", "ignore"]),
                     out=rng.choice(["field", "intensity", "intensity", "last"]))
    if kind == "adjoint":
        return adjoint(log(1, 16), pow2(6, 8), pow2(6, 8), log(17, 128), rng.choice([8, 16, 32]))
    if kind == "psf":
        na = round(rng.uniform(.3, 1.2), 2)
        return psf(2 * log(16, 128), 2 * log(16, 128), 2 * log(16, 128), log(100, 512),
                   na_in=round(na * rng.choice([0., 0., .5]), 2), na_out=na, field=rng.random() < .5)
    if kind == "plane":
        return dict(kind="plane", nx=log(48, 512), ny=log(48, 512), steps=log(100, 400),
                    z=round(rng.uniform(-5., 5.), 2), na=round(rng.uniform(.2, .9), 2))
    return dict(kind="points", n=log(100, 50000), steps=log(100, 400), na=round(rng.uniform(.2, .9), 2))


# ----------------------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------------------

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _volume(nx, ny, nz, g, corr=4., sigma=.02, clip=.06):
    """A smooth random index volume: Gaussian-filtered white noise, clipped."""
    w = torch.randn((nz, ny, nx), device="cuda", generator=g)
    k = 1.
    for d, n in enumerate((nz, ny, nx)):
        f = torch.fft.fftfreq(n, device="cuda").reshape([-1 if i == d else 1 for i in range(3)])
        k = k * torch.exp(-2. * math.pi ** 2 * corr ** 2 * f ** 2)
    f = torch.fft.ifftn(torch.fft.fftn(w) * k).real
    return (f * (sigma / f.std())).clamp_(-clip, clip).float().contiguous()


def _axis(n, d):
    return (torch.arange(n, device="cuda", dtype=torch.float64) - n // 2) * d


def _tilts(fields, nx, ny, g, na=.8):
    """Plane waves with tilts area-uniform inside the aperture, (fields, ny, nx) complex64."""
    r = na * torch.rand(fields, device="cuda", generator=g, dtype=torch.float64).sqrt()
    th = 2. * math.pi * torch.rand(fields, device="cuda", generator=g, dtype=torch.float64)
    k0 = 2. * math.pi / LAM
    ph = (k0 * r * torch.cos(th))[:, None, None] * _axis(nx, UNITS[0])[None, None, :] \
        + (k0 * r * torch.sin(th))[:, None, None] * _axis(ny, UNITS[1])[None, :, None]
    return torch.exp(-1j * ph).to(torch.complex64).contiguous()


def _focused(nx, ny, g):
    """A converging Gaussian beam, slightly off axis, (ny, nx) complex64."""
    c = torch.rand(2, device="cuda", generator=g, dtype=torch.float64) - .5
    r2 = (_axis(nx, UNITS[0])[None, :] - c[0]) ** 2 + (_axis(ny, UNITS[1])[:, None] - c[1]) ** 2
    w, f = .2 * min(nx, ny) * UNITS[0], 10.
    k = 2. * math.pi * N0 / LAM
    return (torch.exp(-r2 / w ** 2) * torch.exp(1j * k * r2 / (2. * f))).to(torch.complex64).contiguous()


def prepare(case, seed):
    g = _generator(seed)
    s = dict(case)
    kind = case["kind"]
    if kind in ("march", "batch", "adjoint"):
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        s["size"] = (nx, ny, nz)
        vol = _volume(nx, ny, nz, g)
        if kind == "march":
            if case["dn"] == "c64":
                vol = torch.complex(vol, -5e-4 * torch.rand(vol.shape, device="cuda", generator=g))
            s["vol"], s["u0"] = vol, _focused(nx, ny, g)
        elif kind == "batch":
            s["vol"], s["u0"] = vol, _tilts(case["fields"], nx, ny, g)
        else:
            s["vol"] = vol.requires_grad_(True)
            s["u0"] = _tilts(case["fields"], nx, ny, g, na=.6)
            s["target"] = .8 + .4 * torch.rand((case["fields"], ny, nx), device="cuda", generator=g)
    elif kind in ("psf", "plane"):
        # the optics vary with the seed a little, as a wavelength scan does
        s["lam"] = .5 + .04 * float(torch.rand(1, device="cuda", generator=g))
    else:
        r = torch.rand((3, case["n"]), device="cuda", generator=g) - .5
        s["x"], s["y"], s["z"] = (20. * r[0]).contiguous(), (20. * r[1]).contiguous(), (10. * r[2]).contiguous()
    return s


# ----------------------------------------------------------------------------------------
# one pass
# ----------------------------------------------------------------------------------------

def run(s):
    kind = s["kind"]
    if kind == "march":
        return bpm_gb300.bpm_3d(s["size"], UNITS, lam=LAM, u0=s["u0"], dn=s["vol"], n0=N0,
                                return_scattering=s["scatter"], return_g=s["scatter"],
                                return_full=s["out"] != "last", return_field=s["out"] != "intensity",
                                absorbing_width=s["absorb"], store_dn_as_half=s["dn"] == "f16", mean_mode=s["mode"])
    if kind == "batch":
        return bpm_gb300.bpm_3d_batched(s["size"], UNITS, lam=LAM, u0=s["u0"], dn=s["vol"], n0=N0,
                                        return_full=s["out"] != "last", return_field=s["out"] != "intensity",
                                        mean_mode=s["mode"])
    if kind == "adjoint":
        exit_planes = propagate_exit(s["vol"], s["u0"], s["size"], UNITS, LAM, N0, ckpt_every=s["ckpt"])
        loss = ((exit_planes.abs() ** 2 - s["target"]) ** 2).sum()
        grad, = torch.autograd.grad(loss, s["vol"])
        return exit_planes.detach(), grad
    if kind == "psf":
        na = [s["na_in"], s["na_out"]] if s["na_in"] else s["na_out"]
        return bpm_gb300.psf((s["nx"], s["ny"], s["nz"]), UNITS, s["lam"], na, N0, s["steps"],
                             return_field=s["field"], device=True)
    if kind == "plane":
        return bpm_gb300.focus_field_debye_plane((s["nx"], s["ny"]), UNITS[:2], s["z"], s["lam"], s["na"],
                                                 n_integration_steps=s["steps"], device=True)
    return bpm_gb300.focus_field_debye_at(s["x"], s["y"], s["z"], LAM, s["na"], N0, s["steps"], device=True)


# ----------------------------------------------------------------------------------------
# what a pass cannot do without
# ----------------------------------------------------------------------------------------

def work(case):
    kind = case["kind"]
    nx, ny, nz = case.get("nx", 1), case.get("ny", 1), case.get("nz", 1)
    if kind in ("march", "batch", "adjoint"):
        plane, fields = nx * ny, case.get("fields", 1)
        # a step: two 2-D transforms (5 N log2 N each) and about 20 pointwise operations
        step = plane * (10. * math.log2(plane) + 20.)
        if kind == "adjoint":
            return {"bytes": 8. * plane * nz + fields * plane * 20., "flops": 2. * fields * (nz - 1) * step}
        dn = {"f32": 4., "f16": 4., "c64": 8.}[case["dn"]]
        vol = {"field": 8. * nz, "intensity": 4. * nz, "last": 8.}[case["out"]]
        return {"bytes": dn * plane * nz + fields * plane * (vol + 8.), "flops": fields * (nz - 1) * step}
    nodes = case["steps"] + 1
    if kind == "psf":
        octant = (nx // 2 + 1) * (ny // 2 + 1) * (nz // 2 + 1)
        return {"bytes": (28. if case["field"] else 4.) * nx * ny * nz, "flops": 12. * octant * nodes}
    # without a grid along z every point has its own Bessel functions per node (about 40
    # operations) and three complex sums
    n = nx * ny if kind == "plane" else case["n"]
    return {"bytes": (8. if kind == "plane" else 40.) * n, "flops": 55. * n * nodes}


# ----------------------------------------------------------------------------------------
# the same in 64 bits
# ----------------------------------------------------------------------------------------

def _freq32(n, d):
    """The float32 frequency recipe of the evanescent cut: i / n / d."""
    i = np.arange(n)
    i = np.where(i < (n - 1) // 2 + 1, i, i - n).astype(np.float32)
    return (i / np.float32(n)) / np.float32(d)


class _Grid:
    """Squared wave numbers on (ny, nx): in 64 bits for the phase, in float32 for the cut."""

    def __init__(self, nx, ny):
        self.k0 = 2. * math.pi / LAM
        kx = 2. * math.pi * torch.fft.fftfreq(nx, UNITS[0], dtype=torch.float64, device="cuda")
        ky = 2. * math.pi * torch.fft.fftfreq(ny, UNITS[1], dtype=torch.float64, device="cuda")
        self.k2 = kx[None, :] ** 2 + ky[:, None] ** 2
        two_pi = np.float32(2.) * np.float32(math.pi)
        kx32, ky32 = two_pi * _freq32(nx, UNITS[0]), two_pi * _freq32(ny, UNITS[1])
        self.kx2 = torch.from_numpy(kx32 * kx32).cuda()[None, :]
        self.ky2 = torch.from_numpy(ky32 * ky32).cuda()[:, None]

    def propagator(self, n):
        """exp(-i kz dz) at the mean index n (a 64-bit tensor of any shape), 0 where evanescent."""
        n = n[..., None, None]
        n32, k32 = n.float(), torch.tensor(self.k0, dtype=torch.float32, device="cuda")
        cut = (((n32 * n32) * k32) * k32 - self.kx2) - self.ky2 >= 0
        kz = (n * n * self.k0 ** 2 - self.k2).clamp(min=0.).sqrt()
        return torch.where(cut, torch.exp(-1j * UNITS[2] * kz), 0.)


def _taper(nx, ny, width):
    x, y = torch.arange(nx, device="cuda"), torch.arange(ny, device="cuda")
    dist = torch.minimum(torch.minimum(x, nx - 1 - x)[None, :], torch.minimum(y, ny - 1 - y)[:, None]).double()
    return torch.where(dist < width, .5 * (1. - torch.cos(math.pi * dist / max(width, 1))), 1.)


def _march64(u0, vol, mode, absorb=0, scatter=False, plane_out=None):
    """The march in 64 bits over a batch u0 (B, ny, nx): plane_out(z, u) for every plane;
    returns the exit planes and the scattering sums."""
    ny, nx = u0.shape[-2:]
    nz = vol.shape[0]
    grid = _Grid(nx, ny)
    k0, dz = grid.k0, UNITS[2]
    n0 = torch.tensor(N0, dtype=torch.float64, device="cuda")
    fixed = grid.propagator(n0) if mode == "ignore" else None
    taper = _taper(nx, ny, absorb) if absorb else None
    p, g = torch.zeros(nz, dtype=torch.float64), torch.zeros(nz, dtype=torch.float64)
    weight = (n0 ** 2 * k0 ** 2 - grid.k2).clamp(min=0.).sqrt() / n0 / k0 if scatter else None
    u = u0.to(torch.complex128)
    if plane_out:
        plane_out(0, u)
    for z in range(1, nz):
        f = torch.fft.fft2(u)
        dn0 = torch.zeros(u.shape[0], dtype=torch.float64, device="cuda")
        if mode == "weighted":
            a = f.abs()
            dn0 = (a * vol[0].real.double()).sum((-2, -1)) / a.sum((-2, -1))
        elif mode == "simple":
            dn0 = dn0 + vol[z].double().mean()
        f = f * (fixed if mode == "ignore" else grid.propagator(n0 + dn0))
        if scatter:
            d = f[0].clone()
            d[0, 0] -= nx * ny * complex(np.exp(-1j * k0 * N0 * z * dz))
            e = d.abs() ** 2
            p[z], g[z] = (weight * e).sum(), (weight ** 2 * e).sum()
        slab = vol[z].to(torch.complex128)
        u = torch.fft.ifft2(f) * torch.exp(-1j * k0 * dz * (slab - dn0[:, None, None]))
        if taper is not None and not vol.is_complex():
            u = u * taper
        if plane_out:
            plane_out(z, u)
    return u, p * (UNITS[0] * UNITS[1] / nx / ny), g / p


def _exact_march(case, s):
    vol, u0 = s["vol"], s["u0"]
    if case["dn"] == "f16":
        vol = vol.half()
    single = case["kind"] == "march"
    u0 = u0[None] if single else u0
    nz, ny, nx = vol.shape
    keep = None
    if case["out"] != "last":
        field = case["out"] == "field"
        keep = torch.empty((u0.shape[0], nz, ny, nx), dtype=torch.complex128 if field else torch.float64, device="cuda")

        def plane_out(z, u):
            keep[:, z] = u if field else u.real ** 2 + u.imag ** 2
    u, p, g = _march64(u0, vol, case["mode"], case.get("absorb", 0), case.get("scatter", False),
                       plane_out if keep is not None else None)
    res = u if keep is None else keep
    res = res[0] if single else res
    return (res, p, g) if case.get("scatter") else res


def _exact_adjoint(case, s):
    vol = s["vol"].detach().double().requires_grad_(True)
    grid = _Grid(case["nx"], case["ny"])
    h = grid.propagator(torch.tensor(N0, dtype=torch.float64, device="cuda"))
    masks = torch.exp(-1j * grid.k0 * UNITS[2] * vol)
    u = s["u0"].to(torch.complex128)
    for z in range(1, case["nz"]):
        u = torch.fft.ifft2(torch.fft.fft2(u) * h) * masks[z]
    loss = ((u.abs() ** 2 - s["target"].double()) ** 2).sum()
    grad, = torch.autograd.grad(loss, vol)
    return u.detach(), grad


def _coords(n, x2, x1=0.):
    """The float32 grid recipe x1 + i (x2 - x1) / (n - 1)."""
    i = np.arange(n, dtype=np.float32)
    x1, x2 = np.float32(x1), np.float32(x2)
    return torch.from_numpy((x1 + (i * (x2 - x1)) / np.float32(n - 1.)).astype(np.float64)).cuda()


def _nodes(na, n0, steps, ends32):
    """Angles and trapezoid weights: steps + 1 nodes an annulus, half weights at the first and
    the last, or (ends32) where the float32 angle meets a limit."""
    t, w = [], []
    al = np.arcsin(np.array([0., na] if np.isscalar(na) else na) / n0).astype(np.float32)
    for a1, a2 in zip(al[0::2], al[1::2]):
        i = np.arange(steps + 1)
        dt = (float(a2) - float(a1)) / (steps - 1.)
        if ends32:
            t32 = a1 + i.astype(np.float32) * ((a2 - a1) / np.float32(steps - 1.))
            end = (t32 == a1) | (t32 == a2)
        else:
            end = (i == 0) | (i == steps)
        t.append(float(a1) + i * dt)
        w.append(np.where(end, .5, 1.) * dt)
    return torch.from_numpy(np.concatenate(t)).cuda(), torch.from_numpy(np.concatenate(w)).cuda()


def _bessel(kr, t, w):
    """w (cos t + 1) J0, w sin t J1, w (cos t - 1) J2 at kr sin t, (len(kr), len(t)) each."""
    x = kr[:, None] * t.sin()[None, :]
    j0, j1 = torch.special.bessel_j0(x), torch.special.bessel_j1(x)
    j2 = torch.where(x.abs() < 1e-3, x * x / 8., 2. * j1 / x.clamp(min=1e-3) - j0)
    return (w * (t.cos() + 1.)) * j0, (w * t.sin()) * j1, (w * (t.cos() - 1.)) * j2


def _vectors(i0, i1, i2, phi):
    ex = i0 + i2 * torch.cos(2. * phi)
    return ex, torch.sin(2. * phi) * i2, -2j * i1 * torch.cos(phi)


def _exact_psf(case, s):
    half = [case[k] // 2 + 1 for k in ("nx", "ny", "nz")]
    x, y, z = (_coords(n, d * (n - 1.)) for n, d in zip(half, UNITS))
    k = 2. * math.pi / float(np.float32(s["lam"] / N0))
    t, w = _nodes([case["na_in"], case["na_out"]], N0, case["steps"], False)
    yy, xx = torch.meshgrid(y, x, indexing="ij")
    a = _bessel(k * (xx ** 2 + yy ** 2).sqrt().ravel(), t, w * t.cos().sqrt())
    e = torch.exp(1j * k * z[None, :] * t.cos()[:, None])
    i0, i1, i2 = (m.to(torch.complex128) @ e for m in a)
    ex, ey, ez = _vectors(i0, i1, i2, torch.atan2(yy, xx).ravel()[:, None])
    u = ex.abs() ** 2 + ey.abs() ** 2 + ez.abs() ** 2
    iz, iy, ix = (torch.from_numpy(np.abs(np.arange(case[n]) - case[n] // 2)).cuda() for n in ("nz", "ny", "nx"))
    front = (torch.arange(case["nz"], device="cuda") <= case["nz"] // 2)[:, None, None]

    def full(v):
        v = v.T.reshape(half[2], half[1], half[0])
        return v.index_select(0, iz).index_select(1, iy).index_select(2, ix)
    if not case["field"]:
        return full(u)
    return (full(u),) + tuple(torch.where(front, v.conj(), v) for v in (full(ex), full(ey), full(ez)))


def _exact_points(xs, ys, zs, lam, n0, na, steps):
    k = 2. * math.pi / float(np.float32(lam / n0))
    t, w = _nodes(na, n0, steps, True)
    a = _bessel(k * (xs ** 2 + ys ** 2).sqrt(), t, w * t.cos().sqrt() * t.sin())
    e = torch.exp(1j * k * zs[:, None] * t.cos()[None, :])
    return _vectors(*((m * e).sum(1) for m in a), torch.atan2(ys, xs))


def exact(case, seed):
    s = prepare(case, seed)
    kind = case["kind"]
    if kind in ("march", "batch"):
        return _exact_march(case, s)
    if kind == "adjoint":
        return _exact_adjoint(case, s)
    if kind == "psf":
        return _exact_psf(case, s)
    if kind == "plane":
        nx, ny = case["nx"], case["ny"]
        x = _coords(nx, (nx - nx // 2) * UNITS[0], -(nx // 2) * UNITS[0])
        y = _coords(ny, (ny - ny // 2) * UNITS[1], -(ny // 2) * UNITS[1])
        yy, xx = torch.meshgrid(y, x, indexing="ij")
        z = torch.full_like(xx, float(np.float32(case["z"])))
        ex = _exact_points(xx.ravel(), yy.ravel(), z.ravel(), s["lam"], 1., case["na"], case["steps"])[0]
        return ex.reshape(ny, nx)
    ex, ey, ez = _exact_points(s["x"].double(), s["y"].double(), s["z"].double(), LAM, N0, case["na"], case["steps"])
    return ex.abs() ** 2, ex, ey, ez
