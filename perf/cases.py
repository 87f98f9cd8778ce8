"""The performance cases of kerrsplat_b200: what a user's program has the library do, and its exact values.

A case is one call (or one short sequence of calls) through the public Python API on a seeded scene:

    thin     `thin_image` of 14-row splats on a regenerated cache (FP64, the default precision)
    refit    `regenerate` at a new spin and inclination, then the thin image (a geometry fit's step)
    render   `render` of thermal splats, every frequency in one call
    movie    `render` of knot, power-law and kappa splats, uneven sample counts, several frames
    grad     `chi2_gradient` against image data (an image fit's step)
    vis      `vis_chi2_gradient` against visibilities (an interferometric fit's step)
    jvp      `jvp` along given directions (a Gauss-Newton step's forward product)

`exact` gives the same outputs in 64-bit torch: the Kerr geodesics in closed form with Gauss-Legendre
quadrature of the time and azimuth, the synchrotron fits, the Stokes steps by the matrix exponential, and
derivatives by torch's own differentiation.
"""
import math

import numpy as np
import torch

import kerrsplat_b200 as ks

NUS = (230e9, 86e9, 345e9, 690e9)
L_SGRA = 6.6742e-8 * 4.0e6 * 1.989e33 / 2.99792458e10 ** 2   # GM/c^2 of 4e6 solar masses, cm
L_M87 = 6.6742e-8 * 6.5e9 * 1.989e33 / 2.99792458e10 ** 2
DIST_M87 = 16.8e6 * 3.0857e18


def _case(op, res, samples, splats, freqs=1, frames=1, precision="mixed", spin=0.5, inc=60.0, fov=20.0, **more):
    na, nb = res if isinstance(res, tuple) else (res, res)
    c = dict(op=op, na=na, nb=nb, samples=samples, splats=splats, freqs=freqs, frames=frames, precision=precision, spin=spin, inc=inc, fov=fov)
    c.update(more)
    return c


def listed():
    out = [
        # an interactive preview: the smallest image anyone asks for, where launches and latency count
        dict(_case("thin", 24, 64, 3, precision="fp64", spin=0.94, inc=17.0, fov=15.0), name="thin_preview"),
        # the thin image of the quick-look workflow (12 splats, 128 x 128, 512 samples)
        dict(_case("thin", 128, 512, 12, precision="fp64", spin=0.94, inc=17.0, fov=15.0), name="thin_screen"),
        # a new spacetime per step (spin and inclination fits): geodesics rebuilt, one thin image
        dict(_case("refit", 192, 768, 12, precision="fp64"), name="refit"),
        # a small polarized image: few rays, little work to fill the chip with
        dict(_case("render", 32, 128, 8), name="pol_small"),
        # the headline polarized image: 256 x 256, 1024 samples, 64 thermal splats, three frequencies
        dict(_case("render", 256, 1024, 64, freqs=3), name="pol_screen"),
        # the default precision of every polarized call, on a ragged screen
        dict(_case("render", (101, 93), 384, 24, precision="fp64"), name="pol_fp64"),
        # a movie: uneven sample counts, three populations, four frequencies, two frames
        dict(_case("movie", 112, 2048, 96, freqs=4, frames=2, spin=0.94, inc=163.0, fov=15.0), name="movie"),
        # a small fit's step (a coarse image early in a fit)
        dict(_case("grad", 40, 200, 12), name="grad_small"),
        # the image fit's step: 64 x 21 parameters, three frequencies, near the headline size
        dict(_case("grad", 224, 896, 64, freqs=3), name="grad_screen"),
        # the default precision of the gradient
        dict(_case("grad", 48, 160, 10, precision="fp64"), name="grad_fp64"),
        # an interferometric fit's step: many splats, one frequency, 600 baselines
        dict(_case("vis", 192, 512, 160, spin=0.7, inc=30.0, fov=16.0, nuv=600), name="vis_fit"),
        # a Gauss-Newton forward product: J v along two directions
        dict(_case("jvp", 96, 256, 24, dirs=2), name="jvp"),
    ]
    return out


def draw(rng):
    """One more case of the same ranges: sizes log-uniform, odd ones included."""
    def span(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["thin", "refit", "render", "render", "movie", "grad", "grad", "vis", "jvp"])
    spin, inc, fov = round(rng.uniform(0.1, 0.98), 3), round(rng.uniform(12.0, 168.0), 1), round(rng.uniform(12.0, 20.0), 1)
    fp64 = op in ("thin", "refit") or (op in ("render", "grad") and rng.random() < 0.35)
    big = {"thin": 128, "refit": 192, "render": 224, "movie": 100, "grad": 192, "vis": 176, "jvp": 96}[op]
    if fp64 and op in ("render", "grad"):
        big = 96 if op == "render" else 48
    na = span(16, big)
    nb = na if op == "vis" else span(16, big)
    samples = span(64, {"movie": 1500, "jvp": 256, "vis": 512}.get(op, 160 if fp64 and op == "grad" else 384 if fp64 and op == "render" else 900))
    splats = span(3, {"thin": 12, "refit": 12, "render": 64, "movie": 96, "grad": 64, "vis": 160, "jvp": 24}[op] if not fp64 else 12)
    c = _case(op, (na, nb), samples, max(3, splats), precision="fp64" if fp64 else "mixed", spin=spin, inc=inc, fov=fov)
    if op in ("render", "grad", "movie"):
        c["freqs"] = rng.randint(1, 4) if op == "movie" else 1 if fp64 else rng.randint(1, 3)
    if op == "movie":
        c["frames"] = rng.randint(1, 2)
    if op == "vis":
        c["nuv"] = span(20, 600)
    if op == "jvp":
        c["dirs"] = rng.randint(1, 2)
    return c


# ---- inputs ----------------------------------------------------------------------------------------

def _splats(rng, n, a, rows, rlo=2.5, rhi=12.0):
    """`n` splats of the row layout with `rows` rows: centres on near-equatorial orbits, log-uniform widths,
    random orientations, Keplerian pattern rates and (polarized) velocities around the circular orbit's."""
    r, th, ph = rng.uniform(rlo, rhi, n), rng.uniform(np.pi / 3, 2 * np.pi / 3, n), rng.uniform(0.0, 2 * np.pi, n)
    p = np.zeros((rows, n))
    p[0:3] = r * np.sin(th) * np.cos(ph), r * np.sin(th) * np.sin(ph), r * np.cos(th)
    p[3:6] = rng.uniform(np.log(0.3), np.log(2.0), (3, n))
    q = rng.standard_normal((4, n))
    p[6:10] = q / np.linalg.norm(q, axis=0)
    p[11] = np.log(1e9)
    p[rows - 1] = 1.0 / (r ** 1.5 + a)
    if rows == 14:
        p[12] = rng.uniform(0.0, np.log(10.0), n)
        return p
    b = rows - 7   # the field's rows and the velocity's follow the population's
    p[12] = rng.uniform(np.log(1e4), np.log(1e6), n)
    p[13] = rng.uniform(0.0, np.log(50.0), n)
    p[b] = np.log(rng.uniform(1.0, 30.0, n))
    p[b + 1] = np.arccos(rng.uniform(-1.0, 1.0, n))
    p[b + 2] = rng.uniform(0.0, 2 * np.pi, n)
    s2, sg, d = np.sin(th) ** 2, r * r + (a * np.cos(th)) ** 2, r * r - 2 * r + a * a
    big = (r * r + a * a) ** 2 - a * a * d * s2
    om, w = 1.0 / (r ** 1.5 + a), 2 * a * r / big
    v = np.sqrt(big * s2 / sg) * (om - w) / np.sqrt(sg * d / big)    # the orbit's speed seen by the ZAMO
    uk = np.zeros((3, n))
    uk[1] = v / np.sqrt(np.maximum(1.0 - v * v, 0.05))
    p[b + 3:b + 6] = uk + 0.1 * np.linalg.norm(uk, axis=0) * rng.standard_normal((3, n))
    return p


def _hyp2f1(kap, w):
    """2F1(kappa - 1/3, kappa + 1; kappa + 2/3; -kappa w) by its Euler integral over ln t."""
    x, g = np.polynomial.legendre.leggauss(20)
    e = np.linspace(-32.0, 0.0, 65)
    v = (0.5 * (e[1:] + e[:-1])[:, None] + 0.25 * x).ravel()
    g = np.tile(0.25 * g, 64)
    b = kap - 1.0 / 3
    return np.array([bi * np.sum(g * np.exp(bi * v) * (1 + k * wi * np.exp(v)) ** -(k + 1)) for bi, k, wi in zip(b, kap, w)])


def _scene(case, seed):
    """Everything the seed decides, in numpy: splat matrices, times, and the data of a fit."""
    rng = np.random.Generator(np.random.PCG64([int(seed), case["na"], case["nb"], case["samples"], case["splats"]]))
    a, n, op = case["spin"], case["splats"], case["op"]
    s = dict(nus=np.array(NUS[:case["freqs"]]), times=10.0 * np.arange(case["frames"]) + rng.uniform(0.0, 5.0), L=L_SGRA)
    if op in ("thin", "refit"):
        s["p"] = _splats(rng, n, a, 14, 3.0, 10.0)
        return s
    if op == "movie":
        m = n // 3
        pt, pp, pk = _splats(rng, m, a, 21), _splats(rng, m, a, 22), _splats(rng, n - 2 * m, a, 22)
        pp[13], pp[14] = rng.uniform(2.5, 3.5, m), np.log(10.0)
        pk[13], pk[14] = rng.uniform(3.0, 6.0, n - 2 * m), rng.uniform(0.0, np.log(50.0), n - 2 * m)
        kt = np.linspace(-80.0, 20.0 + s["times"][-1], 4)
        rho, ph = np.hypot(pt[0], pt[1]), np.arctan2(pt[1], pt[0])
        ang = ph[None] + pt[20][None] * kt[:, None]
        s.update(sets=[("knot", pt), ("power", pp), ("kappa", pk)], knot_times=kt, hyp=_hyp2f1(pk[13], np.exp(pk[14])),
                 knots=np.stack([rho * np.cos(ang), rho * np.sin(ang), np.broadcast_to(pt[2], ang.shape)]))
        return s
    p = _splats(rng, n, a, 21)
    s.update(p=p, sets=[("thermal", p)])
    al, be = _pixels(case)
    spots = rng.uniform(-0.5, 0.5, (2, 5)) * case["fov"], rng.uniform(0.1, 0.25, 5) * case["fov"], rng.uniform(0.3, 1.0, 5)
    if op == "grad":
        # a target image of bright spots with polarized fractions, and one percent noise
        npix, nf, nt = al.size, case["freqs"], case["frames"]
        img = sum(w * np.exp(-((al - x) ** 2 + (be - y) ** 2) / (2 * sd * sd)) for (x, y), sd, w in zip(spots[0].T, spots[1], spots[2]))
        frac = np.concatenate([[1.0], rng.uniform(-0.3, 0.3, 3)])
        peak = 2e-4
        s["data"] = peak * (img[None, None, :, None] * frac + 0.01 * rng.standard_normal((nf, nt, npix, 4)))
        s["sigma"] = 0.01 * peak
    if op == "vis":
        s["L"] = L_M87
        step = 2 * case["fov"] / (case["na"] - 1)
        psize = step * L_M87 / DIST_M87
        rad, ang = 10e9 * np.sqrt(rng.uniform(0.0, 1.0, case["nuv"])), rng.uniform(0.0, 2 * np.pi, case["nuv"])
        u, v = rad * np.cos(ang), rad * np.sin(ang)
        flux = 0.6 * np.exp(-2 * (np.pi * 3.0 * L_M87 / DIST_M87) ** 2 * rad ** 2)
        vis = flux[:, None] * np.exp(2j * np.pi * (u[:, None] * 2 * psize)) * np.concatenate([[1.0], rng.uniform(-0.2, 0.2, 3)])
        noise = 0.02 * (rng.standard_normal((case["nuv"], 4)) + 1j * rng.standard_normal((case["nuv"], 4)))
        s.update(u=u, v=v, psize=psize, scale=psize ** 2 / 1e-23, vis=vis + 0.6 * noise, vsigma=np.full((case["nuv"], 4), 0.012))
    if op == "jvp":
        s["dirs"] = rng.standard_normal((case["dirs"], 21, n)) * np.maximum(np.abs(p), 0.1)
    return s


def _pixels(case):
    cam = _camera(case)
    return cam.alpha, cam.beta


def _camera(case):
    """The screen, pointed a little off the hole (no pixel on the spin axis' projection, where the azimuth is undefined)."""
    f = case["fov"]
    return ks.Camera((0.11 - f, 0.11 + f), (-0.07 - f, f - 0.07), (case["na"], case["nb"]))


def prepare(case, seed):
    """The camera, its cache (regenerated, except where the call itself does that) and the inputs."""
    s = _scene(case, seed)
    cache = ks.GeodesicCache(_camera(case), case["samples"])
    if case["op"] != "refit":
        ks.regenerate(cache, case["spin"], np.deg2rad(case["inc"]), marcher=ks.Fused(64), uneven=_uneven(case))
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    for key in ("p", "data"):
        if key in s:
            s[key] = torch.as_tensor(s[key], device=dev)
    if "sets" in s and case["op"] == "movie":
        s["sets"] = [(kind, torch.as_tensor(p, device=dev)) for kind, p in s["sets"]]
    s.update(case=case, cache=cache, precision=ks.KS_FP64 if case["precision"] == "fp64" else ks.KS_MIXED)
    return s


def _uneven(case):
    return (768.0, min(128, case["samples"])) if case["op"] == "movie" else None


def run(s):
    """One pass: the call as a fit loop or a renderer makes it, with this pass's parameters."""
    case, cache, op, prec = s["case"], s["cache"], s["case"]["op"], s["precision"]
    if op == "refit":
        ks.regenerate(cache, case["spin"], np.deg2rad(case["inc"]), marcher=ks.Fused(64))
    if op in ("thin", "refit"):
        return ks.thin_image(cache, s["p"], s["times"][0], precision=prec)
    if op == "movie":
        (_, pt), (_, pp), (_, pk) = s["sets"]
        model = ks.CompositeModel(ks.KnotSplats(pt, s["knots"], s["knot_times"]), ks.PowerLawSplats(pp), ks.KappaSplats(pk, hyp=s["hyp"]))
        return ks.render(cache, model, s["times"], s["nus"], s["L"], precision=prec)
    model = ks.PolarizedSplats(s["p"])
    if op == "render":
        return ks.render(cache, model, s["times"], s["nus"], s["L"], precision=prec)
    if op == "grad":
        return ks.chi2_gradient(cache, model, s["times"], s["nus"], s["L"], s["data"], s["sigma"], precision=prec)
    if op == "vis":
        return ks.vis_chi2_gradient(cache, model, s["times"][0], s["nus"][0], s["L"], s["u"], s["v"], s["vis"], s["vsigma"], s["psize"],
                                    s["scale"], precision=prec)
    return ks.jvp(cache, model, s["times"], s["nus"], s["L"], s["dirs"], precision=prec)


def work(case):
    """Bytes of the inputs and outputs and the arithmetic of one pass: the march of every ray-sample, the
    evaluations of the (sample, splat) pairs inside a support (about one sample in ninety per splat), one
    exact step per frequency of the samples that any splat reaches."""
    rays, n, nf, nt = case["na"] * case["nb"], case["splats"], case["freqs"], case["frames"]
    per_ray = min(case["samples"], 336) if case["op"] == "movie" else case["samples"]
    samples = rays * per_ray
    rows = 14 if case["op"] in ("thin", "refit") else 21
    out = rays * (1 if rows == 14 else 4 * nf * nt) * 8
    bytes_ = rows * n * 8 + out
    if rows == 14:
        flops = samples * (330 + 40 * n)
        if case["op"] == "refit":
            flops += samples / 4 * 16 * 150
        return {"bytes": bytes_, "flops": flops}
    pairs = samples * n * 0.0112
    steps = samples * nf * (1.0 - math.exp(-n * 0.0033))
    flops = samples * 330 + nt * (pairs * (150 + 200 * nf) + steps * 700)
    if case["op"] in ("grad", "vis"):
        flops = samples * 330 + nt * (pairs * (900 + 1200 * nf) + steps * 2500)
        bytes_ += out + rows * n * 8
    if case["op"] == "jvp":
        flops = samples * 330 + (1 + case["dirs"]) * (flops - samples * 330)
        bytes_ += case["dirs"] * (out + rows * n * 8)
    return {"bytes": bytes_, "flops": flops}


# ---- exact values: the geodesics ---------------------------------------------------------------------

def _rf(x, y, z):
    """Carlson's R_F by duplication."""
    a0 = (x + y + z) / 3
    x0, y0, a, f = x, y, a0, 1.0
    for _ in range(14):
        sx, sy, sz = x.sqrt(), y.sqrt(), z.sqrt()
        lam = sx * sy + sx * sz + sy * sz
        x, y, z, a, f = (x + lam) / 4, (y + lam) / 4, (z + lam) / 4, (a + lam) / 4, f / 4
    p, q = (a0 - x0) * f / a, (a0 - y0) * f / a
    r = -p - q
    e2, e3 = p * q - r * r, p * q * r
    return (1 - e2 / 10 + e3 / 14 + e2 * e2 / 24 - 3 * e2 * e3 / 44) / a.sqrt()


def _ellf(phi, m):
    """F(phi | m)."""
    one = torch.ones_like(phi)
    j = torch.round(phi / math.pi)
    s, c = torch.sin(phi - j * math.pi), torch.cos(phi - j * math.pi)
    return s * _rf(c * c, 1 - m * s * s, one) + 2 * j * _rf(0 * one, 1 - m, one)


class _Jacobi:
    """sn, cn, dn of one modulus per ray by the descending Landen scale."""

    def __init__(self, m, levels=11):
        self.m, a, b, c = m, torch.ones_like(m), (1 - m).sqrt(), m.sqrt()
        self.scale = []
        for _ in range(levels):
            a, b, c = (a + b) / 2, (a * b).sqrt(), c * c / (2 * (a + b))
            self.scale.append((a, c))

    def at(self, u):
        phi = self.scale[-1][0] * u * 2.0 ** len(self.scale)
        for a, c in reversed(self.scale):
            phi = (phi + torch.asin(torch.clamp(c * torch.sin(phi) / a, -1, 1))) / 2
        s = torch.sin(phi)
        return s, torch.cos(phi), (1 - self.m * s * s).sqrt()


class _Rays:
    """The closed-form geodesics of a batch of screen points (columns: rays, rows: Mino times)."""

    def __init__(self, al, be, a, tho):
        self.al, self.be, self.a = al, be, a
        ct, st = math.cos(tho), math.sin(tho)
        self.st = st
        self.rp, self.rm = 1 + math.sqrt(1 - a * a), 1 - math.sqrt(1 - a * a)
        eta, lam = (al * al - a * a) * ct * ct + be * be, -al * st
        self.eta, self.lam = eta, lam
        A, B, C = a * a - eta - lam * lam, 2 * (eta + (lam - a) ** 2), -a * a * eta
        P, Q = -A * A / 12 - C, -A / 3 * ((A / 6) ** 2 - C) - B * B / 8
        disc = torch.complex((P / 3) ** 3 + (Q / 2) ** 2, torch.zeros_like(P)).sqrt()
        w = (-Q / 2 + disc)
        w = torch.polar(w.abs() ** (1 / 3), w.angle() / 3)
        z = (torch.clamp((w - P / (3 * w)).real - A / 3, min=0) / 2).sqrt()
        d12, d34 = -A / 2 - z * z + B / (4 * z), -A / 2 - z * z - B / (4 * z)
        s12, s34 = torch.complex(d12, 0 * d12).sqrt(), torch.complex(d34, 0 * d34).sqrt()
        r1, r2, r3, r4 = -z - s12, -z + s12, z - s34, z + s34
        real = [r.real for r in (r1, r2, r3, r4)]
        c2, c4 = (d12 >= 0) & (d34 >= 0), (d12 < 0) & (d34 < 0)
        c3 = ~(c2 | c4)
        self.c2, self.c3, self.c4 = c2, c3, c4
        one = torch.ones_like(al)

        def pick(x2, x3, x4):
            return torch.where(c2, x2, torch.where(c3, x3, x4))

        # four real roots
        q1, q2, q3, q4 = real
        r31, r32, r41, r42 = q3 - q1, q3 - q2, q4 - q1, q4 - q2
        k2, cc2 = r32 * r41 / (r31 * r42), (r31 * r42).abs().sqrt() / 2
        # two real roots
        r21 = (r2 - r1).real
        Aa, Bb = (r3 - r2).abs(), (r3 - r1).abs()
        k3, cc3 = ((Aa + Bb) ** 2 - r21 ** 2) / (4 * Aa * Bb), (Aa * Bb).sqrt()
        # none
        a1, a2, b1, b2 = s34.imag.abs(), s12.imag.abs(), real[3], real[1]
        Cc, Dd = ((a1 - a2) ** 2 + (b1 - b2) ** 2).sqrt(), ((a1 + a2) ** 2 + (b1 - b2) ** 2).sqrt()
        k4, cc4 = 4 * Cc * Dd / (Cc + Dd) ** 2, (Cc + Dd) / 2
        g0 = torch.clamp((4 * a2 ** 2 - (Cc - Dd) ** 2) / ((Cc + Dd) ** 2 - 4 * a2 ** 2), min=0).sqrt()
        self.k = torch.clamp(pick(k2, k3, k4), 0, 1 - 1e-16)
        self.c = pick(cc2, cc3, cc4)
        phi0 = pick(torch.asin(torch.clamp(r31 / r41, 0, 1).sqrt()), torch.acos(torch.clamp((Aa - Bb) / (Aa + Bb), -1, 1)),
                    math.pi / 2 + torch.atan(g0))
        self.fo = _ellf(torch.nan_to_num(phi0), self.k) / self.c
        self.m0 = pick(q1, -Aa * q1 + Bb * q2, a2)
        self.m1 = pick(q3, Aa * q1 + Bb * q2, b1)
        self.m2 = pick(r41, Bb - Aa, g0)
        self.m3 = pick(q4 - q3, Aa + Bb, one)
        rh = self.rp
        x2 = torch.asin(torch.clamp(r31 * (q4 - rh) / (r41 * (q3 - rh)), 0, 1).sqrt())
        x3 = torch.acos(torch.clamp((self.m0 - rh * self.m2) / (rh * self.m3 - self.m1), -1, 1))
        w4 = -(rh + b1) / a2
        x4 = torch.atan((g0 - w4) / (1 + w4 * g0))
        x4 = torch.where(x4 < 0, x4 + math.pi, x4)
        hit = self.fo - _ellf(torch.nan_to_num(pick(x2, x3, x4)), self.k) / self.c
        plunge = c2 & (q4 < rh)
        self.total = torch.where(c2, 2 * self.fo, hit)
        self.valid = torch.where(plunge, hit, torch.full_like(hit, math.inf))
        self.scatter, self.r4 = c2 & ~plunge, q4
        # polar motion
        dth = (1 - (eta + lam * lam) / (a * a)) / 2
        dsc = (dth * dth + eta / (a * a)).sqrt()
        up, um = dth + dsc, dth - dsc
        vort = eta < 0
        self.vort, self.um, self.dup, self.sqrt_up = vort, um, up - um, up.sqrt()
        kq = torch.where(vort, 1 - up / um, up / um)
        self.tf = 1 / (um * a * a).abs().sqrt()
        sb = torch.sign(be)
        arg = torch.where(vort, torch.clamp((ct * ct - um) / (up - um), 0, 1).sqrt(), torch.clamp(ct / up.sqrt(), -1, 1))
        g = self.tf * _ellf(torch.asin(arg), kq)
        sigma = -1.0 if tho > math.pi / 2 else 1.0
        self.off = torch.where(vort, sigma * sb * g, sb * g)
        self.psign = torch.where(vort, sigma * one, sb)
        self.pmu, self.ps = -kq / (1 - kq), (1 - kq).sqrt()
        self.jr, self.jt = _Jacobi(self.k), _Jacobi(self.pmu)
        # the split of the time and azimuth integrals
        E, Em, h = self.rp ** 2 + a * a - a * lam, self.rm ** 2 + a * a - a * lam, self.rp - self.rm
        self.sp, self.sm = -E.abs(), -Em.abs()
        self.qt, self.qtm = (self.rp ** 2 + a * a) * E / h, -(self.rm ** 2 + a * a) * Em / h
        self.qp, self.qpm = a * (2 * self.rp - a * lam) / h, -a * (2 * self.rm - a * lam) / h
        self.qc = torch.where(vort, 1 / (1 - um), one)
        self.qn = torch.where(vort, (up - um) / (1 - um), up)
        self.eps = torch.clamp(1 - self.qn, min=0).sqrt()
        mneg = -self.pmu / (1 - self.pmu)
        self.gc, self.mp = 1 / (1 - mneg).sqrt(), mneg / (1 - mneg)
        self.k2 = 2 * _rf(0 * one, 1 - self.pmu, one) / self.ps
        self.ct = ct

    def polar(self, tau):
        s, c, d = self.jt.at(self.ps * (tau + self.off) / self.tf)
        sx = s / (self.ps * d)
        cth = torch.where(self.vort, self.psign * torch.clamp(self.um + self.dup * sx * sx, min=0).sqrt(), self.psign * self.sqrt_up * sx)
        nu = torch.where(self.vort, self.psign * s * c > 0, self.psign * c > 0)
        return torch.clamp(cth, -1, 1), nu, sx, c / d, 1 / d

    def radius(self, tau):
        s, c, _ = self.jr.at(self.c * (self.fo - tau))
        q = self.m2 * c * c
        r2 = (self.m1 * q - self.m0 * self.m3) / (q - self.m3)
        r3 = (self.m0 + self.m1 * c) / (self.m2 + self.m3 * c)
        sc = s / c
        r4 = -(self.m0 * (self.m2 - sc) / (1 + self.m2 * sc) + self.m1)
        return torch.where(self.c2, r2, torch.where(self.c3, r3, r4))

    def rates(self, tau):
        """The smooth parts of dt/dtau and dphi/dtau (large r, both horizons and the polar axis taken out)."""
        r = self.radius(tau)
        cth, _, sn, cn, di = self.polar(tau)
        a, lam = self.a, self.lam
        d, p = r * r - 2 * r + a * a, r * r + a * a - a * lam
        s = torch.where(tau < self.fo, -1.0, 1.0) * torch.clamp(p * p - d * (self.eta + (lam - a) ** 2), min=0).sqrt()
        wp, wm = s * self.rp / (r * (r - self.rp)) / self.sp, s * self.rm / (r * (r - self.rm)) / self.sm
        q = self.eta + (lam - a) ** 2
        far = d * q / (p + s.abs()) * (1 + 2 / r) + 2 * (2 * r - a * a) * p / (r * d)
        near = (r * r + a * a) * p / d - s.abs() * (1 + 2 / r)
        gt = torch.where((r > 64) & (p > 0), far, near) + a * (lam - a * (1 - cth * cth)) - self.qt * wp - self.qtm * wm
        pol = lam * self.qc * (1 - self.gc * di * (1 - self.mp * cn * cn / 2)) / (1 - self.qn * sn * sn)
        gp = a * (2 * r - a * lam) / d - self.qp * wp - self.qpm * wm + pol
        return gt, gp

    def closed(self, tau, sn, cn):
        x = (tau + self.off) / self.tf
        nw = torch.floor((x + self.k2 / 2) / self.k2) * math.pi
        t = sn / cn
        e = self.eps * self.eps
        A = (torch.atan(self.eps * t) + nw) / self.eps
        return self.lam * self.qc * self.tf * self.gc * ((1 + self.mp * e / (2 * self.qn)) * A - self.mp / (2 * self.qn) * (torch.atan(t) + nw))

    def integral(self, lo, hi, nodes):
        """Gauss-Legendre integrals of both rates over [lo, hi]; the step at fo is split by the caller."""
        x, w = np.polynomial.legendre.leggauss(nodes)
        mid, half = (lo + hi) / 2, (hi - lo) / 2
        it, ip = torch.zeros_like(mid), torch.zeros_like(mid)
        for xi, wi in zip(x, w):
            gt, gp = self.rates(mid + half * xi)
            it, ip = it + wi * gt, ip + wi * gp
        return half * it, half * ip

    def march(self, count, nmax):
        """Every sample of every ray, (nmax, rays); `count` samples per ray."""
        k = torch.arange(1, nmax + 1, device=self.al.device, dtype=torch.float64)[:, None]
        dtau = self.total / (count + 1)
        tau = k * dtau
        inside = k <= count
        tau = torch.where(inside, tau, count * dtau)
        prev = torch.cat([torch.zeros_like(tau[:1]), tau[:-1]])
        split = self.scatter & (prev < self.fo) & (self.fo < tau)
        it, ip = self.integral(prev, torch.where(split, self.fo, tau), 6 if nmax > 96 else 16)
        at = split.any(0)
        first = torch.where(at, torch.where(split, tau, torch.zeros_like(tau)).sum(0), self.fo + 1)
        i2, p2 = self.integral(self.fo[None], first[None], 16)
        i1, p1 = self.integral(torch.zeros_like(tau[:1]), tau[:1], 40)
        it[0], ip[0] = torch.where(split[0], it[0], i1[0]), torch.where(split[0], ip[0], p1[0])
        it, ip = it + torch.where(split, i2, 0.0), ip + torch.where(split, p2, 0.0)
        it, ip = it.cumsum(0), ip.cumsum(0)
        r = self.radius(tau)
        cth, nuth, sn, cn, _ = self.polar(tau)
        f, f4 = r + 2 * r.log(), self.r4 + 2 * torch.clamp(self.r4, min=1e-3).log()
        lead = torch.where(self.scatter & (tau > self.fo), f - 2 * f4, -f)
        lp, lm = torch.log((r - self.rp) / r) / self.sp, torch.log((r - self.rm) / r) / self.sm
        zero = torch.zeros_like(self.al)
        _, _, sn0, cn0, _ = self.polar(zero)
        t = lead + self.qt * lp + self.qtm * lm + it
        phi = self.qp * lp + self.qpm * lm + self.closed(tau, sn, cn) - self.closed(zero, sn0, cn0) + ip
        # visibility: a sample inside the polar cap needs |beta| above the cap's boundary
        s2 = 1 - cth * cth
        cap = (cth > abs(self.ct)) & (self.al.abs() >= self.a * s2.sqrt() + 2.220446049250313e-16)
        edge = torch.clamp((self.ct ** 2 - cth * cth) * (self.al ** 2 - self.a ** 2 * s2) / (cth * cth - 1), min=0).sqrt()
        ok = inside & (tau <= self.valid) & ~(cap & (self.be.abs() + 2.220446049250313e-16 < edge))
        return dict(t=t, r=r, cth=cth, phi=phi, nur=tau < self.fo, nuth=nuth, ok=ok & (r > self.rp * (1 + 1e-3)), dtau=dtau)


# ---- exact values: the plasma ---------------------------------------------------------------------------

ME, CL, EE, HPL, NU0 = 9.1093826e-28, 2.99792458e10, 4.80320680e-10, 6.6260693e-27, 1e11


def _bessel(x):
    """K0, K1 by the trapezoidal rule on their integral over t (exp(-x) left out: only ratios are used)."""
    t = torch.arange(0, 260, device=x.device, dtype=torch.float64)[:, None] * 0.045
    e = torch.exp(-x * (torch.cosh(t) - 1)) * torch.where(t == 0, 0.5, 1.0)
    return e.sum(0), (e * torch.cosh(t)).sum(0)


def _thermal(c, ne, B, nu, st, ct):
    Te, f0, kr = c["Te"], c["f0"], c["kr"]
    w0, wp2, w = EE * B / (ME * CL), 4 * math.pi * ne * EE * EE / ME, 2 * math.pi * nu
    a, b = w0 / w, wp2 / (w * w)
    x = Te * torch.sqrt(math.sqrt(2) * st * 1e3 * a)
    sw = 0.5 + 0.5 * torch.tanh((torch.log(x) - math.log(120.0)) / 0.1)
    extra = (0.011 * torch.exp(-x / 47.2) - 2 ** (-1 / 3) / 3 ** (23 / 6) * math.pi * 1e4 * (x + 1e-16) ** (-8 / 3)) * sw
    ffn = 2.011 * torch.exp(-x ** 1.035 / 4.7) - torch.cos(x / 2) * torch.exp(-x ** 1.2 / 2.73) - 0.011 * torch.exp(-x / 47.2) + extra
    rQ = w / (2 * CL) * ffn * b * a * a * (kr + 6 * Te) * st * st
    rV = w / CL * b * a * f0 * (1 - 0.11 * torch.log(1 + 0.035 * x)) * ct
    xs = nu / (3 * EE * B * st / (4 * math.pi * ME * CL) * Te * Te + 1)
    c3 = xs ** (-1 / 3)
    e3 = torch.exp(-1.8899 / c3)
    pre = ne * EE * EE * nu / (2 * math.sqrt(3) * CL * Te * Te)
    jI = pre * 2.5651 * (1 + 1.92 * c3 + 0.9977 * c3 * c3) * e3
    jQ = pre * 2.5651 * (1 + 0.93193 * c3 + 0.499873 * c3 * c3) * e3
    jV = 2 * ne * EE * EE * nu * ct / st / (3 * math.sqrt(3) * CL * Te ** 3) * (1.81384 / xs + 3.42319 * c3 * c3 + 0.0292545 * xs ** -0.5 + 2.03773 * c3) * e3
    y = HPL * nu / (ME * CL * CL * Te)
    bn = 2 * HPL * nu ** 3 / (CL * CL) / torch.expm1(y)
    return jI, jQ, jV, jI / bn, jQ / bn, jV / bn, rQ, rV


def _power(c, ne, B, nu, st, ct):
    p, gmin, span, gj, ga = c["p"], c["gmin"], c["span"], c["gj"], c["ga"]
    nc = EE * B / (2 * math.pi * ME * CL)
    xx = nu / (nc * st)
    jI = ne * EE * EE * nc / CL * 3 ** (p / 2) * (p - 1) * st / (2 * (p + 1) * span) * gj * xx ** (-(p - 1) / 2)
    jQ = (p + 1) / (p + 7 / 3) * jI
    jV = 171 / 250 * p ** 0.49 * ct / st * (xx / 3) ** -0.5 * jI
    aI = ne * EE * EE / (nu * ME * CL) * 3 ** ((p + 1) / 2) * (p - 1) / (4 * span) * ga * xx ** (-(p + 2) / 2)
    aQ = aI * (17 / 500 * p - 43 / 1250) ** 0.086
    aV = aI * (0.71 * p + 22 / 625) ** 0.394 * torch.clamp(3.1 * st ** -1.92 - 3.1, min=0) ** 0.512 * xx ** -0.5 * torch.sign(ct)
    nb = nc * st
    rp = ne * EE * EE * (p - 1) / (ME * CL * nb * span)
    rQ = -rp * (nb / nu) ** 3 * gmin ** (2 - p) * (1 - (gmin * gmin * nb / nu) ** (p / 2 - 1)) / (p / 2 - 1)
    rV = 2 * (p + 2) / (p + 1) * rp * (nb / nu) ** 2 * gmin ** -(p + 1) * torch.log(gmin) * ct / st
    return jI, jQ, jV, aI, aQ, aV, rQ, rV


_RHO_Q = ((17, 3, 7, 30, 0.1, 1.5, 0.471), (46 / 3, 5 / 3, 17 / 3, 18, 1 / 6, 1.75, 0.5), (14, 13 / 8, 4.5, 12, 0.25, 2.0, 0.525),
          (12.5, 1, 5, 8, 0.375, 2.25, 0.541))


def _kappa(c, ne, B, nu, st, ct):
    k, w, hyp = c["kap"], c["w"], c["hyp"]
    nc = EE * B / (2 * math.pi * ME * CL)
    X = nu / ((w * k) ** 2 * nc * st)
    pre, sg = ne * EE * EE * nc * st / CL, torch.sign(ct)

    def bridge(lo, hi, x, slope):   # the fits' join of their low- and high-frequency limits
        return lo * (1 + X ** (x * slope) * (lo / hi) ** x) ** (-1 / x)

    g = 4 * math.pi * c["g43"] / (3 ** (7 / 3) * c["g2"])
    hk = 0.25 * 3 ** ((k - 1) / 2) * (k - 2) * (k - 1) * c["gq"] * c["gp"]
    sj, X3 = (3 * k - 4) / 6, X ** (1 / 3)
    jI = pre * X3 * bridge(g, hk, 3 * k ** -1.5, sj)
    jQ = pre * X3 * bridge(0.5 * g, (0.64 + k / 50) * hk, 3.7 * k ** -1.6, sj)
    lowV = 0.5625 * torch.clamp(st ** -2.4 - 1, min=1e-300) ** 0.48 * k ** -0.528 / w * X ** -0.35 * g
    highV = 0.765625 * torch.clamp(st ** -2.5 - 1, min=1e-300) ** 0.44 * k ** -0.44 / w * X ** -0.5 * hk
    jV = pre * X3 * bridge(lowV, highV, 3 * k ** -1.5, sj) * sg
    ap, ck = ne * EE / (B * st), (k - 2) * (k - 1) * k
    base = 3 ** (1 / 6) * 10 / 41 * 4 * math.pi ** 2 / (w * k) ** (16 / 3 - k) * ck / (3 * k - 1) * math.gamma(5 / 3) * hyp
    hi = 2 * math.pi ** 2.5 / 3 * ck / (w * k) ** 5 * (2 * c["gk2"] / (2 + k) - 1)
    sa, X5 = (3 * k - 1) / 6, X ** (-5 / 3)
    aI = ap * X5 * bridge(base, hi * ((3 / k) ** 4.75 + 0.6), (-1.75 + 1.6 * k) ** -0.86, sa)
    aQ = ap * X5 * bridge(25 / 48 * base, (441 * k ** -5.76 + 0.55) * hi, 1.4 * k ** -1.15, sa)
    lowA = 0.77 / w * torch.clamp(st ** -2.28 - 1, min=1e-300) ** 0.446 * X ** -0.35 * k ** -0.7 * base
    highA = 14.3 * w ** -0.928 * torch.clamp(st ** -2.05 - 1, min=1e-300) ** 0.5 * (169 * k ** -8 + 13 / 2500 * k - 263 / 5000 + 47 / (200 * k)) * X ** -0.5 * hi
    aV = ap * X5 * bridge(lowA, highA, 1.22 * k ** -1.136 + 0.007, sa) * sg
    sw, e5, xm = w.sqrt(), torch.exp(-5 * w), X ** -0.5
    fq = torch.stack([(q[0] * w - q[1] * sw + q[2] * sw * e5) * (1 - torch.exp(-X ** 0.84 / q[3]) - torch.sin(q[4] * X) * torch.exp(-q[5] * X ** q[6]))
                      for q in _RHO_Q])
    fv = torch.stack([(w * w + 2 * w + 1) / (3.125 * w * w + 4 * w + 1) * (1 - 0.17 * torch.log(1 + 0.447 * xm)),
                      (w * w + 54 * w + 50) / (30 / 11 * w * w + 134 * w + 50) * (1 - 0.17 * torch.log(1 + 0.391 * xm)),
                      (w * w + 43 * w + 38) / (7 / 3 * w * w + 92.5 * w + 38) * (1 - 0.17 * torch.log(1 + 0.348 * xm)),
                      (w + 13 / 14) / (2 * w + 13 / 14) * (1 - 0.17 * torch.log(1 + 0.313 * xm))])
    kc = torch.clamp(k, 3.5, 5)
    i = torch.clamp(torch.floor((kc - 3.5) * 2), 0, 2)
    f, i = (kc - 3.5) * 2 - i, i.long()[None]
    fq = (1 - f) * fq.gather(0, i)[0] + f * fq.gather(0, i + 1)[0]
    fv = (1 - f) * fv.gather(0, i)[0] + f * fv.gather(0, i + 1)[0]
    rQ = -ne * (EE * nc * st) ** 2 / (ME * CL * nu ** 3) * fq
    rV = 2 * ne * EE * EE * nc * ct / (ME * CL * nu * nu) * c["kb"] * fv
    return jI, jQ, jV, aI, aQ, aV, rQ, rV


_FITS = {"thermal": _thermal, "knot": _thermal, "power": _power, "kappa": _kappa}


def _constants(kind, p, scene):
    """What a splat's column fixes, differentiable in the column."""
    b = 14 if kind in ("thermal", "knot") else 15
    q = p[6:10] / p[6:10].norm(dim=0)
    w, x, y, z = q
    R = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y), 2 * (x * y + w * z), 1 - 2 * (x * x + z * z),
                     2 * (y * z - w * x), 2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)])
    c = dict(kind=kind, pos=p[0:3], es=torch.exp(-p[3:6]), R=R, t0=p[10], iw=torch.exp(-p[11]), om=p[-1], ne=torch.exp(p[12]),
             reach=13.815510557964274 * 2 * torch.exp(2 * p[3:6].max(0).values), B=torch.exp(p[b]), u=p[b + 3:b + 6],
             bh=torch.stack([torch.sin(p[b + 1]) * torch.cos(p[b + 2]), torch.sin(p[b + 1]) * torch.sin(p[b + 2]), torch.cos(p[b + 1])]))
    if kind in ("thermal", "knot"):
        Te = torch.exp(p[13])
        k0, k1 = _bessel(1 / Te)
        kk = k0 + 2 * k1 * Te
        c.update(Te=Te, f0=k0 / kk, kr=k1 / kk)
    elif kind == "power":
        q, gm = p[13], torch.exp(p[14])
        c.update(p=q, gmin=gm, span=gm ** (1 - q) - 1e5 ** (1 - q), gj=torch.exp(torch.lgamma((3 * q - 1) / 12) + torch.lgamma((3 * q + 19) / 12)),
                 ga=torch.exp(torch.lgamma((3 * q + 2) / 12) + torch.lgamma((3 * q + 22) / 12)))
    else:
        k, w = p[13], torch.exp(p[14])
        k0, k1 = _bessel(1 / w)
        c.update(kap=k, w=w, hyp=torch.as_tensor(scene["hyp"], device=p.device), kb=k0 / (k0 + 2 * k1 * w),
                 **{n: torch.exp(torch.lgamma(v)) for n, v in (("g43", k - 4 / 3), ("g2", k - 2), ("gq", k / 4 - 1 / 3), ("gp", k / 4 + 4 / 3), ("gk2", 2 + k / 2))})
    if kind == "knot":
        c.update(knots=torch.as_tensor(scene["knots"], device=p.device), kt=torch.as_tensor(scene["knot_times"], device=p.device))
    return c


def _exponent(c, i, t, x, y, z, own=None):
    """The Gaussian's exponent of splats `i` at the points (`own`: their constants, if gathered already)."""
    own = own or _pairs_of(c, i)
    if c["kind"] == "knot":
        kt, kn = c["kt"], c["knots"]
        j = torch.clamp(torch.searchsorted(kt, t.detach(), right=True) - 1, 0, kt.numel() - 2)
        f = torch.clamp((t - kt[j]) / (kt[j + 1] - kt[j]), 0, 1)
        d = [v - ((1 - f) * kn[a, j, i] + f * kn[a, j + 1, i]) for a, v in enumerate((x, y, z))]
        e = d
    else:
        ph = own["om"] * (t - own["t0"])
        s, co = torch.sin(ph), torch.cos(ph)
        px, py, pz = own["pos"]
        d = [x - (px * co - py * s), y - (px * s + py * co), z - pz]
        e = [d[0] * co + d[1] * s, -d[0] * s + d[1] * co, d[2]]
    R, q = own["R"], 0.0
    for a in range(3):
        q = q + ((R[a] * e[0] + R[3 + a] * e[1] + R[6 + a] * e[2]) * own["es"][a]) ** 2
    return (q + ((t - own["t0"]) * own["iw"]) ** 2) / 2


def _frame(S, j, u, bh):
    """Redshift, pitch angle and the screen rotation of pairs: sample rows `j`, fluid velocity, field direction."""
    a, r, cth, lam, eta = S["a"], S["r"][j], S["cth"][j], S["lam"][j], S["eta"][j]
    s2 = 1 - cth * cth
    sth = s2.sqrt()
    Sg, D = r * r + a * a * cth * cth, r * r - 2 * r + a * a
    A = (r * r + a * a) ** 2 - a * a * D * s2
    Pr = r * r + a * a - a * lam
    pr = torch.where(S["nur"][j], 1.0, -1.0) * torch.clamp(Pr * Pr - D * (eta + (lam - a) ** 2), min=0).sqrt() / D
    pth = torch.where(S["nuth"][j], 1.0, -1.0) * torch.clamp(eta + a * a * cth * cth - (lam * cth) ** 2 / s2, min=0).sqrt()
    gtp = -2 * a * r / (Sg * D)
    p0, p1, p2, p3 = A / (Sg * D) + gtp * lam, D / Sg * pr, pth / Sg, -gtp + (D - a * a * s2) / (Sg * D * s2) * lam
    lapse, om, varpi = (Sg * D / A).sqrt(), 2 * a * r / A, (A / Sg).sqrt() * sth
    z = [lapse * p0, (Sg / D).sqrt() * p1, varpi * (p3 - om * p0), -Sg.sqrt() * p2]
    gam = (1 + u[0] ** 2 + u[1] ** 2 + u[2] ** 2).sqrt()
    ud = u[0] * z[1] + u[1] * z[2] + u[2] * z[3]
    g = 1 / (gam * z[0] - ud)
    k = [(z[m + 1] - u[m] * z[0] + u[m] * ud / (gam + 1)) * g for m in range(3)]
    cosb = k[0] * bh[0] + k[1] * bh[1] + k[2] * bh[2]
    f = [k[1] * bh[2] - k[2] * bh[1], k[2] * bh[0] - k[0] * bh[2], k[0] * bh[1] - k[1] * bh[0]]
    n = (f[0] ** 2 + f[1] ** 2 + f[2] ** 2).sqrt()
    f = [v / n for v in f]
    fd = u[0] * f[0] + u[1] * f[1] + u[2] * f[2]
    fz = [f[m] + u[m] * fd / (gam + 1) for m in range(3)]
    ft, fr, fth, fph = fd / lapse, (D / Sg).sqrt() * fz[0], -fz[2] / Sg.sqrt(), om / lapse * fd + fz[1] / varpi
    Aw = p0 * fr - p1 * ft + a * s2 * (p1 * fph - p3 * fr)
    Bw = ((r * r + a * a) * (p3 * fth - p2 * fph) - a * (p0 * fth - p2 * ft)) * sth
    k1, k2 = Aw * r - Bw * a * cth, -(Aw * a * cth + Bw * r)
    mu, be = -(S["al"][j] + a * S["st"]), S["be"][j]
    y, x = -(be * k2 - mu * k1), be * k1 + mu * k2
    h = x * x + y * y
    return g, cosb, 2 * x * y / h, (x * x - y * y) / h


def _cap(I, Q, V):
    p = torch.sqrt(torch.clamp(Q * Q + V * V, min=1e-300) / torch.clamp(I * I, min=1e-300))
    return torch.where(p > 0.99, 0.99 / p, torch.ones_like(p))


class _Take(torch.autograd.Function):
    """v[..., i] for ascending i, whose derivative sums runs of equal i."""

    @staticmethod
    def forward(ctx, v, i):
        ctx.save_for_backward(i)
        ctx.n = v.numel()
        return v[i]

    @staticmethod
    def backward(ctx, g):
        (i,) = ctx.saved_tensors
        ends = torch.searchsorted(i, torch.arange(ctx.n + 1, device=i.device))
        run = torch.cat([torch.zeros_like(g[:1]), g.cumsum(0)])
        return run[ends[1:]] - run[ends[:-1]], None


def _pairs_of(c, i):
    """The splats' constants at every pair (splats in ascending order)."""
    def take(v):
        return _Take.apply(v, i) if v.requires_grad else v[i]

    return {k: [take(x) for x in v] if v.dim() == 2 else take(v) for k, v in c.items() if torch.is_tensor(v) and k not in ("kt", "knots", "reach")}


def _coefficients(S, consts, pairs, nus, count):
    """The summed screen-basis coefficients (active samples, frequencies, 11) and which are active."""
    out = torch.zeros(count, len(nus), 11, device=S["r"].device, dtype=torch.float64)
    for c, (j, i, row) in zip(consts, pairs):
        if not j.numel():
            continue
        own = _pairs_of(c, i)
        q = _exponent(c, i, S["time"][j], S["x"][j], S["y"][j], S["z"][j], own)
        g, cosb, s2c, c2c = _frame(S, j, own["u"], own["bh"])
        ct = torch.clamp(cosb, -1, 1)
        sb = torch.clamp((1 - ct) * (1 + ct), min=1e-30).sqrt()
        cols = []
        for nu in nus:
            nf = nu / g
            jI, jQ, jV, aI, aQ, aV, rQ, rV = _FITS[c["kind"]](own, own["ne"] * torch.exp(-q), own["B"], nf, sb, ct)
            fe, fa, nh = _cap(jI, jQ, jV), _cap(aI, aQ, aV), nf / NU0
            jQ, aQ, rQ = jQ * fe / nh ** 2, aQ * fa * nh, rQ * nh
            cols.append(torch.stack([jI / nh ** 2, jQ * c2c, jQ * s2c, jV * fe / nh ** 2, nh * aI, aQ * c2c, aQ * s2c, aV * fa * nh,
                                     rQ * c2c, rQ * s2c, nh * rV], -1))
        out = out.index_add(0, row, torch.stack(cols, 1))
    return out


def _steps(C, D):
    """O and E of the exact Stokes steps: one exponential of the matrix with the emission as a fifth column."""
    j, (aI, aQ, aU, aV), (rQ, rU, rV) = C[..., :4], C[..., 4:8].unbind(-1), C[..., 8:].unbind(-1)
    big = torch.clamp(j.detach().abs().amax(-1, keepdim=True), min=1e-300)
    zero = torch.zeros_like(aI)
    K = torch.stack([aI, aQ, aU, aV, aQ, aI, rV, -rU, aU, -rV, aI, rQ, aV, rU, -rQ, aI], -1).reshape(*aI.shape, 4, 4)
    col = (j / big)[..., None] / D.detach()[..., None, None]
    M = torch.cat([torch.cat([-K, col], -1), torch.stack([zero] * 5, -1)[..., None, :]], -2) * D[..., None, None]
    flat = M.reshape(-1, 5, 5)
    ex = torch.cat([torch.linalg.matrix_exp(m) for m in flat.split(400000)]) if flat.shape[0] else flat
    ex = ex.reshape(M.shape)
    return ex[..., :4, :4], ex[..., :4, 4] * big * D.detach()[..., None]


def _batches(case, scene, dev, frame):
    """The samples near splats, rays a batch at a time: sample data, (sample, splat) pairs, active rows."""
    al, be = (torch.as_tensor(v, device=dev) for v in _pixels(case))
    a, tho = case["spin"], math.radians(case["inc"])
    step = max(64, int(1.2e6) // case["samples"])
    with torch.no_grad():
        consts = [_constants(kind, torch.as_tensor(p, device=dev), scene) for kind, p in scene.get("sets", [])]
    for lo in range(0, al.numel(), step):
        with torch.no_grad():
            R = _Rays(al[lo:lo + step], be[lo:lo + step], a, tho)
            n = torch.full_like(R.al, float(case["samples"]))
            if _uneven(case):
                n = torch.clamp(64 * torch.ceil(768.0 * R.total / 64), _uneven(case)[1], case["samples"])
            m = R.march(n, case["samples"])
            temp = math.sqrt(1 - a * a)
            ph = m["phi"] + a / (2 * temp) * torch.log(((m["r"] - R.rp) / (m["r"] - R.rm)).abs()) - torch.atan2(torch.full_like(m["r"], a), m["r"])
            rho = m["r"] * (1 - m["cth"] ** 2).sqrt()
            pos = dict(x=rho * ph.cos(), y=rho * ph.sin(), z=m["r"] * m["cth"])
            keep = m["ok"] & (m["r"] < 1e3)
            k, ray = keep.nonzero(as_tuple=True)
            S = {q: v[k, ray] for q, v in dict(m, **pos).items() if q not in ("dtau", "ok", "phi")}
            S.update(a=a, st=math.sin(tho), lam=R.lam[ray], eta=R.eta[ray], al=R.al[ray], be=R.be[ray], ray=ray, k=k)
            S["time"] = scene["times"][frame] - S["t"]
            S["len"] = (S["r"] ** 2 + (a * S["cth"]) ** 2) * m["dtau"][ray]
            pairs = []
            rr, zz = (S["x"] ** 2 + S["y"] ** 2).sqrt(), S["z"]
            for c in consts:
                js, is_ = [], []
                for i in range(c["ne"].numel()):
                    if c["kind"] == "knot":
                        near = torch.arange(rr.numel(), device=dev)
                    else:
                        near = ((rr - torch.hypot(c["pos"][0, i], c["pos"][1, i])) ** 2 + (zz - c["pos"][2, i]) ** 2 <= c["reach"][i]).nonzero()[:, 0]
                    ii = torch.full_like(near, i)
                    one = {k: [x[i] for x in v] if v.dim() == 2 else v[i] for k, v in c.items() if torch.is_tensor(v) and k not in ("kt", "knots")}
                    q = _exponent(c, ii, S["time"][near], S["x"][near], S["y"][near], S["z"][near], one)
                    hit = q < 13.815510557964274
                    js.append(near[hit]); is_.append(ii[hit])
                pairs.append((torch.cat(js), torch.cat(is_)))
            used = torch.zeros(rr.numel(), dtype=torch.bool, device=dev)
            for j, _ in pairs:
                used[j] = True
            act = used.nonzero()[:, 0]
            row = torch.cumsum(used, 0) - 1
            pairs = [(j, i, row[j]) for j, i in pairs]
            # the order of a ray's active samples, and their place in the padded (rank, ray) table
            order = torch.argsort(S["ray"][act] * (case["samples"] + 1) + S["k"][act])
            rays = S["ray"][act][order]
            per = torch.bincount(rays, minlength=R.al.numel())
            rank = torch.empty_like(order)
            rank[order] = torch.arange(order.numel(), device=dev) - (torch.cumsum(per, 0) - per)[rays]
        yield dict(lo=lo, rays=R.al.numel(), S=S, pairs=pairs, act=act, rank=rank, depth=int(per.max()) if per.numel() else 0)


def _compose(b, O, E, keep=True):
    """The Stokes vectors of a batch's rays, back to front, and (`keep`) the tail behind every active sample."""
    ray, F = b["S"]["ray"][b["act"]], O.shape[1]
    T = torch.zeros(b["rays"], F, 4, device=O.device, dtype=torch.float64)
    tails = torch.zeros_like(E)
    at = torch.full((b["depth"], b["rays"]), -1, dtype=torch.long, device=O.device)
    at[b["rank"], ray] = torch.arange(ray.numel(), device=O.device)
    for d in range(b["depth"] - 1, -1, -1):
        m = at[d]
        live = (m >= 0)[:, None, None]
        idx = torch.clamp(m, min=0)
        if keep:
            tails[m[m >= 0]] = T[m >= 0]
        T = torch.where(live, E[idx] + (O[idx] @ T[..., None])[..., 0], T)
    return T, tails, at


def _image(case, scene, dev, dirs=None, kept=None):
    """(1 + len(dirs), frequencies, frames, pixels, 4): the image and its derivatives along `dirs`; the batches go to `kept`."""
    nus = [float(v) for v in scene["nus"]]
    n = case["na"] * case["nb"]
    nd = 0 if dirs is None else len(dirs)
    out = torch.zeros(1 + nd, len(nus), case["frames"], n, 4, device=dev, dtype=torch.float64)
    cube = torch.tensor([(v / NU0) ** 3 for v in nus], device=dev)[:, None]
    D0 = torch.tensor([scene["L"] / (v / NU0) for v in nus], device=dev)
    base = [torch.as_tensor(p, device=dev) for _, p in scene["sets"]]
    for f in range(case["frames"]):
        for b in _batches(case, scene, dev, f):
            if not b["act"].numel():
                continue
            if kept is not None:
                kept.append((f, b))
            sl = slice(b["lo"], b["lo"] + b["rays"])
            dlen = b["S"]["len"][b["act"]][:, None] * D0

            def stokes(ps):
                consts = [_constants(kind, p, scene) for (kind, _), p in zip(scene["sets"], ps)]
                O, E = _steps(_coefficients(b["S"], consts, b["pairs"], nus, b["act"].numel()), dlen)
                return (_compose(b, O, E, keep=False)[0] * cube).transpose(0, 1)

            with torch.no_grad():
                if not nd:
                    out[0, :, f, sl] = stokes(base)
            for d in range(nd):
                with torch.no_grad(), torch.autograd.forward_ad.dual_level():
                    T = stokes([torch.autograd.forward_ad.make_dual(base[0], torch.as_tensor(dirs[d], device=dev))])
                    v = torch.autograd.forward_ad.unpack_dual(T)
                    out[0, :, f, sl], out[1 + d, :, f, sl] = v.primal, v.tangent
    return out


def _gradient(scene, dev, seeds, kept):
    """d(sum seeds image) / d(parameters), (21, splats), from the image's batches."""
    nus = [float(v) for v in scene["nus"]]
    cube = torch.tensor([(v / NU0) ** 3 for v in nus], device=dev)[:, None]
    D0 = torch.tensor([scene["L"] / (v / NU0) for v in nus], device=dev)
    p = torch.as_tensor(scene["p"], device=dev).clone().requires_grad_(True)
    total = torch.zeros_like(p)
    for f, b in kept:
        C = _coefficients(b["S"], [_constants("thermal", p, scene)], b["pairs"], nus, b["act"].numel())
        dlen = b["S"]["len"][b["act"]][:, None] * D0
        Cd = C.detach()
        with torch.no_grad():
            O, E = _steps(Cd, dlen)
            _, tails, at = _compose(b, O, E)
            w = (seeds[:, f, b["lo"]:b["lo"] + b["rays"]].transpose(0, 1) * cube).clone()
            W = torch.zeros_like(E)
            for d in range(b["depth"]):
                live, idx = at[d] >= 0, torch.clamp(at[d], min=0)
                W[idx[live]] = w[live]
                w = torch.where(live[:, None, None], (O[idx].transpose(-1, -2) @ w[..., None])[..., 0], w)
        bar = torch.empty_like(Cd)
        for q in range(0, Cd.shape[0], 200000):
            Cq = Cd[q:q + 200000].clone().requires_grad_(True)
            O, E = _steps(Cq, dlen[q:q + 200000])
            l = (W[q:q + 200000] * (E + (O @ tails[q:q + 200000][..., None])[..., 0])).sum()
            bar[q:q + 200000] = torch.autograd.grad(l, Cq)[0]
        total += torch.autograd.grad(C, p, bar)[0]
    return total


def exact(case, seed):
    """What `run` returns for these inputs in 64-bit torch."""
    scene, op = _scene(case, seed), case["op"]
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    if op in ("thin", "refit"):
        p = torch.as_tensor(scene["p"], device=dev)
        n = p.shape[1]
        out = torch.zeros(case["na"] * case["nb"], device=dev, dtype=torch.float64)
        q, full = torch.zeros(21, n, dtype=torch.float64, device=dev), dict(scene, sets=[])
        q[:12], q[20] = p[:12], p[13]
        c = _constants("thermal", q, scene)
        for b in _batches(case, full, dev, 0):
            S, j = b["S"], torch.zeros_like(b["S"]["r"])
            for i in range(n):
                e = _exponent(c, torch.full_like(S["k"], i), S["time"], S["x"], S["y"], S["z"])
                j = j + torch.exp(p[12, i] - e)
            # seen by the ZAMO: fluid at rest, the field's direction does not enter
            rest = [torch.zeros_like(j)] * 3
            g = _frame(S, torch.arange(j.numel(), device=dev), rest, [torch.ones_like(j), rest[0], rest[0]])[0]
            out[b["lo"]:b["lo"] + b["rays"]].index_add_(0, S["ray"], g * g * j * S["len"])
        return out.reshape(case["nb"], case["na"]).t()
    if op in ("render", "movie"):
        return _image(case, scene, dev)[0]
    if op == "jvp":
        return _image(case, scene, dev, scene["dirs"])[1:].cpu().numpy()
    kept = []
    img = _image(case, scene, dev, kept=kept)[0]
    if op == "grad":
        r = (img - torch.as_tensor(scene["data"], device=dev)) / scene["sigma"]
        return float((r * r).sum()), _gradient(scene, dev, 2 * r / scene["sigma"], kept).cpu().numpy()
    # the sky: l to the east (-alpha), m to the north, pixel centres `psize` apart about the screen's centre
    i = np.arange(case["na"] * case["nb"])
    x, y = (case["na"] - 1) / 2 - i % case["na"], i // case["na"] - (case["nb"] - 1) / 2
    img = img[0, 0]
    chi = torch.zeros((), device=dev, dtype=torch.float64)
    l, m = (torch.as_tensor(v, device=dev) for v in (x * scene["psize"], y * scene["psize"]))
    u, v = (torch.as_tensor(scene[q], device=dev) for q in ("u", "v"))
    seed_ = torch.zeros_like(img)
    for q in range(0, u.numel(), 256):
        E = torch.exp(2j * math.pi * (u[q:q + 256, None] * l + v[q:q + 256, None] * m))
        V = scene["scale"] * (E @ img.to(torch.complex128))
        r = (V - torch.as_tensor(scene["vis"][q:q + 256], device=dev)) / torch.as_tensor(scene["vsigma"][q:q + 256], device=dev)
        chi = chi + (r.abs() ** 2).sum()
        wts = 2 * r / torch.as_tensor(scene["vsigma"][q:q + 256], device=dev)
        seed_ += scene["scale"] * (E.conj().t() @ wts).real
    return float(chi), _gradient(scene, dev, seed_[None, None], kept).cpu().numpy()
