"""Performance cases of irs_b200: what a user of the package runs, through its public classes.

Each case is one pass of one object: an IPM or IRS map, a batch of maps, an
adaptive map, the critical curves of a star field, or a caustic-crossing map.
`prepare` makes the object a program keeps (with its star field, when the
program holds one), `run` is the call it makes for a result.

Lens settings, mass functions and map sizes are those of the repository's own
configurations (bench.py, tests/cases.py, irs_b200/batch.py); `draw` spreads
over the sizes, shapes, types and options between and around them.

A map holds fixed-point sums that do not depend on the order of work, so equal
arithmetic gives equal bits; the tolerances below are what another
evaluation of the same lens at the same precision would show.
"""
import math

import numpy as np
import torch

SALPETER = -2.35
MASS = {"equal": (1.0, 1.0), "salpeter": (0.08, 1.0), "kroupa": (0.01, 1.5)}
FIELD_SCALE = 1.45  # radius of a star field held by the program, in units of the shooting region's
FIELD_CHECK = 1.2   # safety_scale of an object that gets such a field (its realised moments scatter)


def listed():
    plain = dict(kappa=0.45, shear=0.40, kappa_star=0.225, theta=2.31, mass="salpeter", rays=1, double=False,
                 rect=False, approx=True, parities=False, hist=True, given=True, loss=0.001, order=0)
    kroupa = dict(plain, kappa=0.7, shear=0.2, kappa_star=0.63, theta=1.0, mass="kroupa", rect=True, given=False)
    equal = dict(plain, kappa=0.4, shear=0.3, kappa_star=0.4, theta=1.0, mass="equal", loss=0.01, rays=100,
                 given=False)
    return [
        # a first look at a lens, or one of many small maps in a loop: launches, copies and host work count
        dict(plain, name="ipm_128", kind="ipm", n1=128, n2=128, half=4.0, loss=0.01),
        # the plain map of the benchmark: the ordinary call
        dict(plain, name="ipm_2000", kind="ipm", n1=2000, n2=2000, half=25.0, order=12),
        # the double-precision library, a map that is not square
        dict(plain, name="ipm_double_1000", kind="ipm", n1=1000, n2=751, half=12.5, double=True),
        # minima and saddles kept apart, rectangular Kroupa field, odd sizes
        dict(kroupa, name="ipm_parities_333", kind="ipm", n1=333, n2=221, half=3.33, parities=True),
        # a large map of a dense rectangular field: many stars, cells stretched over many pixels
        dict(kroupa, name="ipm_rect_4096", kind="ipm", n1=4096, n2=4096, half=25.0, hist=False, order=16),
        # the plain ray-shooting map
        dict(equal, name="irs_500", kind="irs", n1=500, n2=500, half=10.0, order=8),
        # ray shooting in double precision with parities
        dict(equal, name="irs_double_301", kind="irs", n1=301, n2=257, half=5.0, double=True, parities=True, rays=64),
        # many lenses at once (a light-curve or parameter study)
        dict(name="batch_24", kind="batch", count=24, n1=1024, half=12.0),
        # learned subdivision of one map
        dict(name="adaptive_1024", kind="adaptive", kappa=0.6, shear=0.3, smooth=0.3, n1=1024, n2=1024, half=7.5),
        # critical curves and caustics, the default field size and a larger one
        dict(name="ccf_137", kind="ccf", stars=137, phi=100, branches=1, scales=False),
        dict(name="ccf_1000", kind="ccf", stars=1000, phi=100, branches=1, scales=True),
        # caustic crossings of such a field, default map size
        dict(name="ncc_1000", kind="ncc", curves=2000, points=101, n1=1000, n2=1000, over=2),
    ]


def draw(rng):
    """One more case: the kinds as often as they are listed, sizes over the same ranges."""
    while True:
        c = _draw(rng)
        if c["kind"] not in ("ipm", "irs") or (_points(c) < 8e7 and 20 < _stars(c) < 2e5):
            return c


def _draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["ipm"] * 5 + ["irs"] * 2 + ["batch", "adaptive", "ccf", "ccf", "ncc"])
    if kind == "ccf":
        return dict(kind=kind, stars=size(20, 1000), phi=2 * rng.choice([4, 6, 12]) * rng.randint(2, 8),
                    branches=rng.choice([1, 1, 2]), scales=rng.random() < 0.5)
    if kind == "ncc":
        n = size(100, 1000)
        return dict(kind=kind, curves=size(50, 2000), points=rng.choice([51, 101, 201]), n1=n,
                    n2=int(n * rng.uniform(0.6, 1.6)) + 1, over=rng.choice([0, 1, 2]))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(2, 16), n1=size(128, 1024), half=12.0)
    if kind == "adaptive":
        n = size(256, 1024)
        return dict(kind=kind, kappa=rng.uniform(0.4, 0.65), shear=rng.uniform(0.1, 0.3), smooth=rng.uniform(0.2, 0.6),
                    n1=n, n2=int(n * rng.uniform(0.7, 1.0)), half=n * 7.5 / 1024)
    while True:
        kappa, shear = rng.uniform(0.1, 0.9), rng.uniform(0.0, 0.8)
        if abs(1 - kappa - shear) > 0.1 and abs(1 - kappa + shear) > 0.1:
            break
    n1 = size(64, 2000) if kind == "ipm" else size(64, 600)
    n2 = max(40, int(n1 * rng.uniform(0.6, 1.5)))
    rect = rng.random() < 0.35
    mass = rng.choice(["equal", "salpeter", "kroupa"])
    theta = {"equal": 1.0, "salpeter": 2.31, "kroupa": 1.5}[mass]
    return dict(kind=kind, kappa=kappa, shear=shear, kappa_star=kappa * rng.uniform(0.2, 1.0), theta=theta, mass=mass,
                rays=1 if kind == "ipm" else rng.choice([16, 36, 100]), double=rng.random() < 0.3, rect=rect,
                approx=not (rect and n1 < 300 and rng.random() < 0.3), parities=rng.random() < 0.3,
                hist=rng.random() < 0.6, given=not rect and mass != "kroupa" and rng.random() < 0.5,
                loss=rng.choice([0.001, 0.01]), order=0, n1=n1, n2=n2, half=n1 * rng.uniform(0.008, 0.03))


def prepare(case, seed):
    import irs_b200
    kind, seed = case["kind"], int(seed)
    if kind in ("ipm", "irs"):
        cls = irs_b200.IPM if kind == "ipm" else irs_b200.IRS
        lo, hi = MASS[case["mass"]]
        m = cls(kappa_tot=case["kappa"], shear=case["shear"], kappa_star=case["kappa_star"], theta_star=case["theta"],
                mass_function=case["mass"], m_lower=lo, m_upper=hi, light_loss=case["loss"], rectangular=case["rect"],
                approx=case["approx"], half_length_y1=case["half"], half_length_y2=_half2(case),
                num_pixels_y1=case["n1"], num_pixels_y2=case["n2"], num_rays_y=case["rays"],
                random_seed=1 + seed % 1000000, write_parities=case["parities"], write_histograms=case["hist"],
                is_double=case["double"], expansion_order=case["order"])
        if case["given"]:
            stars, radius = _field(case, seed)
            m.safety_scale = FIELD_CHECK
            m.set_stars(stars, rectangular=False, corner=(radius, 0.0), theta_star=case["theta"])
        return {"kind": kind, "m": m}
    if kind == "batch":
        from irs_b200.batch import random_realizations
        reals, _ = random_realizations(case["count"], seed=1000, first_seed=1000 + 300 * (seed % 1000000),
                                       num_pixels=case["n1"], half_length=case["half"])
        return {"kind": kind, "m": irs_b200.BatchIPM(reals)}
    if kind == "adaptive":
        m = irs_b200.AdaptiveIPM(kappa_tot=case["kappa"], shear=case["shear"], smooth_fraction=case["smooth"],
                                 mass_function="salpeter", m_lower=0.08, m_upper=1.0, theta_star=1.0,
                                 half_length_y1=case["half"], half_length_y2=case["half"] * case["n2"] / case["n1"],
                                 num_pixels_y1=case["n1"], num_pixels_y2=case["n2"], random_seed=1 + seed % 1000000,
                                 write_histograms=0)
        return {"kind": kind, "m": m}
    if kind == "ccf":
        m = irs_b200.CCF(kappa_tot=0.3, shear=0.3, kappa_star=0.27, theta_star=1.0, mass_function="equal",
                         num_stars=case["stars"], num_phi=case["phi"], num_branches=case["branches"],
                         random_seed=1 + seed % 1000000, write_length_scales=case["scales"])
        return {"kind": kind, "m": m}
    caustics, half = _caustics(case, seed)
    m = irs_b200.NCC(half_length_y1=half, half_length_y2=half, num_pixels_y1=case["n1"], num_pixels_y2=case["n2"],
                     over_sample=case["over"])
    m.set_caustics(caustics)
    return {"kind": kind, "m": m}


def run(state):
    kind, m = state["kind"], state["m"]
    m.run()
    if kind in ("ipm", "irs"):
        out = {"map": m.magnifications, "stars": m.stars}
        if m.magnifications_minima is not None:
            out["minima"], out["saddles"] = m.magnifications_minima, m.magnifications_saddles
        return out
    if kind == "batch":
        return {"maps": m.maps}
    if kind == "adaptive":
        return {"map": m.magnifications, "levels": m.levels()}
    if kind == "ccf":
        out = {"curves": m.critical_curves, "caustics": m.caustics, "stars": m.stars}
        if m.mu_length_scales is not None:
            out["scales"] = m.mu_length_scales
        return out
    return {"crossings": m.num_caustic_crossings}


def work(case):
    """Bytes: stars read and maps written. Operations: per lattice point the
    lens equation (11 per near-field star, about 16 of them, 8 per expansion
    order, about 12, 30 for the rest), per cell whose image is on the map 150
    for each of its two triangles; CCF: 10 per reciprocal, every root against
    every star and other root, 4 updates a step; NCC: the fine map's sums."""
    kind = case["kind"]
    if kind in ("ipm", "irs"):
        pix, es = case["n1"] * case["n2"], 8 if case["double"] else 4
        pts = _points(case)
        flops = pts * 302.0
        if kind == "ipm":
            flops += pix * abs(_mu(case["kappa"], case["shear"])) * 300.0
        maps = (3 if case["parities"] else 1) * pix * (4 if kind == "irs" else es)
        return {"bytes": _stars(case) * 3 * es + maps, "flops": flops}
    if kind == "batch":
        from irs_b200.batch import random_realizations
        reals, _ = random_realizations(case["count"], num_pixels=case["n1"], half_length=case["half"])
        flops = 0.0
        for r in reals:
            c = dict(kappa=r["kappa_tot"], shear=r["shear"], kappa_star=r["kappa_tot"] * (1 - r["smooth_fraction"]),
                     theta=1.0, mass=r["mass_function"], n1=case["n1"], n2=case["n1"], half=case["half"], rays=1,
                     loss=0.001, rect=False, given=False)
            flops += _points(c) * 302.0 + case["n1"] ** 2 * abs(_mu(c["kappa"], c["shear"])) * 300.0
        return {"bytes": case["count"] * case["n1"] ** 2 * 4.0, "flops": flops}
    if kind == "adaptive":
        pix = case["n1"] * case["n2"]
        cells = pix * abs(_mu(case["kappa"], case["shear"])) * 64.0  # level 8 where the image is on the map
        return {"bytes": pix * 4.0, "flops": cells * (302.0 + 300.0)}
    if kind == "ccf":
        n, rows = case["stars"], case["phi"] + case["branches"]
        return {"bytes": 2.0 * n * rows * 16 * 2, "flops": 2.0 * n * rows * 4 * 3 * n * 10}
    fine = case["n1"] * case["n2"] * 4.0 ** case["over"]
    return {"bytes": case["curves"] * case["points"] * 16.0 + case["n1"] * case["n2"] * 4.0, "flops": 2 * fine}


def tolerance(case):
    """Counts and the adaptive levels are whole numbers. Critical curves are
    followed to the root's last digits; what a different order of the FP64
    sums leaves is far below 1e-6 of the field. Maps in single precision:
    about four times what the FP32 and FP64 forms of the lens equation differ
    by on one field (total maps 4e-6 to 1.2e-4, minima and saddles up to
    4e-4; single pixels on a caustic a few per cent)."""
    kind = case["kind"]
    if kind in ("irs", "ncc"):
        return "exact"
    if kind == "ccf":
        return {"rel": 1e-6, "max": 1e-3}
    if kind == "adaptive":
        return {"rel": 5e-4, "max": 0.15, "differ": 1e-3}
    if kind == "ipm" and case["double"]:
        return {"rel": 1e-8, "max": 1e-4}
    if kind == "ipm" and not case["parities"]:
        return {"rel": 5e-4, "max": 0.12}
    return {"rel": 1.6e-3, "max": 0.15}


def exact(case, seed):
    """The map in 64 bits: every star summed directly, every triangle cut by
    every pixel it touches. Circular fields held by the program (a field that
    the library draws, and the series of the rectangular sheet, have no plain
    form here), up to a size that takes seconds."""
    if case["kind"] != "ipm" or not case["given"] or case["rect"] or case["parities"]:
        return None
    if _points(case) * _stars(case) > 6e10:
        return None
    return {"map": _exact_map(case, int(seed)), "stars": None}


# ---------------------------------------------------------------- sizes


def _half2(c):
    return c["half"] * c["n2"] / c["n1"]


def _mu(kappa, shear):
    return 1.0 / ((1 - kappa) ** 2 - shear ** 2)


def _moments(mass):
    """<m> and <m^2> of a mass function (Kroupa: slopes -0.3, -1.3, -2.3)."""
    lo, hi = MASS[mass]
    if mass == "equal":
        return 1.0, 1.0
    if mass == "salpeter":
        parts = [(lo, hi, SALPETER, 1.0)]
    else:
        parts, c = [], 1.0
        for a, b, s, nxt in ((0.01, 0.08, -0.3, -1.3), (0.08, 0.5, -1.3, -2.3), (0.5, 1.5, -2.3, None)):
            parts.append((a, b, s, c))
            if nxt is not None:
                c *= b ** (s - nxt)

    def moment(k):
        return sum(c * (b ** (s + k + 1) - a ** (s + k + 1)) / (s + k + 1) for a, b, s, c in parts)
    return moment(1) / moment(0), moment(2) / moment(0)


def _region(c):
    """Half lengths of the shooting region and lattice points along each axis."""
    m1, m2 = _moments(c["mass"])
    t = c["theta"] * math.sqrt(c["kappa_star"] * m2 / (m1 * c["loss"]))
    pix = 2 * c["half"] / c["n1"]
    hx = (c["half"] + t) / abs(1 - c["kappa"] + c["shear"])
    hy = (_half2(c) + t) / abs(1 - c["kappa"] - c["shear"])
    per = math.sqrt(c["rays"]) / pix
    return hx, hy, 2 * hx * per, 2 * hy * per


def _points(c):
    _, _, nx, ny = _region(c)
    return nx * ny


def _stars(c):
    hx, hy, _, _ = _region(c)
    m1, _ = _moments(c["mass"])
    if c["rect"]:
        return 4 * 1.37 ** 2 * hx * hy * c["kappa_star"] / (math.pi * c["theta"] ** 2 * m1)
    s = FIELD_SCALE if c["given"] else 1.37
    return s * s * (hx * hx + hy * hy) * c["kappa_star"] / (c["theta"] ** 2 * m1)


# ---------------------------------------------------------------- inputs


def _field(c, seed):
    """A circular field (n, 3) in the library's type, and its radius."""
    n = int(math.ceil(_stars(c)))
    m1, _ = _moments(c["mass"])
    radius = math.sqrt(c["theta"] ** 2 * n * m1 / c["kappa_star"])
    rng = np.random.default_rng(seed)
    r, a, u = radius * np.sqrt(rng.random(n)), 2 * np.pi * rng.random(n), rng.random(n)
    lo, hi = MASS[c["mass"]]
    s = SALPETER + 1
    m = np.ones(n) if c["mass"] == "equal" else (lo ** s + u * (hi ** s - lo ** s)) ** (1 / s)
    stars = np.stack([r * np.cos(a), r * np.sin(a), m], 1)
    return stars.astype(np.float64 if c["double"] else np.float32), radius


def _caustics(c, seed):
    """Closed cusped curves run through clockwise, as rows of points, and the
    half length of a map that holds most of them."""
    rng = np.random.default_rng(seed)
    k, n = c["curves"], c["points"]
    half = 0.5 * math.sqrt(k)
    ctr = rng.uniform(-1.2 * half, 1.2 * half, (k, 2, 1))
    size = np.exp(rng.normal(-0.5, 0.7, (k, 2, 1)))
    t = -np.linspace(0.0, 2 * np.pi, n)[None, :] + rng.uniform(0, 2 * np.pi, (k, 1))
    z = (ctr[:, 0] + size[:, 0] * np.cos(t) ** 3) + 1j * (ctr[:, 1] + size[:, 1] * np.sin(t) ** 3)
    z[:, -1] = z[:, 0]
    return z, half


# ---------------------------------------------------------------- 64-bit map


def _exact_map(c, seed):
    stars, radius = _field(c, seed)
    F = np.float64 if c["double"] else np.float32  # the inputs and the lattice are in the library's type
    m = stars[:, 2]
    theta, loss, kappa, shear = F(c["theta"]), F(c["loss"]), F(c["kappa"]), F(c["shear"])
    n1, n2, h1, h2, rad = c["n1"], c["n2"], F(c["half"]), F(_half2(c)), F(radius)
    mt, mt2 = float(m.astype(np.float64).sum()), float((m * m).astype(np.float64).sum())
    kstar = F(mt * float(theta) * float(theta) / float(rad * rad))
    mean, mean2 = F(mt / len(m)), F(mt2 / len(m))
    per_area = F(1.0 * c["rays"] * n1 * n2 / float(2 * h1 * 2 * h2))
    div = 2 * np.sqrt(per_area)
    rx, ry = np.sqrt(h1 / h2 * F(n2) / F(n1)) / div, np.sqrt(h2 / h1 * F(n1) / F(n2)) / div
    t = theta * np.sqrt(kstar * mean2 / (mean * loss))
    kx = int((h1 + t) / np.abs(1 - kappa + shear) / (2 * rx)) + 1
    ky = int((h2 + t) / np.abs(1 - kappa - shear) / (2 * ry)) + 1
    lx, ly = 2 * rx * F(kx), 2 * ry * F(ky)
    factor = float(2 * rx * ry * F(n1) * F(n2) / (2 * h1 * 2 * h2))

    dev, f64 = torch.device("cuda" if torch.cuda.is_available() else "cpu"), torch.float64
    S = torch.tensor(stars.astype(np.float64), device=dev)
    sx, sy, sm = S[:, 0], S[:, 1], S[:, 2] * float(theta) ** 2
    x = -float(lx) + 2.0 * (float(rx) * torch.arange(2 * kx + 1, dtype=f64, device=dev))
    out = torch.zeros(n1 * n2, dtype=f64, device=dev)
    k, g, ks = float(kappa), float(shear), float(kstar)

    def row_images(j):
        """Images of the corner rows j (pixel units, rows flipped): (len(j), 2 kx + 1) each."""
        y = -float(ly) + 2.0 * (float(ry) * j)
        X, Y = x.expand(len(j), -1).reshape(-1), y[:, None].expand(-1, len(x)).reshape(-1)
        wx, wy = (1 - k + ks + g) * X, (1 - k + ks - g) * Y
        for a in range(0, len(sx), 4096):
            step = max(1, int(3e7 // min(4096, len(sx))))
            for b in range(0, len(X), step):
                dx, dy = X[b:b + step, None] - sx[a:a + 4096], Y[b:b + step, None] - sy[a:a + 4096]
                q = sm[a:a + 4096] / (dx * dx + dy * dy)
                wx[b:b + step] -= (q * dx).sum(1)
                wy[b:b + step] -= (q * dy).sum(1)
        px = (wx + float(h1)) * n1 / (2 * float(h1))
        py = n2 - (wy + float(h2)) * n2 / (2 * float(h2))
        return px.reshape(len(j), -1), py.reshape(len(j), -1)

    band = max(1, int(2e6 // len(x)))
    for j0 in range(0, 2 * ky, band):
        j1 = min(2 * ky, j0 + band)
        px, py = row_images(torch.arange(j0, j1 + 1, dtype=f64, device=dev))
        c0 = (px[1:, 1:], py[1:, 1:])
        c1, c2, c3 = (px[1:, :-1], py[1:, :-1]), (px[:-1, :-1], py[:-1, :-1]), (px[:-1, 1:], py[:-1, 1:])
        for tri in ((c0, c1, c2), (c2, c3, c0)):
            X, Y = (torch.stack([v[i].reshape(-1) for v in tri], 1) for i in (0, 1))
            _spread(X, Y, factor, n1, n2, out)
    return out.reshape(n2, n1).cpu().numpy()


def _spread(X, Y, factor, n1, n2, out):
    """Adds factor * |triangle within pixel| / |triangle| to every pixel; triangles as (n, 3) corners."""
    area = 0.5 * ((X[:, 1] - X[:, 0]) * (Y[:, 2] - Y[:, 0]) - (X[:, 2] - X[:, 0]) * (Y[:, 1] - Y[:, 0]))
    a0, a1 = X.amin(1).clamp(min=0).floor(), X.amax(1).clamp(max=n1 - 1).floor()
    b0, b1 = Y.amin(1).clamp(min=0).floor(), Y.amax(1).clamp(max=n2 - 1).floor()
    use = (area != 0) & (area.abs() < 1e4 * factor) & (a1 >= a0) & (b1 >= b0)
    use &= (X.amax(1) > 0) & (Y.amax(1) > 0) & (X.amin(1) < n1) & (Y.amin(1) < n2)
    X, Y, area, a0, a1, b0, b1 = (v[use] for v in (X, Y, area, a0, a1, b0, b1))
    w = (a1 - a0 + 1).long()
    count = w * (b1 - b0 + 1).long()
    ends = torch.cumsum(count, 0)
    first = 0
    while first < len(count):
        before = int(ends[first - 1]) if first else 0
        last = max(first + 1, int(torch.searchsorted(ends, before + 8_000_000, right=True)))
        sl = slice(first, last)
        t = torch.repeat_interleave(torch.arange(first, last, device=X.device), count[sl])
        i = torch.arange(len(t), device=X.device) - (ends[t] - count[t] - before)
        col, row = a0[t] + (i % w[t]), b0[t] + torch.div(i, w[t], rounding_mode="floor")
        part = torch.zeros_like(col)
        for e in range(3):
            x1, y1 = X[t, e] - col, Y[t, e] - row
            x2, y2 = X[t, (e + 1) % 3] - col, Y[t, (e + 1) % 3] - row
            dx = x2 - x1
            slope = torch.where(dx != 0, (y2 - y1) / torch.where(dx != 0, dx, 1.0), 0.0)
            xs, xe = x1.clamp(0, 1), x2.clamp(0, 1)
            ys, ye = y1 + (xs - x1) * slope, y1 + (xe - x1) * slope
            # mean over the piece of the height clamped to the pixel
            lo, hi, dy = ys.clamp(0, 1), ye.clamp(0, 1), ye - ys
            flat = dy.abs() < 1e-7
            mean = (0.5 * (lo + hi) * (hi - lo) + (ye - 1).clamp(min=0) - (ys - 1).clamp(min=0)) / torch.where(
                flat, 1.0, dy)
            part += (xe - xs) * torch.where(flat, (0.5 * (ys + ye)).clamp(0, 1), mean)
        out.index_add_(0, (row * n1 + col).long(), factor * part.abs() / area[t].abs())
        first = last
