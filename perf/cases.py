"""Timed cases of the library: the work its users have it do, one pass at a time.

Every case goes through the public Python mirror of the C ABI
(msmodel_gb300.api), which takes host arrays (scatterer positions, wave
numbers) and returns host arrays; the whole call counts.  Scatterers are drawn
uniformly from the ball of unit density, the reference's default medium.

  listed()            the cases
  draw(rng)           one more case of the same ranges
  prepare(case, seed) the media and wave numbers a program has in hand
  run(state)          one pass
  work(case)          bytes and real flops no method can do without
  exact(case, seed)   the same outputs in plain 64-bit torch / numpy
"""
import math

import numpy as np
import torch

import msmodel_gb300.api as ms

TWOPI = 2.0 * math.pi


# --------------------------------------------------------------------------- cases
def listed():
    return [
        # one dlogf, as a root finder or a user of dk_log_det_ms calls it: the reference's own test medium
        {"name": "dlogf_one_d2_n50", "kind": "dlogf", "d": 2, "nmin": 50, "nmax": 50, "media": 1, "points": 1,
         "precision": "fp64", "model": "hardsphere"},
        # tracelog_lu of one matrix the caller holds: the call the reference's map loops make per point
        {"name": "lu_one_n300", "kind": "matrix", "d": 3, "n": 300},
        # cross sections of many seeds on a grid of real k (the crsec random function)
        {"name": "amps_d3_n100", "kind": "amps", "d": 3, "n": 100, "media": 16, "points": 20, "precision": "fp64"},
        # the complex map of a small medium, both arithmetics
        {"name": "map_d3_n64_mixed", "kind": "map", "d": 3, "n": 64, "nx": 64, "ny": 64, "imk": -0.5,
         "precision": "mixed"},
        {"name": "map_d3_n64_fp64", "kind": "map", "d": 3, "n": 64, "nx": 64, "ny": 64, "imk": -0.5,
         "precision": "fp64"},
        # the complex cut of a large medium (kcut sample = 64: 198 points), both arithmetics
        {"name": "cut_d3_n1024_fp64", "kind": "cut", "d": 3, "n": 1024, "samples": 64, "precision": "fp64"},
        {"name": "cut_d3_n1024_mixed", "kind": "cut", "d": 3, "n": 1024, "samples": 98, "precision": "mixed"},
        # part of the largest complex map: d = 2, N = 2048, down to Im k = -0.3
        {"name": "map_d2_n2048_mixed", "kind": "map", "d": 2, "n": 2048, "nx": 19, "ny": 16, "imk": -0.3,
         "precision": "mixed"},
        # one sweep of the resonance search over realisations of uneven size, 32 targets each
        {"name": "dlogf_uneven_mixed", "kind": "dlogf", "d": 3, "nmin": 100, "nmax": 600, "media": 16, "points": 32,
         "precision": "mixed", "model": "maximum"},
        # the resonance search of one realisation, whole
        {"name": "roots_d3_n100_fp64", "kind": "roots", "d": 3, "n": 100, "targets": 32, "precision": "fp64"},
        # the wavefunction task: one k, one realisation, a picture
        {"name": "wave_d3_n1024_mixed", "kind": "wave", "d": 3, "n": 1024, "nx": 512, "ny": 512,
         "precision": "mixed"},
        # eigenvalues behind the mu-plane histograms
        {"name": "eig_d3_n256", "kind": "eig", "d": 3, "n": 256, "media": 64, "mtype": "msmatrix"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dlogf_one", "matrix", "amps", "map", "cut", "dlogf", "roots", "wave", "eig"])
    prec = rng.choice(["fp64", "mixed"])
    d = rng.choice([2, 3])
    if kind == "dlogf_one":
        n = _log_int(rng, 20, 300)
        return {"kind": "dlogf", "d": d, "nmin": n, "nmax": n, "media": 1, "points": rng.randint(1, 4),
                "precision": prec, "model": rng.choice(["hardsphere", "maximum"])}
    if kind == "matrix":
        return {"kind": "matrix", "d": d, "n": _log_int(rng, 40, 700)}
    if kind == "amps":
        return {"kind": "amps", "d": d, "n": _log_int(rng, 40, 400), "media": rng.randint(1, 16),
                "points": rng.randint(1, 20), "precision": prec}
    if kind == "map":
        n = _log_int(rng, 32, 400)
        cap = min(4096, int(4e10 / n ** 3)) if prec == "fp64" else min(4096, int(3e11 / n ** 3))
        nx = rng.randint(8, max(8, min(64, cap // 8)))
        return {"kind": "map", "d": d, "n": n, "nx": nx, "ny": max(2, min(64, cap // nx)),
                "imk": round(-rng.uniform(0.05, 0.5), 3), "precision": prec}
    if kind == "cut":
        n = _log_int(rng, 200, 1200 if prec == "fp64" else 1600)
        cap = max(2, int((5e10 if prec == "fp64" else 4e11) / n ** 3) // 3 - 2)
        return {"kind": "cut", "d": 3, "n": n, "samples": rng.randint(2, min(150, max(2, cap))), "precision": prec}
    if kind == "dlogf":
        lo = rng.randint(40, 200)
        return {"kind": "dlogf", "d": 3, "nmin": lo, "nmax": lo + rng.randint(50, 400), "media": rng.randint(2, 12),
                "points": rng.choice([8, 16, 32]), "precision": prec, "model": "maximum"}
    if kind == "roots":
        return {"kind": "roots", "d": 3, "n": rng.randint(40, 120), "targets": rng.choice([16, 32]),
                "precision": "fp64"}
    if kind == "wave":
        return {"kind": "wave", "d": 3, "n": _log_int(rng, 100, 1200 if prec == "mixed" else 600),
                "nx": rng.randint(100, 512), "ny": rng.randint(100, 400), "precision": prec}
    n = rng.randint(50, 280)
    return {"kind": "eig", "d": d, "n": n, "media": rng.randint(8, 100), "mtype": rng.choice(["msmatrix", "normalized"])}


# --------------------------------------------------------------------------- inputs
def _ball(rng, d, n):
    """n points uniform in the d-ball of volume n (density 1)."""
    radius = (n / (math.pi if d == 2 else 4.0 * math.pi / 3.0)) ** (1.0 / d)
    x = rng.standard_normal((n, d))
    x /= np.linalg.norm(x, axis=1, keepdims=True)
    return x * (radius * rng.random((n, 1)) ** (1.0 / d))


def _kmap(nx, ny, xmin, xmax, ymin, ymax):
    """Row-major grid of k from the top row, as kplane_args."""
    x = xmin + np.arange(nx) * (xmax - xmin) / (nx - 1)
    y = ymax + np.arange(ny) * (ymin - ymax) / (ny - 1)
    return (x[None, :] + 1j * y[:, None]).reshape(-1)


def _kcut(ns, zmin, zmax):
    """3 (ns + 2) points along a cut and its two neighbours across, as kcut samples them."""
    dz = (zmax - zmin) / (ns - 1)
    i = np.arange(-1, ns + 1)[:, None]
    return (zmin + i * dz + 1j * dz * np.array([-1.0, 0.0, 1.0])[None, :]).reshape(-1)


def _inputs(case, seed):
    """(positions of every medium, model, params, k per item, medium per item)."""
    rng = np.random.default_rng([seed, 20])
    d, kind = case["d"], case["kind"]
    model, params = "maximum", ()
    if kind == "dlogf":
        sizes = rng.integers(case["nmin"], case["nmax"] + 1, case["media"])
        pos = [_ball(rng, d, int(n)) for n in sizes]
        if case["model"] == "hardsphere":
            model, params = "hardsphere", (0.4,)
        ks = rng.uniform(0.5, 3.0, (case["media"], case["points"])) - 1j * rng.uniform(
            0.0, 1.0 if d == 3 else 0.3, (case["media"], case["points"]))
        return pos, model, params, ks.reshape(-1), np.repeat(np.arange(case["media"]), case["points"])
    media = case.get("media", 1)
    pos = [_ball(rng, d, case["n"]) for _ in range(media)]
    if kind == "map":
        ks = _kmap(case["nx"], case["ny"], 0.5, 3.0, case["imk"], 0.0)
    elif kind == "cut":
        ks = _kcut(case["samples"], 0.5 - 0.05j, 3.0 - 0.05j)
    elif kind == "amps":
        ks = np.tile(np.sort(rng.uniform(0.5, 3.0, case["points"])), media).astype(np.complex128)
        return pos, model, params, ks, np.repeat(np.arange(media), case["points"])
    elif kind == "eig":
        return pos, model, params, np.full(media, rng.uniform(0.8, 2.0) + 0j), np.arange(media)
    else:
        ks = np.array([rng.uniform(0.5, 3.0) + 0j])
    return pos, model, params, ks, np.zeros(ks.size, dtype=np.int64)


def prepare(case, seed):
    pos, model, params, ks, im = _inputs(case, seed)
    state = {"case": case, "ks": ks, "im": im.astype(np.int32),
             "media": [ms.Medium(case["d"], p.shape[0], pos=p, model=model, params=params) for p in pos]}
    if case["kind"] == "matrix":
        # the matrix is the caller's own, at a k below the real axis
        p = torch.from_numpy(pos[0]).to("cuda" if torch.cuda.is_available() else "cpu")
        state["matrix"] = _matrix(p, case["d"], complex(ks[0]) - 0.1j, model, params).cpu().numpy()
    if case["kind"] == "wave":
        r = (case["n"] / (4.0 * math.pi / 3.0)) ** (1.0 / 3.0)
        state["dom"] = (-r, r, -r, r)
    return state


# --------------------------------------------------------------------------- one pass
def run(state):
    case, media = state["case"], state["media"]
    kind = case["kind"]
    if kind == "matrix":
        value, info = ms.tracelog_lu(state["matrix"])
        return np.array([value]), info
    if kind in ("map", "cut"):
        return ms.tracelog_batch(media, state["ks"], state["im"], case["precision"])
    if kind == "dlogf":
        return ms.dk_log_det_batch(media, state["ks"], state["im"], case["precision"])
    if kind == "amps":
        sigma, amps, status = ms.amplitude_batch(media, state["ks"], state["im"], case["precision"])
        return sigma, np.concatenate(amps), status
    if kind == "roots":
        roots, _ = ms.find_eigenstates(media, (0.5, 3.0, -1.0, 0.0), case["targets"], precision=case["precision"])
        out = np.zeros(case["targets"], dtype=np.complex128)  # one place per target, the roots found first
        out[:roots[0].size] = roots[0]
        return out
    if kind == "wave":
        fun, den, psi, amps = ms.wave_function(media, state["ks"][0], case["nx"], case["ny"], state["dom"],
                                               case["precision"])
        return fun, den, psi, amps[0]
    mu, status = ms.eigvals_batch(media, state["ks"], state["im"], mtype=case["mtype"])
    return np.concatenate([np.sort_complex(m) for m in mu]), status


# --------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    kind, d = case["kind"], case["d"]
    n = case.get("n") or 0.5 * (case["nmin"] + case["nmax"])
    lu = 8.0 / 3.0 * n ** 3
    media = case.get("media", 1)
    pos = 8.0 * n * d * media
    if kind == "matrix":
        return {"bytes": 16.0 * n * n + 16, "flops": lu}
    if kind == "map":
        pts = case["nx"] * case["ny"]
        return {"bytes": pos + 32.0 * pts, "flops": lu * pts}
    if kind == "cut":
        pts = 3 * (case["samples"] + 2)
        return {"bytes": pos + 32.0 * pts, "flops": lu * pts}
    if kind == "dlogf":
        pts = case["points"] * media
        return {"bytes": pos + 32.0 * pts, "flops": (lu + 8.0 * n ** 3) * pts}
    if kind == "amps":
        pts = case["points"] * media
        return {"bytes": pos + pts * (32.0 + 16.0 * n), "flops": (lu + 8.0 * n * n) * pts}
    if kind == "roots":
        # every target needs a few dlogf at least; ten is what a converged Aberth search takes
        return {"bytes": pos + 16.0 * case["targets"], "flops": 10.0 * case["targets"] * (lu + 8.0 * n ** 3)}
    if kind == "wave":
        px = case["nx"] * case["ny"]
        return {"bytes": pos + 32.0 * px + 16.0 * n, "flops": lu + 8.0 * n * n + 30.0 * px * n}
    # Hessenberg reduction 40/3 n^3 and QR about 32 n^3 real flops
    return {"bytes": pos + 16.0 * n * media, "flops": media * (40.0 / 3.0 + 32.0) * n ** 3}


# --------------------------------------------------------------------------- 64-bit values
def _hankel(nu, z):
    """H_nu^(1)(z), nu = 0 or 1, complex z with Re z > 0: ascending series below |z| = 4.5,
    else the integral 2/Gamma(nu+1/2) int_0^inf e^{-t^2} t^{2 nu} (1 + i t^2/(2z))^{nu-1/2} dt
    by the trapezoidal rule (the integrand is even and entire enough: error below 1e-16)."""
    out = torch.empty_like(z)
    small = z.abs() < 4.5
    zs = z[small]
    if zs.numel():
        q = -0.25 * zs * zs
        term = torch.ones_like(zs) if nu == 0 else 0.5 * zs
        jsum, ysum = torch.zeros_like(zs), torch.zeros_like(zs)
        psi1 = -0.5772156649015328606
        psi2 = psi1 if nu == 0 else psi1 + 1.0
        for k in range(40):
            jsum = jsum + term
            ysum = ysum + (psi1 + psi2) * term
            psi1 += 1.0 / (k + 1)
            psi2 += 1.0 / (k + 1 + nu)
            term = term * q / ((k + 1) * (k + 1 + nu))
        y = (2.0 / math.pi) * torch.log(0.5 * zs) * jsum - ysum / math.pi
        if nu == 1:
            y = y - 2.0 / (math.pi * zs)
        out[small] = torch.complex(jsum.real - y.imag, jsum.imag + y.real)
    zl = z[~small]
    if zl.numel():
        h, acc = 0.18, torch.zeros_like(zl)
        w = 0.5j / zl
        for j in range(36):
            t = j * h
            f = math.exp(-t * t) * (0.5 if j == 0 else 1.0) * (t * t if nu else 1.0)
            root = torch.sqrt(1.0 + w * (t * t))
            acc = acc + f * (root if nu else 1.0 / root)
        pre = torch.sqrt(2.0 / (math.pi * zl)) * torch.exp(1j * (zl - nu * math.pi / 2 - math.pi / 4))
        out[~small] = pre * acc * (2.0 * h / math.gamma(nu + 0.5))
    return out


def _green(r, d, k):
    if d == 3:
        return -torch.exp(1j * k * r) / (4.0 * math.pi * r)
    return -0.25j * _hankel(0, k * r)


def _invf(d, k, model, params):
    i0 = 0.25 if d == 2 else k / (4.0 * math.pi)
    if model == "maximum":
        return 1j * i0
    a = torch.tensor([params[0]], dtype=torch.complex128)
    if d == 3:
        ka = k * params[0]
        g = -np.exp(1j * ka) / (4.0 * math.pi * params[0])
        return -i0 * g / (np.sin(ka) / (4.0 * math.pi * params[0]))
    h = complex(_hankel(0, k * a)[0])
    j = complex((0.5 * (_hankel(0, k * a) + torch.conj(_hankel(0, torch.conj(k * a)))))[0])
    return -i0 * (-0.25j * h) / (0.25 * j)


def _distances(pos):
    """Pair distances summed coordinate by coordinate; ones on the diagonal."""
    r2 = sum((pos[:, None, c] - pos[None, :, c]) ** 2 for c in range(pos.shape[1]))
    return torch.sqrt(r2 + torch.eye(pos.shape[0], dtype=r2.dtype, device=r2.device))


def _matrix(pos, d, k, model, params, r=None):
    r = _distances(pos) if r is None else r
    m = -_green(r.to(torch.complex128) if d == 2 else r, d, k)
    m.fill_diagonal_(complex(_invf(d, k, model, params)))
    return m


def _dk_matrix(pos, d, k, model, params, r):
    if d == 3:
        m = 1j * torch.exp(1j * k * r) / (4.0 * math.pi)
    else:
        m = -0.25j * r * _hankel(1, k * r.to(torch.complex128))
    h = 1e-4  # the diagonal is defined as this central difference
    m.fill_diagonal_(complex((_invf(d, k + h, model, params) - _invf(d, k - h, model, params)) / (2 * h)))
    return m


def _lndet(m):
    """ln det / n on the branch of the LU's diagonal: sum of logs and arguments, pi for an odd permutation."""
    lu, piv = torch.linalg.lu_factor(m)
    u = torch.diagonal(lu)
    n = u.numel()
    odd = int((piv.cpu() != torch.arange(1, n + 1)).sum()) % 2
    return complex(float(u.abs().log().sum()), float(u.angle().sum()) + (math.pi if odd else 0.0)) / n


def exact(case, seed):
    kind, d = case["kind"], case["d"]
    if kind == "roots" or work(case)["flops"] > 1.5e12 and kind != "wave":
        return None  # a search has no closed value; the largest maps take minutes
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    pos, model, params, ks, im = _inputs(case, seed)
    p = [torch.from_numpy(x).to(dev) for x in pos]
    r = [_distances(x) for x in p]
    if kind == "matrix":
        m = _matrix(p[0], d, complex(ks[0]) - 0.1j, model, params, r[0])
        return np.array([_lndet(m.cpu())]), 0
    if kind in ("map", "cut"):
        small = case["n"] <= 400
        out = []
        for k in ks:
            m = _matrix(p[0], d, complex(k), model, params, r[0])
            out.append(_lndet(m.cpu() if small else m))
        return np.array(out), np.zeros(ks.size, dtype=np.int32)
    if kind == "dlogf":
        out = []
        for i, k in zip(im, ks):
            a = _matrix(p[i], d, complex(k), model, params, r[i])
            b = _dk_matrix(p[i], d, complex(k), model, params, r[i])
            out.append(complex(torch.diagonal(torch.linalg.solve(a, b)).sum()))
        return np.array(out), np.zeros(ks.size, dtype=np.int32)
    if kind == "amps":
        sigma, amps = [], []
        for i, k in zip(im, ks):
            phi = torch.exp(1j * k.real * p[i][:, 0])
            a = torch.linalg.solve(_matrix(p[i], d, complex(k), model, params, r[i]), phi)
            amps.append(a.cpu().numpy())
            sigma.append(-float((phi.conj() * a).sum().imag) / k.real)
        return np.array(sigma) + 0j, np.concatenate(amps), np.zeros(ks.size, dtype=np.int32)
    if kind == "wave":
        k = complex(ks[0])
        phi = torch.exp(1j * k.real * p[0][:, 0])
        a = torch.linalg.solve(_matrix(p[0], d, k, model, params, r[0]), phi)
        nx, ny = case["nx"], case["ny"]
        rad = (case["n"] / (4.0 * math.pi / 3.0)) ** (1.0 / 3.0)
        px = -rad + torch.arange(nx, dtype=torch.float64, device=dev) * (2 * rad / (nx - 1))
        py = rad - torch.arange(ny, dtype=torch.float64, device=dev) * (2 * rad / (ny - 1))
        rows = []
        for y in py:
            dist = torch.sqrt((px[:, None] - p[0][None, :, 0]) ** 2 + (y - p[0][None, :, 1]) ** 2 + p[0][None, :, 2] ** 2)
            rows.append(torch.exp(1j * k.real * px) + (_green(dist, d, k) * a[None, :]).sum(1))
        psi = torch.cat(rows).cpu().numpy()
        return psi.real.copy(), np.abs(psi) ** 2, psi, a.cpu().numpy()
    mus = []
    for i, k in zip(im, ks):
        m = _matrix(p[i], d, complex(k), model, params, r[i])
        if case["mtype"] == "normalized":
            m = m / (k.real / (4.0 * math.pi) if d == 3 else 0.25)
            m.fill_diagonal_(1j)
        mus.append(np.sort_complex(np.linalg.eigvals(m.cpu().numpy())))
    return np.concatenate(mus), np.zeros(ks.size, dtype=np.int32)
