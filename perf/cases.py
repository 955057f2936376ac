"""The work that users of this library have it do, as cases that can be timed and compared.

Most of it is the Fisher build: cells and counts in, eigenvalues and Fisher matrix out, on the
three kinds of grid the library takes (full-sky shells, Cartesian boxes, patches of sky), from a
unit-test size to 65,536 cells, one at a time or as a batch of mock surveys.  The rest are the
stages that users call by themselves: the xi tables of a new P(k), a block of the signal matrix,
the projection of caller-supplied modes, the estimate from stored covariances.

A build is compared by its eigenvalues and the three sums it forms over the modes: the Fisher
matrix F, the bias f and the quadratic sum q (the record holds q - f).  The window, the mixing
matrix, the band estimates and their covariance follow from these three by N_b x N_b algebra
that multiplies any rounding by F's condition number (10^3 to 10^5 here); that algebra has its
own case, "estimate", on given inputs, where every record is compared.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from opsec_gpu import api, synth

LOG4096 = (256, 4096, 10.0, 20000.0)   # 4096 log-spaced r beyond 10 Mpc/h (the benchmark's tables)
DEFAULT = (512, 256, 200.0, 20000.0)   # the reference's table layout
TWO_PI = 2.0 * math.pi


def listed():
    return [
        # a unit-test sized survey: what is left is launches, host work and the xi tables
        {"name": "shell-96", "kind": "shell", "nr": 3, "nmu": 4, "nphi": 8, "rmin": 200.0, "rmax": 1000.0,
         "nbands": 4, "kmax": 0.2, "nmodes": 40, "log4096": False},
        # one small mock survey (the low end of the batch's range)
        {"name": "shell-2k", "kind": "shell", "nr": 8, "nmu": 16, "nphi": 16, "rmin": 200.0, "rmax": 1000.0,
         "nbands": 20, "kmax": 0.2, "nmodes": 513, "log4096": False},
        # an ordinary survey on a grid of odd sizes: no reflection symmetry of the cells in mu to
        # split the azimuthal blocks by, ragged blocks and tiles
        {"name": "shell-10k-odd", "kind": "shell", "nr": 37, "nmu": 15, "nphi": 18, "rmin": 150.0, "rmax": 900.0,
         "nbands": 20, "kmax": 0.2, "nmodes": 2497, "log4096": True},
        # the benchmark's survey
        {"name": "shell-32k", "kind": "shell", "nr": 32, "nmu": 32, "nphi": 32, "rmin": 200.0, "rmax": 1000.0,
         "nbands": 40, "kmax": 0.4, "nmodes": 8192, "log4096": True},
        # the largest survey, 64 bands
        {"name": "shell-65k", "kind": "shell", "nr": 64, "nmu": 32, "nphi": 32, "rmin": 200.0, "rmax": 1000.0,
         "nbands": 64, "kmax": 0.4, "nmodes": 16384, "log4096": True},
        # mock surveys of uneven sizes in one call, worker threads and streams
        {"name": "mocks-16", "kind": "mocks", "nmocks": 16, "workers": 8, "lo": 2000, "hi": 20000, "nbands": 20,
         "kmax": 0.2},
        # a galaxy survey in a Cartesian box: dense eigensolve, dense projection
        {"name": "box-1728", "kind": "box", "nx": 12, "ny": 12, "nz": 12, "cell": 50.0, "nbands": 20, "kmax": 0.2,
         "nmodes": 500, "log4096": True},
        # a survey of part of the sky, odd grid sizes
        {"name": "patch-3150", "kind": "patch", "nr": 14, "nmu": 15, "nphi": 15, "nbands": 20, "kmax": 0.2,
         "nmodes": 787, "log4096": True},
        # a new P(k): the xi and band tables of the benchmark's layout
        {"name": "xi-40", "kind": "xi", "nbands": 40, "kmax": 0.4, "n1": 256, "n2": 4096, "r1": 10.0, "r2": 20000.0},
        # a new P(k), then rows of the signal matrix (the signal-matrix drop-in)
        {"name": "signal-2k", "kind": "signal", "nr": 8, "nmu": 16, "nphi": 16, "rmin": 200.0, "rmax": 1000.0,
         "nbands": 20, "kmax": 0.2, "nrows": 256, "log4096": False},
        # the comma program: covariances of the caller's own modes on the Q tables at hand
        {"name": "comma-1575", "kind": "comma", "nr": 7, "nmu": 15, "nphi": 15, "nbands": 20, "kmax": 0.2,
         "nmodes": 300},
        # the estimate program: stored covariances, eigenvalues and pixel values to the estimates
        {"name": "estimate-500", "kind": "estimate", "nbands": 20, "kmax": 0.2, "nmodes": 500},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(("shell", "shell", "shell", "mocks", "box", "patch", "xi", "signal", "comma", "estimate"))
    nbands = rng.randint(4, 40)
    kmax = 0.01 * nbands
    if kind in ("shell", "signal"):
        n = _log(rng, 96, 40000) if kind == "shell" else _log(rng, 500, 6000)
        nphi = rng.randint(8, 12) if n < 1000 else rng.randint(12, 36)
        nmu = rng.randint(4, 8) if n < 1000 else rng.randint(9, 33)
        nr = max(3, int(n / (nmu * nphi)))
        while nr * nmu > 1000 * (1 if nmu % 2 else 2):  # the block solver's range
            nr -= 1
        rmin = round(rng.uniform(100.0, 300.0), 1)
        c = {"kind": kind, "nr": nr, "nmu": nmu, "nphi": nphi, "rmin": rmin,
             "rmax": round(rmin + rng.uniform(500.0, 900.0), 1), "nbands": nbands, "kmax": kmax,
             "log4096": rng.random() < 0.6}
        ncells = nr * nmu * nphi
        if kind == "shell":  # bands that the cells can tell apart
            nbands = c["nbands"] = min(nbands, max(3, ncells // 30))
            c["kmax"] = min(kmax, 0.01 * max(20, nbands))
            c["nmodes"] = max(nbands + 8, int(ncells * rng.uniform(0.15, 0.4)))
        else:
            c["nrows"] = rng.randint(3, min(ncells, 400))
        return c
    if kind == "mocks":
        return {"kind": kind, "nmocks": rng.randint(3, 16), "workers": rng.randint(1, 12), "lo": 2000,
                "hi": int(_log(rng, 3000, 20000)), "nbands": min(nbands, 20), "kmax": 0.01 * min(nbands, 20)}
    if kind == "box":
        nx, ny, nz = (rng.randint(5, 14) for _ in range(3))
        nbands = min(nbands, 20, nx * ny * nz // 30)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "cell": round(rng.uniform(35.0, 70.0), 1),
                "nbands": nbands, "kmax": 0.01 * nbands, "nmodes": int(nx * ny * nz * rng.uniform(0.2, 0.4)),
                "log4096": rng.random() < 0.7}
    if kind in ("patch", "comma"):
        nr, nmu, nphi = rng.randint(4, 14), rng.randint(6, 16), rng.randint(6, 15)
        nbands = min(nbands, 20, nr * nmu * nphi // 30)
        c = {"kind": kind, "nr": nr, "nmu": nmu, "nphi": nphi, "nbands": nbands, "kmax": 0.01 * nbands,
             "nmodes": int(nr * nmu * nphi * rng.uniform(0.15, 0.3))}
        if kind == "patch":
            c["log4096"] = rng.random() < 0.7
        return c
    if kind == "xi":
        return {"kind": kind, "nbands": rng.randint(4, 64), "kmax": round(rng.uniform(0.1, 0.6), 3),
                "n1": rng.randint(100, 512), "n2": int(_log(rng, 200, 4096)), "r1": round(rng.uniform(5.0, 200.0), 1),
                "r2": round(_log(rng, 3000.0, 20000.0), 1)}
    return {"kind": "estimate", "nbands": rng.randint(3, 40), "kmax": 0.2, "nmodes": int(_log(rng, 30, 700))}


# ---------------------------------------------------------------- inputs
def _layout(case):
    if case["kind"] == "xi":
        return (case["n1"], case["n2"], case["r1"], case["r2"])
    return LOG4096 if case.get("log4096") else DEFAULT


def _bands(case):
    return synth.band_edges(case["nbands"], 0.0, case["kmax"])


def _pk(seed):
    """A P(k) of the benchmark's form, its amplitude and turnover from the seed."""
    rng = np.random.default_rng([seed, 11])
    k, _ = synth.pk_table()
    amp, k0 = 2e4 * rng.uniform(0.9, 1.1), 0.02 * rng.uniform(0.9, 1.1)
    return k, amp * k / (1.0 + (k / k0) ** 2) ** 1.5


def _survey(case):
    kind = case["kind"]
    if kind in ("shell", "signal"):
        return synth.shell_survey(case["nr"], case["nmu"], case["nphi"], rmin=case["rmin"], rmax=case["rmax"],
                                  rc=0.5 * (case["rmin"] + case["rmax"]), width=0.31 * (case["rmax"] - case["rmin"]))
    if kind == "box":
        n, s = (case["nx"], case["ny"], case["nz"]), case["cell"]
        sv = synth.Survey(synth.COORD_CARTESIAN, (0.0, n[0] * s, 0.0, n[1] * s, 0.0, n[2] * s), n)
        side = (n[0] * n[1] * n[2]) ** (1.0 / 3.0) * s

        def sel(x, y, z):  # a selection without symmetry, as a real survey's
            q = (x - 0.42 * side) ** 2 + 1.3 * (y - 0.57 * side) ** 2 + 0.8 * (z - 0.5 * side) ** 2 + 0.2 * x * y
            return 3e-4 * np.exp(-q / (0.5 * side) ** 2)

        return sv, synth.make_cells(sv, sel, nquad=3)
    sv = synth.Survey(synth.COORD_SPHERICAL, (200.0, 1000.0, -0.5, 0.8, 0.3, 2.0),
                      (case["nr"], case["nmu"], case["nphi"]))

    def nbar(r, mu, phi):
        return 3e-4 * np.exp(-(((r - 600.0) / 250.0) ** 2)) * (1.0 + 0.3 * mu * np.cos(1.7 * phi))

    return sv, synth.make_cells(sv, nbar, nquad=3)


def _mock_list(case, seed):
    mocks = synth.mock_batch(case["nmocks"], seed=case["nmocks"], ncells_range=(case["lo"], case["hi"]))
    rng = np.random.default_rng([seed, 5])
    for m in mocks:
        m["counts"] = rng.poisson(m["cells"]["Nbar"]).astype(np.float64)
    return mocks


def _host_inputs(case, seed):
    """Everything random of a case, on the host, from the seed alone."""
    k, P = _pk(seed)
    d = {"k": k, "P": P}
    rng = np.random.default_rng([seed, 7])
    kind = case["kind"]
    if kind in ("shell", "box", "patch", "signal", "comma"):
        d["survey"], d["cells"] = _survey(case)
        d["counts"] = rng.poisson(d["cells"]["Nbar"]).astype(np.float64)
    if kind == "signal":
        n = d["cells"].size
        d["rows"] = np.sort(rng.choice(n, min(case["nrows"], n), replace=False)).astype(np.int32)
    if kind == "comma":
        n = d["cells"].size
        d["modes"] = np.ascontiguousarray(np.linalg.qr(rng.standard_normal((n, case["nmodes"])))[0].T)
    if kind == "estimate":
        M, nb = case["nmodes"], case["nbands"]
        d["evals"] = np.sort(_power(rng, M))[::-1].copy()
        # derivative matrices as a band's are: a smooth profile over the modes, noise off the diagonal
        j = np.repeat(np.arange(M), np.arange(1, M + 1))
        i = np.arange(M * (M + 1) // 2) - j * (j + 1) // 2
        cov = np.empty((nb, i.size))
        for p in range(nb):
            prof = np.exp(-0.5 * ((np.arange(M) - M * (p + 0.5) / nb) / (0.6 * M / nb + 2.0)) ** 2)
            cov[p] = 1e-3 * np.sqrt(prof[i] * prof[j]) * (rng.standard_normal(i.size) * 0.1 + (i == j))
        d["cov"] = cov
        d["y"] = rng.standard_normal(M) * np.sqrt(1.0 + d["evals"])
    if kind == "mocks":
        d["mocks"] = _mock_list(case, seed)
        d["survey"] = d["mocks"][0]["survey"]
    return d


def _power(rng, M):
    return 8.0 * (np.arange(1, M + 1) / M) ** -0.7 * rng.uniform(0.9, 1.1, M)


def prepare(case, seed):
    d = _host_inputs(case, seed)
    sv = d.get("survey") or synth.Survey(synth.COORD_SPHERICAL, (200.0, 1000.0, -1.0, 1.0, 0.0, TWO_PI), (3, 4, 8))
    e = api.Engine(api.make_config(sv, bands=_bands(case), nmodes=case.get("nmodes"), layout=_layout(case)))
    e.set_pk(d["k"], d["P"])
    d["engine"], d["case"] = e, case
    return d


def run(state):
    case, e = state["case"], state["engine"]
    kind = case["kind"]
    if kind in ("shell", "box", "patch"):
        r = e.fisher_build(state["cells"], state["counts"], case["nmodes"])
        return {"evals": r["evals"], "F": r["F"], "f": r["f"], "q": r["q"] + r["f"]}
    if kind == "mocks":
        return {"F": e.batch_fisher(state["mocks"], workers=case["workers"])["F"]}
    if kind == "xi":
        e.set_pk(state["k"], state["P"])
        r, xi = e.xi_tables()
        return {"r": r, "xi": xi}
    if kind == "signal":
        e.set_pk(state["k"], state["P"])
        return e.signal_block(state["cells"], rows=state["rows"])
    if kind == "comma":
        return e.comma(state["cells"], state["modes"])
    return e.estimate(state["evals"], state["cov"], state["y"])


# ---------------------------------------------------------------- work
def _keys(case):
    """Integrals a build needs: one per symmetry key."""
    kind = case["kind"]
    if kind == "box":
        return case["nx"] * case["ny"] * case["nz"]
    H = case["nr"] * case["nmu"]
    if kind in ("patch", "comma"):
        return H * (H + 1) // 2 * case["nphi"]
    return H * (H + 1) // 4 * (case["nphi"] // 2 + 1)  # both arcs reflected: half of them


def _xi_terms(nbands, layout):
    return (layout[0] + layout[1]) * (32769.0 + 8193.0 * nbands)


def _build_flops(case):
    nb = case["nbands"]
    fl = _keys(case) * 4096.0 * 30.0  # separation, table index and two weights of a point pair
    fl += _keys(case) * 100.0 * 2.0 * (1 + nb)
    if case["kind"] in ("box", "patch"):
        N = case["nx"] * case["ny"] * case["nz"] if case["kind"] == "box" else case["nr"] * case["nmu"] * case["nphi"]
        M = case["nmodes"]
        fl += 4.0 / 3.0 * N ** 3 + 2.0 * N * N * M + nb * (2.0 * N * N * M + N * M * (M + 1.0))
    else:
        npar = 1 if case["nmu"] % 2 else 2
        n, nblk = case["nr"] * case["nmu"] // npar, (case["nphi"] // 2 + 1) * npar
        k = case["nmodes"] * n / (case["nr"] * case["nmu"] * case["nphi"])
        fl += nblk * (4.0 / 3.0 * n ** 3 + 2.0 * n * n * k + nb * (2.0 * n * n * k + 2.0 * n * k * k))
    return fl


def work(case):
    kind, nb = case["kind"], case["nbands"]
    if kind == "xi":
        lay = _layout(case)
        # the tables out, P(k) in; the sum over k of each r as a convolution of a few terms per node
        return {"bytes": 8.0 * (lay[0] + lay[1]) * (2 + nb), "flops": _xi_terms(nb, lay)}
    if kind == "estimate":
        M = case["nmodes"]
        tri = M * (M + 1.0) / 2
        return {"bytes": 8.0 * tri * nb + 16.0 * M, "flops": tri * nb * (nb + 8.0)}
    if kind == "comma":
        N, M = case["nr"] * case["nmu"] * case["nphi"], case["nmodes"]
        return {"bytes": 8.0 * N * M + 80.0 * N + 8.0 * nb * M * (M + 1) / 2,
                "flops": nb * (2.0 * N * N * M + N * M * (M + 1.0))}
    if kind == "mocks":
        total = 0.0
        bytes_ = 0.0
        for m in synth.mock_batch(case["nmocks"], seed=case["nmocks"], ncells_range=(case["lo"], case["hi"])):
            c = {"kind": "shell", "nr": m["nr"], "nmu": m["nmu"], "nphi": m["nphi"], "nbands": nb,
                 "nmodes": m["nmodes"]}
            total += _build_flops(c)
            bytes_ += 88.0 * m["nr"] * m["nmu"] * m["nphi"]
        return {"bytes": bytes_, "flops": total}
    if kind == "signal":
        n = case["nr"] * case["nmu"] * case["nphi"]
        rows = min(case["nrows"], n)
        return {"bytes": 80.0 * n + 8.0 * rows * n, "flops": _keys(case) * 4096.0 * 30.0 + _xi_terms(nb, _layout(case))}
    n = {"box": case.get("nx", 0) * case.get("ny", 0) * case.get("nz", 0)}.get(
        kind, case.get("nr", 0) * case.get("nmu", 0) * case.get("nphi", 0))
    return {"bytes": 88.0 * n + 8.0 * (case["nmodes"] + nb * nb + 2 * nb),
            "flops": _build_flops(case) + _xi_terms(nb, _layout(case))}


# ---------------------------------------------------------------- the same in 64 bits
DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=DEV)


class _Spline:
    """Cubic spline through (x, y) with the end conditions of Forsythe, Malcolm and Moler: the third
    derivative at each end is that of the cubic through the last four points."""

    def __init__(self, x, y):
        n = x.size
        h = np.diff(x)
        s = np.diff(y) / h
        lo, di, up, rhs = np.zeros(n), np.zeros(n), np.zeros(n), np.zeros(n)
        lo[1:-1], up[1:-1], di[1:-1] = h[:-1], h[1:], 2 * (h[:-1] + h[1:])
        rhs[1:-1] = s[1:] - s[:-1]
        dd = rhs[1:-1] / (x[2:] - x[:-2])
        di[0], up[0], di[-1], lo[-1] = -h[0], h[0], -h[-1], h[-1]
        rhs[0] = (dd[1] - dd[0]) * h[0] ** 2 / (x[3] - x[0])
        rhs[-1] = -(dd[-1] - dd[-2]) * h[-1] ** 2 / (x[-1] - x[-4])
        for i in range(1, n):
            t = lo[i] / di[i - 1]
            di[i] -= t * up[i - 1]
            rhs[i] -= t * rhs[i - 1]
        c = np.zeros(n)
        c[-1] = rhs[-1] / di[-1]
        for i in range(n - 2, -1, -1):
            c[i] = (rhs[i] - up[i] * c[i + 1]) / di[i]
        self.x, self.y, self.h = x, y, h
        self.b = s - h * (c[1:] + 2 * c[:-1])
        self.c, self.d = 3 * c[:-1], (c[1:] - c[:-1]) / h

    def __call__(self, k):
        i = np.clip(np.searchsorted(self.x, k, side="right") - 1, 0, self.x.size - 2)
        u = k - self.x[i]
        v = self.y[i] + u * (self.b[i] + u * (self.c[i] + u * self.d[i]))
        return np.where((k >= self.x[0]) & (k < self.x[-1]), v, 0.0)


def _r_grid(layout):
    n1, n2, r1, r2 = layout
    return np.concatenate([np.arange(n1) * r1 / n1, r1 * np.exp(np.arange(n2) * math.log(r2 / r1) / (n2 - 1))])


def _exact_xi(spl, bands, layout):
    """Simpson sums of k^2 P(k) exp(-k^2) j0(kr) / (2 pi^2) at every r of the layout; j0 below x^2 =
    1e-4 by the series the library's reference uses (its x^4 term has the other sign)."""
    r = _t(_r_grid(layout))
    out = torch.zeros((1 + len(bands), r.numel()), dtype=torch.float64, device=DEV)
    for t in range(1 + len(bands)):
        nk, lo, hi = (32768, 0.0, 10.0) if t == 0 else (8192, float(bands[t - 1][0]), float(bands[t - 1][1]))
        j = np.arange(nk + 1)
        k = lo + j * ((hi - lo) / nk)
        P = spl(k) if t == 0 else ((k >= lo) & (k < hi)).astype(np.float64)
        w = (2.0 + 2.0 * (j % 2) - (j == 0) - (j == nk)) * P * k * k * np.exp(-k * k)
        w *= ((hi - lo) / nk / 3.0) / (2.0 * math.pi ** 2)
        k, w = _t(k), _t(w)
        for a in range(0, r.numel(), 1024):
            x = r[a:a + 1024, None] * k[None, :]
            x2 = x * x
            j0 = torch.where(x2 < 1e-4, 1 - x2 * (1 / 6. + x2 * (1 / 120. - x2 * (1 / 5040.))),
                             torch.sin(x) / torch.where(x2 < 1e-4, torch.ones_like(x), x))
            out[t, a:a + 1024] = j0 @ w
    return r, out


def _gauss(n=4):
    x, w = np.polynomial.legendre.leggauss(n)
    return 0.5 * (x + 1.0), 0.5 * w


def _cell_points(sv, d):
    """Cartesian Gauss points [cell][64][3] of the grid cells d [cell][3], and their weights."""
    u, w = _gauss()
    b, n = sv.bounds, sv.n
    ax = []
    for a in range(3):
        lo = b[2 * a] + d[:, a] * (b[2 * a + 1] - b[2 * a]) / n[a]
        hi = b[2 * a] + (d[:, a] + 1) * (b[2 * a + 1] - b[2 * a]) / n[a]
        if sv.coordsys == synth.COORD_SPHERICAL and a == 0:
            ax.append(np.cbrt(lo[:, None] ** 3 * (1 - u) + hi[:, None] ** 3 * u))
        else:
            ax.append(lo[:, None] * (1 - u) + hi[:, None] * u)
    x = [np.broadcast_to(v, (d.shape[0], 4, 4, 4)).reshape(d.shape[0], 64)
         for v in (ax[0][:, :, None, None], ax[1][:, None, :, None], ax[2][:, None, None, :])]
    if sv.coordsys == synth.COORD_SPHERICAL:
        s = x[0] * np.sqrt(1 - x[1] ** 2)
        x = [s * np.cos(x[2]), s * np.sin(x[2]), x[0] * x[1]]
    return _t(np.stack(x, axis=2)), _t((w[:, None, None] * w[None, :, None] * w[None, None, :]).ravel())


def _exact_q(sv, d1, d2, tabT, layout):
    """[pair][table]: the 4^3 x 4^3 Gauss rule of the interpolated tables over pairs of grid cells."""
    n1, n2, r1, r2 = layout
    out = torch.empty((d1.shape[0], tabT.shape[1]), dtype=torch.float64, device=DEV)
    step = 8192
    for a in range(0, d1.shape[0], step):
        x, w = _cell_points(sv, d1[a:a + step])
        y, _ = _cell_points(sv, d2[a:a + step])
        r = torch.sqrt(((x[:, :, None, :] - y[:, None, :, :]) ** 2).sum(dim=3)).reshape(-1, 4096)
        t = torch.where(r < r1, r * (n1 / r1), n1 + torch.log(torch.clamp(r, min=r1) / r1) * ((n2 - 1) / math.log(r2 / r1)))
        t = torch.clamp(t, max=float(n1 + n2 - 1))
        i = torch.clamp(t.floor(), max=float(n1 + n2 - 2))
        fr = t - i
        i = i.long()
        ww = (w[:, None] * w[None, :]).reshape(1, 4096)
        idx = torch.stack([i, i + 1], dim=2).reshape(i.shape[0], -1)
        wt = torch.stack([ww * (1 - fr), ww * fr], dim=2).reshape(i.shape[0], -1)
        out[a:a + step] = torch.nn.functional.embedding_bag(idx, tabT, mode="sum", per_sample_weights=wt)
    return out


def _key_q(sv, tabT, layout):
    """Q of every symmetry key and, for every cell pair, its key."""
    N1, N2, N3 = sv.n
    if sv.coordsys == synth.COORD_CARTESIAN:
        g = np.indices(sv.n).reshape(3, -1).T
        return _exact_q(sv, np.zeros_like(g), g, tabT, layout)
    H = N1 * N2
    nf = N3 // 2 + 1 if sv.full_sky() else N3
    ha, hb = np.triu_indices(H)
    ha, hb, df = np.repeat(ha, nf), np.repeat(hb, nf), np.tile(np.arange(nf), ha.size)
    return _exact_q(sv, np.stack([ha // N2, ha % N2, 0 * ha], 1), np.stack([hb // N2, hb % N2, df], 1), tabT, layout)


def _pair_keys(sv, cells):
    d = [torch.as_tensor(cells[n].astype(np.int64), device=DEV) for n in ("d1", "d2", "d3")]
    N1, N2, N3 = sv.n
    df = [torch.abs(x[:, None] - x[None, :]) for x in d]
    if sv.coordsys == synth.COORD_CARTESIAN:
        return (df[0] * N2 + df[1]) * N3 + df[2]
    H = N1 * N2
    h = d[0] * N2 + d[1]
    ha, hb = torch.minimum(h[:, None], h[None, :]), torch.maximum(h[:, None], h[None, :])
    f, nf = df[2], N3
    if sv.full_sky():
        f, nf = torch.minimum(f, N3 - f), N3 // 2 + 1
    return (ha * H - ha * (ha - 1) // 2 + hb - ha) * nf + f


def _exact_build(case, d):
    sv, cells = d["survey"], d["cells"]
    spl = _Spline(d["k"], d["P"])
    bands, layout = _bands(case), _layout(case)
    tabT = _exact_xi(spl, bands, layout)[1].T.contiguous()
    Q = _key_q(sv, tabT, layout)
    key = _pair_keys(sv, cells)
    rt = torch.sqrt(_t(cells["Nbar"]))
    rr = rt[:, None] * rt[None, :]
    if case["kind"] == "comma":
        B = _t(d["modes"])
    else:
        lam, V = torch.linalg.eigh(rr * Q[:, 0][key])
        lam, V = torch.flip(lam, (0,)), torch.flip(V, (1,))
        M = case["nmodes"]
        if M < lam.numel() and float(lam[M - 1] - lam[M]) < 1e-9 * float(lam[0]):
            # the cut splits the (cos, sin) pair of an azimuthal order; the cos mode is kept: the one
            # that does not change when phi cell d becomes -d
            n3 = sv.n[2]
            flip = torch.arange(cells.size, device=DEV).reshape(-1, n3)[:, (-torch.arange(n3, device=DEV)) % n3]
            pair = V[:, M - 1:M + 1]
            _, rot = torch.linalg.eigh(pair.T @ pair[flip.reshape(-1)])
            V[:, M - 1] = pair @ rot[:, 1]
        lam, B = lam[:M], V[:, :M].T.contiguous()
    Cp = torch.stack([B @ (rr * Q[:, 1 + p][key]) @ B.T for p in range(len(bands))])
    if case["kind"] == "comma":
        j, i = torch.tril_indices(B.shape[0], B.shape[0], device=DEV)
        return Cp[:, i, j].cpu().numpy()
    k256 = [spl(lo + (np.arange(256) + 0.5) * (hi - lo) / 256).mean() for lo, hi in bands]
    w = 1.0 / (1.0 + lam)
    y = B @ _t((d["counts"] - cells["Nbar"]) / np.sqrt(cells["Nbar"]))
    G = (0.5 * Cp * (w[:, None] * w[None, :])).reshape(len(bands), -1)
    R = torch.diag(1.0 + lam) - torch.tensordot(_t(np.array(k256)), Cp, dims=1)
    out = {"evals": lam, "F": G @ Cp.reshape(len(bands), -1).T, "f": G @ R.reshape(-1),
           "q": G @ (y[:, None] * y[None, :]).reshape(-1)}
    return {n: v.cpu().numpy() for n, v in out.items()}


def _exact_estimate(case, d):
    spl = _Spline(d["k"], d["P"])
    prior = _t(np.array([spl(lo + (np.arange(256) + 0.5) * (hi - lo) / 256).mean() for lo, hi in _bands(case)]))
    M = case["nmodes"]
    j, i = torch.tril_indices(M, M, device=DEV)
    D, lam, y = _t(d["cov"]), _t(d["evals"]), _t(d["y"])
    on = (i == j).double()
    w = 1.0 / (1.0 + lam)
    G = D * ((1.0 - 0.5 * on) * w[i] * w[j])
    F, f, q = G @ D.T, G @ (on * (1.0 + lam[i]) - prior @ D), G @ (y[i] * y[j])
    Mx = torch.linalg.inv(F)
    Mx = Mx / (Mx @ F).T.sum(dim=1)[:, None]
    out = {"phat": Mx @ (q - f), "pcov": Mx.T @ Mx @ F, "F": F, "W": (Mx @ F).T, "M": Mx, "q": q - f, "f": f}
    return {n: v.cpu().numpy() for n, v in out.items()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "mocks":
        return None
    if kind in ("shell", "box", "patch", "comma"):
        n = case["nx"] * case["ny"] * case["nz"] if kind == "box" else case["nr"] * case["nmu"] * case["nphi"]
        if n > 4000 or _keys(case) > 300000:
            return None
    d = _host_inputs(case, seed)
    if kind == "xi":
        r, xi = _exact_xi(_Spline(d["k"], d["P"]), _bands(case), _layout(case))
        return {"r": r.cpu().numpy(), "xi": xi.cpu().numpy()}
    if kind == "estimate":
        return _exact_estimate(case, d)
    if kind == "signal":
        cells, rows = d["cells"], d["rows"]
        if rows.size * cells.size > 1200000:
            return None
        tabT = _exact_xi(_Spline(d["k"], d["P"]), [], _layout(case))[1].T.contiguous()
        g = np.stack([cells["d1"], cells["d2"], cells["d3"]], axis=1).astype(np.int64)
        a, b = np.repeat(rows, cells.size), np.tile(np.arange(cells.size), rows.size)
        Q = _exact_q(d["survey"], g[a], g[b], tabT, _layout(case))[:, 0].cpu().numpy()
        return (np.sqrt(cells["Nbar"][a] * cells["Nbar"][b]) * Q).reshape(rows.size, cells.size)
    return _exact_build(case, d)
