"""Timed workloads of the framework: tomographic reconstructions as a user's program runs them,
through the package's public entry points.

Six kinds of case, each over the sizes and options it is used with:

* ``sirt``  Cimmino or SART on a matrix the program keeps (host call, or device-resident vectors);
* ``art``   Kaczmarz sweeps (natural, symmetric, random order) in FP64;
* ``adj``   the reverse-mode adjoint of unrolled SIRT steps (gradients for training loops);
* ``mf``    SIRT on the matrix-free projector pair (nothing of the size of the matrix stored);
* ``batch`` many independent problems advanced together;
* ``cli``   one whole command-line style job: the matrix is traced, used once and dropped.

Sizes, angles and bins follow the tests and the benchmark: parallel beam with angles over [0, pi),
fan beam with R = 2N, unit bins and angles over [0, 2 pi). Measured data are the exact line
integrals of random ellipses plus 1% noise, so no case needs the code under test to make its
inputs. Reduced-precision reconstructions are handed on as FP32 images, which is what they are.
"""
import ctypes as C
import math

import numpy as np
import torch

import fortran_airtools_gb300 as F
from fortran_airtools_gb300._clib import check, lib


def listed():
    return [
        # a thumbnail of the kind the unit tests and quick looks use: launches and latency
        dict(name="sirt_par40_f64", kind="sirt", beam="par", n=40, p=58, nth=60, prec="f64",
             method="sart", its=20, box="lower", entry="host", nprob=1),
        # the plain FP64 fan-beam reconstruction, 181 bins, 100 Cimmino iterations
        dict(name="sirt_fan128_f64", kind="sirt", beam="fan", n=128, p=181, nth=360, prec="f64",
             method="cimmino", its=100, box="lower", entry="host", nprob=1),
        # an odd-sized everyday slice in FP32, nothing tuned
        dict(name="sirt_par363_f32", kind="sirt", beam="par", n=363, p=515, nth=360, prec="f32",
             method="sart", its=30, box="both", entry="host", nprob=1),
        # the large mixed-precision slice on device vectors, on the layouts the autotuner settles on
        dict(name="sirt_par1024_q16", kind="sirt", beam="par", n=1024, p=1448, nth=720, prec="q16",
             method="cimmino", its=10, box="none", entry="device", nprob=1),
        # row-action reconstructions: natural order on the small fan, symmetric with a box on the large
        dict(name="art_fan128", kind="art", beam="fan", n=128, p=181, nth=360, prec="f64",
             method="kaczmarz", its=10, box="lower", entry="host", nprob=1),
        dict(name="art_fan512_sym", kind="art", beam="fan", n=512, p=725, nth=720, prec="f64",
             method="symkaczmarz", its=4, box="both", entry="host", nprob=1),
        # gradients of 20 unrolled steps for a training batch of 16 images
        dict(name="adj_par256_f32", kind="adj", beam="par", n=256, p=362, nth=360, prec="f32",
             method="sart", its=20, box="none", entry="host", nprob=16),
        # the same in FP64 with nonnegativity for a few images of a small odd-sized fan
        dict(name="adj_fan101_f64", kind="adj", beam="fan", n=101, p=144, nth=180, prec="f64",
             method="cimmino", its=9, box="lower", entry="host", nprob=3),
        # matrix-free reconstructions, parallel and fan beam
        dict(name="mf_par1024_f32", kind="mf", beam="par", n=1024, p=1448, nth=720, prec="f32",
             method="cimmino", its=10, box="none", entry="host", nprob=1),
        dict(name="mf_fan512_f32", kind="mf", beam="fan", n=512, p=728, nth=720, prec="f32",
             method="sart", its=10, box="lower", entry="host", nprob=1),
        # uneven fan-beam problems solved together
        dict(name="batch_fan24_f32", kind="batch", beam="fan", n=352, p=500, nth=300, prec="f32",
             method="sart", its=20, box="both", entry="host", nprob=24),
        # the default test problem of the command-line program: build, reconstruct, drop
        dict(name="cli_par256_f64", kind="cli", beam="par", n=256, p=362, nth=360, prec="f64",
             method="sart", its=10, box="lower", entry="host", nprob=1),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("sirt", "art", "adj", "mf", "batch", "cli"))
    beam = rng.choice(("par", "fan"))
    box = rng.choice(("none", "lower", "both"))
    method = rng.choice(("sart", "cimmino"))
    entry, prec, nprob = "host", "f64", 1
    if kind == "sirt":
        n, its = _logint(rng, 40, 512), _logint(rng, 5, 50)
        nth = _logint(rng, 60, 360)
        prec = rng.choice(("f64", "f32", "f16", "q16"))
        entry = rng.choice(("host", "device"))
    elif kind == "art":
        n, its = _logint(rng, 40, 256), 2 * rng.randint(1, 3)
        nth = _logint(rng, 60, 360)
        method = rng.choice(("kaczmarz", "symkaczmarz", "randkaczmarz"))
        if method == "randkaczmarz":
            n = min(n, 96)
    elif kind == "adj":
        n, its = _logint(rng, 48, 256), rng.randint(4, 20)
        nth = _logint(rng, 60, 360)
        prec = rng.choice(("f32", "f64"))
        nprob = rng.randint(1, 16)
        if prec == "f32":
            box = "none"  # a value at its bound would switch its gradient on the last FP32 bit
    elif kind == "mf":
        n, its = _logint(rng, 64, 768 if beam == "par" else 448), rng.randint(2, 10)
        nth = _logint(rng, 90, 720)
        prec = rng.choice(("f32", "f32", "f64"))
        if prec == "f64":
            n = min(n, 256)
    elif kind == "batch":
        n, its = _logint(rng, 64, 352), rng.randint(5, 20)
        nth = _logint(rng, 60, 300)
        prec = rng.choice(("f32", "q16", "f64"))
        nprob = rng.randint(2, 24)
    else:
        n, its = _logint(rng, 48, 320), _logint(rng, 2, 20)
        nth = _logint(rng, 60, 360)
    p = int(math.ceil(1.42 * n))
    p += (p - n) % 2  # bins as symmetric about the grid as the pixels are: no ray along a grid line
    if beam == "fan":
        p += p % 2
    return dict(kind=kind, beam=beam, n=n, p=p, nth=nth, prec=prec, method=method, its=its, box=box,
                entry=entry, nprob=nprob)


# ---- inputs -------------------------------------------------------------------------------------
def _theta(g):
    return (math.pi if g["beam"] == "par" else 2.0 * math.pi) * np.arange(g["nth"]) / g["nth"]


def _problems(case):
    """The geometries of a batch (its first is the case's own, the others smaller); else one."""
    out = [dict(beam=case["beam"], n=case["n"], p=case["p"], nth=case["nth"])]
    rng = np.random.default_rng(2)
    while case["kind"] == "batch" and len(out) < case["nprob"]:
        n = int(rng.integers(max(32, case["n"] // 5), case["n"] + 1))
        p = int(math.ceil(1.42 * n))
        p += p % 2 if case["beam"] == "fan" else (p - n) % 2
        nth = int(rng.integers(max(30, case["nth"] // 3), case["nth"] + 1))
        out.append(dict(beam=case["beam"], n=n, p=p, nth=nth))
    return out


def _data(g):
    if g["beam"] == "par":
        return F.Data(n=g["n"], p=g["p"], nth=g["nth"], theta=_theta(g))
    return F.Data(n=g["n"], p=g["p"], nth=g["nth"], r=2.0, dw=g["p"] / g["n"], sd=2.0, theta=_theta(g))


def _matrix(g):
    return F.paralleltomo(_data(g)) if g["beam"] == "par" else F.fanlineartomo(_data(g))


def _rays(g):
    """Start point and unit direction of every ray: four arrays (nth, p)."""
    n, p, th = g["n"], g["p"], _theta(g)
    c, s = np.cos(th)[:, None], np.sin(th)[:, None]
    if g["beam"] == "par":
        x = (np.arange(p) - 0.5 * (p - 1))[None, :]
        one = np.ones((1, p))
        return c * x, s * x, -s * one, c * one
    R, sd = 2.0 * n, 2.0 * n
    if p % 2:  # the reference's bin angles for odd p: the lower half is not the mirror of the upper
        at = np.arctan(sd / np.arange(1, (p - 1) // 2 + 1))
        om = np.concatenate([at[::-1] - 0.5, [0.0], 0.5 * math.pi - at])
    else:
        at = np.arctan(sd / (np.arange(1, p // 2 + 1) - 0.5))
        om = np.concatenate([at[::-1] - 0.5 * math.pi, 0.5 * math.pi - at])
    co, so = np.cos(om)[None, :], np.sin(om)[None, :]
    x0, y0 = -s * R, c * R
    ua, ub = s, -c
    one = np.ones((1, p))
    return x0 * one, y0 * one, co * ua - so * ub, so * ua + co * ub


def _ellipses(rng, n, count=8):
    """Random ellipses inside the unit disc: amplitude, semi-axes, centre, angle (in pixels)."""
    a, b = rng.uniform(0.06, 0.45, (2, count)) * 0.5 * n
    x0, y0 = rng.uniform(-0.35, 0.35, (2, count)) * 0.5 * n
    return rng.uniform(0.1, 1.0, count), a, b, x0, y0, rng.uniform(0, math.pi, count)


def _image(e, n):
    """The ellipses on the pixel grid, column by column from the top."""
    c = np.arange(n) + 0.5 - 0.5 * n
    X, Y = c[:, None], c[::-1][None, :]
    v = np.zeros((n, n))
    for amp, a, b, x0, y0, phi in zip(*e):
        u = (X - x0) * math.cos(phi) + (Y - y0) * math.sin(phi)
        w = (Y - y0) * math.cos(phi) - (X - x0) * math.sin(phi)
        v += amp * ((u / a) ** 2 + (w / b) ** 2 <= 1.0)
    return (v / max(v.max(), 1e-12)).reshape(-1)


def _sinogram(e, g, rng):
    """Line integrals of the ellipses along every ray, with 1% noise."""
    x, y, dx, dy = _rays(g)
    b = np.zeros((g["nth"], g["p"]))
    for amp, ax, ay, x0, y0, phi in zip(*e):
        c, s = math.cos(phi), math.sin(phi)
        px, py = ((x - x0) * c + (y - y0) * s) / ax, ((y - y0) * c - (x - x0) * s) / ay
        qx, qy = (dx * c + dy * s) / ax, (dy * c - dx * s) / ay
        A, B, K = qx * qx + qy * qy, px * qx + py * qy, px * px + py * py - 1.0
        b += amp * 2.0 * np.sqrt(np.maximum(B * B - A * K, 0.0)) / A
    b = b.reshape(-1) / 2.0
    e = rng.standard_normal(b.size)
    return b + 0.01 * np.linalg.norm(b) / np.linalg.norm(e) * e


def _inputs(case, seed):
    """Measured data (and, for the adjoint, relaxation parameters and dL/dx) as numpy arrays."""
    rng = np.random.default_rng([int(seed), case["n"], case["nth"]])
    out = {}
    if case["kind"] == "adj":
        es = [_ellipses(rng, case["n"]) for _ in range(case["nprob"])]
        out["b"] = np.asfortranarray(np.stack([_sinogram(e, case, rng) for e in es], 1))
        out["lam"] = rng.uniform(0.6, 1.4, case["nprob"])
        gx = np.stack([_image(e, case["n"]) for e in es], 1)
        out["gx"] = np.asfortranarray(-0.3 * gx + 0.05 * rng.standard_normal(gx.shape))
    else:
        out["b"] = np.concatenate([_sinogram(_ellipses(rng, g["n"]), g, rng) for g in _problems(case)])
    return out


def _bounds(case):
    return {"none": (None, None), "lower": (0.0, None), "both": (0.0, 1.0)}[case["box"]]


def _relax(case):
    return 0.25 if case["kind"] == "art" else 1.0


# ---- the calls ----------------------------------------------------------------------------------
def prepare(case, seed):
    S = dict(case=case, **_inputs(case, seed))
    lo, up = _bounds(case)
    S["opts"] = F.airms.options(relaxpar=_relax(case), lbound=lo, ubound=up,
                                rowprobability=case["method"] == "randkaczmarz")
    kind = case["kind"]
    if kind in ("sirt", "art", "adj"):
        S["A"] = A = _matrix(case)
        A.set_precision(case["prec"])
        if kind == "sirt" and case["entry"] == "device":
            S["stream"] = torch.cuda.Stream()
            A.set_stream(S["stream"].cuda_stream)
            if case["n"] >= 768:
                check(lib().fair_sirt_set_lanes(A.handle, (C.c_int32 * 4)(8, 8, 14, 14)))
            check(lib().fair_sirt_prepare(A.handle, case["method"].encode(), C.byref(S["opts"])))
            S["d_b"] = torch.from_numpy(S["b"]).cuda()
            S["d_x"] = torch.zeros(A.n, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
    elif kind == "mf":
        S["A"] = F.MatrixFree(_data(case), case["prec"], beam="parallel" if case["beam"] == "par" else "fan")
    elif kind == "batch":
        S["A"] = F.Batch(case["prec"], layout="tiled")
        for g in _problems(case):
            A = _matrix(g)
            S["A"].add(A, take=True)
            A.close()
    else:
        S["dat"] = _data(case)
    return S


def _image_out(case, x):
    """Reduced-precision reconstructions leave as FP32 images."""
    if case["prec"] == "f64":
        return x
    return x.to(torch.float32) if isinstance(x, torch.Tensor) else x.astype(np.float32)


def run(S):
    case = S["case"]
    kind, method, its = case["kind"], case["method"], case["its"]
    if kind == "cli":
        A = _matrix(case)
        x = F.airms.sirt(method, A, S["b"], its, opts=S["opts"])
        A.close()
        return x
    A = S["A"]
    if kind == "sirt" and case["entry"] == "device":
        with torch.cuda.stream(S["stream"]):
            S["d_x"].zero_()
            check(lib().fair_sirt_run_device(A.handle, S["d_b"].data_ptr(), S["d_x"].data_ptr(), its))
            return _image_out(case, S["d_x"])
    if kind == "sirt":
        return _image_out(case, F.airms.sirt(method, A, S["b"], its, opts=S["opts"]))
    if kind == "art":
        if method == "randkaczmarz":
            F.airms.random_seed(4)
        return np.ascontiguousarray(F.airms.art(method, A, S["b"], its, opts=S["opts"])[:, 0])
    if kind == "adj":
        x, gb, gx0, gl = F.airms.sirt_adjoint(method, A, S["b"], its, S["lam"], S["gx"], opts=S["opts"])
        return dict(x=_image_out(case, x), gb=_image_out(case, gb), gx0=_image_out(case, gx0),
                    glam=_image_out(case, np.asarray(gl)))
    return _image_out(case, A.sirt(method, S["b"], its, opts=S["opts"]))


def _nnz(g):
    """Nonzeros of the geometry's matrix: pixels x angles x the mean number of rays through a pixel."""
    return 4.0 / math.pi * g["nth"] * g["n"] ** 2


def work(case):
    """Products with A and A' read each stored value once; matrix-free ones only the vectors."""
    size = {"f64": 8, "f32": 4, "f16": 2, "q16": 2}[case["prec"]]
    nnz = sum(_nnz(g) for g in _problems(case))
    m = sum(g["nth"] * g["p"] for g in _problems(case))
    n = sum(g["n"] ** 2 for g in _problems(case))
    its, k = case["its"], case["nprob"] if case["kind"] == "adj" else 1
    products = {"adj": 6, "art": 2 if case["method"] == "symkaczmarz" else 1}.get(case["kind"], 2) * its
    if case["method"] == "symkaczmarz":
        products //= 2
    flops = 2.0 * nnz * products * k * (2 if case["kind"] == "art" else 1)
    if case["kind"] == "mf":
        return dict(bytes=float(its * size * 2 * (m + 2 * n)), flops=flops)
    vec = products * k * size * (m + 2 * n)
    traced = nnz * 12.0 if case["kind"] == "cli" else 0.0
    return dict(bytes=products * nnz * size + vec + traced, flops=flops)


# ---- the same in 64 bits, from the mathematics --------------------------------------------------
def _trace(g, dev):
    """Rows, columns and lengths of the ray-traced matrix, row by row in ray order (FP64, torch)."""
    n, p, nth = g["n"], g["p"], g["nth"]
    x, y, dx, dy = (torch.from_numpy(np.ascontiguousarray(np.broadcast_to(v, (nth, p)))).to(dev) for v in _rays(g))
    if g["beam"] == "par":
        flat = torch.from_numpy(np.abs(np.cos(_theta(g))) < 1e-15).to(dev)
        dy[flat] = 0.0
    grid = torch.arange(n + 1, dtype=torch.float64, device=dev) - 0.5 * n
    step = max(1, int(2.5e7 // (p * (2 * n + 2))))
    out, hi = ([], [], []), 0.5 * n
    for i in range(0, nth, step):
        X, Y, U, V = (v[i:i + step].reshape(-1, 1) for v in (x, y, dx, dy))
        tx, ty = (grid - X) / U, (grid - Y) / V
        yx, xy = Y + V * tx, X + U * ty
        t = torch.cat([torch.where(yx.abs() <= hi, tx, math.inf), torch.where(xy.abs() <= hi, ty, math.inf)], 1)
        t = torch.where(torch.isfinite(t), t, math.inf)
        t = torch.sort(t, dim=1).values
        a, b = t[:, :-1], t[:, 1:]
        d = torch.where(torch.isfinite(b), b - a, 0.0)
        keep = d > 1e-10
        mid = 0.5 * (a + b)
        cx = torch.floor(X + U * mid + hi)
        cy = torch.floor(Y + V * mid + hi)
        keep &= (cx >= 0) & (cx < n) & (cy >= 0) & (cy < n)
        r = torch.arange(X.shape[0], device=dev).unsqueeze(1).expand_as(keep)[keep] + i * p
        out[0].append(r.to(torch.int32))
        out[1].append((cx * n + (n - 1 - cy))[keep].to(torch.int32))
        out[2].append(d[keep])
    return tuple(torch.cat(v) for v in out)


class _Products:
    """A x and A' y over the traced entries, for vectors or blocks of columns."""

    def __init__(self, g, dev):
        self.r, self.c, self.v = _trace(g, dev)
        self.m, self.n = g["nth"] * g["p"], g["n"] ** 2

    def _sum(self, where, size, src, x):
        out = torch.zeros((size,) + tuple(x.shape[1:]), dtype=torch.float64, device=x.device)
        part = max(1, int(4e8) // max(1, x[0].numel()))
        for i in range(0, self.v.numel(), part):
            s = slice(i, i + part)
            v = self.v[s].reshape((-1,) + (1,) * (x.ndim - 1))
            out.index_add_(0, where[s], v * x.index_select(0, src[s]))
        return out

    def ax(self, x):
        return self._sum(self.r, self.m, self.c, x)

    def aty(self, y):
        return self._sum(self.c, self.n, self.r, y)

    def weights(self, method):
        """1/M and 1/D, 0 where a row or column is empty."""
        z = torch.zeros(self.m, dtype=torch.float64, device=self.v.device)
        if method == "sart":
            M = z.index_add_(0, self.r, self.v)
            D = torch.zeros(self.n, dtype=torch.float64, device=z.device).index_add_(0, self.c, self.v)
        else:
            M = self.m * z.index_add_(0, self.r, self.v * self.v)
            D = torch.ones(self.n, dtype=torch.float64, device=z.device)
        inv = lambda w: torch.where(w > 0, 1.0 / w, 0.0)  # noqa: E731
        return inv(M), inv(D)


def _clamp(x, lo, up):
    if up is not None:
        x = torch.clamp(x, max=up)
    if lo is not None:
        x = torch.clamp(x, min=lo)
    return x


def _sirt64(case, g, b, dev):
    P = _Products(g, dev)
    Mi, Di = P.weights(case["method"])
    lo, up = _bounds(case)
    b = torch.from_numpy(b).to(dev)
    x = torch.zeros(P.n, dtype=torch.float64, device=dev)
    for _ in range(case["its"]):
        x = _clamp(x + Di * P.aty(Mi * (b - P.ax(x))), lo, up)
    return x.cpu().numpy()


def _adjoint64(case, I, dev):
    P = _Products(case, dev)
    Mi, Di = (w.unsqueeze(1) for w in P.weights(case["method"]))
    lo, up = _bounds(case)
    b, lam, gx = (torch.from_numpy(np.ascontiguousarray(I[k])).to(dev) for k in ("b", "lam", "gx"))
    x = torch.zeros((P.n, case["nprob"]), dtype=torch.float64, device=dev)
    zs, gs = [], []
    for _ in range(case["its"]):
        gs.append(Di * P.aty(Mi * (b - P.ax(x))))
        zs.append(x + lam * gs[-1])
        x = _clamp(zs[-1], lo, up)
    gb, glam = torch.zeros_like(b), torch.zeros_like(lam)
    for z, g in zip(reversed(zs), reversed(gs)):
        on = torch.ones_like(z, dtype=torch.bool)
        if up is not None:
            on &= z < up
        if lo is not None:
            on &= z > lo
        gz = torch.where(on, gx, 0.0)
        glam += (gz * g).sum(0)
        w = Mi * P.ax(Di * gz)
        gb += lam * w
        gx = gz - lam * P.aty(w)
    out = dict(x=x, gb=gb, gx0=gx, glam=glam)
    return {k: v.cpu().numpy() for k, v in out.items()}


def _kaczmarz64(case, b, dev):
    r, c, v = _trace(case, dev)
    m = case["nth"] * case["p"]
    ptr = np.concatenate([[0], np.cumsum(np.bincount(r.cpu().numpy(), minlength=m))])
    c, v = c.cpu().numpy().astype(np.int64), v.cpu().numpy()
    lo, up = _bounds(case)
    relax = _relax(case)
    x = np.zeros(case["n"] ** 2)
    rows = [(c[ptr[i]:ptr[i + 1]], v[ptr[i]:ptr[i + 1]], b[i]) for i in range(m) if ptr[i + 1] > ptr[i]]
    rows = [(q, w, bi, relax / float(w @ w)) for q, w, bi in rows]
    sym = case["method"] == "symkaczmarz"
    for _ in range(case["its"] // 2 if sym else case["its"]):
        for order in (rows, rows[::-1]) if sym else (rows,):
            for q, w, bi, k in order:
                t = x[q]
                t += (k * (bi - float(w @ t))) * w
                if lo is not None:
                    np.maximum(t, lo, out=t)
                if up is not None:
                    np.minimum(t, up, out=t)
                x[q] = t
    return x


def exact(case, seed):
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    I = _inputs(case, seed)
    if case["kind"] == "art":
        steps = case["its"] * case["nth"] * case["p"]
        if case["beam"] == "fan" and case["p"] % 2:
            steps //= 2  # the lower half of the bins misses the image
        if case["method"] == "randkaczmarz" or steps > 1.2e6:
            return None  # the library's own random stream; or too many sequential steps
        return _kaczmarz64(case, I["b"], dev)
    if case["kind"] == "adj":
        return _adjoint64(case, I, dev)
    out, at = [], 0
    for g in _problems(case):
        m = g["nth"] * g["p"]
        out.append(_sirt64(case, g, I["b"][at:at + m], dev))
        at += m
    return np.concatenate(out)
