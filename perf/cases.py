"""The work that users have this framework do, as cases to measure.

A case is a dict of plain sizes.  `prepare` makes what a user's program holds
before the call (seeded inputs on the GPU, the operators it keeps), `run` is
one pass through the public entry points, `work` counts the bytes and the
operations that the path cannot do without, and `exact` states the outputs in
64 bits with torch alone.

Kinds:
  call         Forward_XRD on numpy arrays, the drop-in call of a script
  counts       forward, coherent and Compton counts, device arrays
  matrix       the same with the model matrix
  tables       forward_tables, nearest or bilinear cross-section lookups
  op_forward   Operator.forward, one pattern per voxel
  op_adjoint   Operator.adjoint
  mlem         Batch.mlem on one or several operators
  matrix_mlem  mlem_matrix on a stored model matrix
  ct           ct_sinogram
  basis        basis_expand
"""
from __future__ import annotations

import math

import numpy as np
import torch

import xrd_tomography_gb300 as xt
from xrd_tomography_gb300 import synth

DEV = "cuda:0"
_state = {}


def _stream():
    """One stream and one library context on it, as a program keeps them."""
    if not _state:
        _state["stream"] = torch.cuda.Stream(DEV)
        _state["ctx"] = xt.Context(0, stream=_state["stream"].cuda_stream)
    return _state["stream"], _state["ctx"]


# ---- the cases -----------------------------------------------------------------

def _scan(kind, nx, ny, views, px, es, ed, dnrg, nwt, nqf, mats, r_src, r_det, col, **more):
    return dict(kind=kind, nx=nx, ny=ny, views=views, px=px, es=es, ed=ed, dnrg=dnrg, nwt=nwt, nqf=nqf, mats=mats,
                r_src=r_src, r_det=r_det, col=col, **more)


def _fan(side, px):
    """A fan scanner for a phantom of `side` 2 mm voxels (source and detector
    radius, pixel pitch in mm) that keeps both outside it."""
    return dict(r_src=3.0 * side, r_det=2.2 * side, col=5.2 * side / px)


def listed():
    return [
        # the drop-in call from a script on host arrays, all three outputs: a
        # small phantom, where the call's own overhead is what a user waits for
        _scan("call", 12, 12, 4, 8, 12, 12, 2, 32, 64, 3, 75.0, 60.0, 2.0, name="call_host_12"),
        # an odd-sized slice with the tabulated cross-sections, bilinear
        _scan("tables", 45, 33, 10, 75, 37, 29, 4, 32, 64, 3, bilinear=True, **_fan(45, 75), name="tables_45x33"),
        # the model matrix of a 64^2 phantom for a reconstruction with unknowns per material
        _scan("matrix", 64, 64, 32, 128, 40, 32, 5, 64, 64, 4, 300.0, 200.0, 1.0, name="matrix_64"),
        # counts of an ordinary slice
        _scan("counts", 128, 128, 32, 128, 40, 32, 5, 32, 64, 4, 300.0, 200.0, 1.0, name="counts_128"),
        # counts in the configuration that the reference is compiled for
        dict(kind="counts", preset=100, name="counts_reference_100"),
        # counts of a large slice, a quarter of its 180 views
        _scan("counts", 256, 256, 45, 512, 64, 64, 5, 32, 128, 8, 600.0, 500.0, 1.0, name="counts_256"),
        # forward and backward of the operator with one pattern per voxel, as an
        # outer optimisation loop calls them
        _scan("op_forward", 128, 128, 32, 128, 40, 32, 5, 32, 64, 4, 300.0, 200.0, 1.0, name="op_forward_128"),
        _scan("op_adjoint", 96, 78, 27, 110, 40, 32, 5, 40, 64, 4, 250.0, 180.0, 1.0, name="op_adjoint_96x78"),
        # MLEM of several small phantoms in one batch
        _scan("mlem", 48, 48, 16, 32, 64, 64, 5, 32, 128, 4, n=12, iters=2, **_fan(48, 32), name="mlem_batch_12"),
        # MLEM on the stored matrix of a 64^2 phantom: 131072 rays x 64 bins x 4 materials
        dict(kind="matrix_mlem", rays=131072, K=256, iters=10, name="matrix_mlem_131072x256"),
        # the transmission sinogram of a large slice
        _scan("ct", 256, 256, 180, 512, 64, 64, 5, 32, 128, 8, 600.0, 500.0, 1.0, name="ct_256"),
        # coefficients of a dense basis expanded onto the fine q grid, every voxel of a 384^2 slice
        dict(kind="basis", M=147456, K=64, N=256, name="basis_147456x64x256"),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["call", "tables", "matrix", "counts", "counts", "counts", "op_forward", "op_adjoint", "mlem",
                       "matrix_mlem", "ct", "basis"])
    if kind == "matrix_mlem":
        return dict(kind=kind, rays=log(500, 131072), K=4 * log(8, 64), iters=rng.randint(2, 10))
    if kind == "basis":
        return dict(kind=kind, M=log(500, 147456), K=8 * rng.randint(1, 8), N=16 * rng.randint(1, 16))
    nx = log(12, 200 if kind == "ct" else 40 if kind == "call" else 110)
    ny = max(8, int(nx * rng.uniform(0.7, 1.0)))
    views, px = log(4, 60), log(8, 160)
    if kind == "call":
        views, px = log(4, 10), log(8, 32)
    if kind == "mlem":
        views, px, nx = log(4, 16), log(8, 32), log(12, 48)
        ny = nx
    ed = rng.choice([12, 24, 29, 32, 48, 64])
    es = ed if rng.random() < 0.5 else ed + rng.randint(1, 12)
    c = _scan(kind, nx, ny, views, px, es, ed, rng.choice([2, 4, 5]), rng.choice([24, 32, 40, 64]),
              rng.choice([64, 96, 128, 256]), rng.randint(2, 8), **_fan(nx, px))
    if kind == "matrix":
        c["nwt"], c["mats"] = 32, rng.randint(2, 4)
        while c["views"] * c["px"] * c["ed"] > 100000:
            c["views"], c["px"] = max(4, c["views"] // 2), max(8, (c["px"] * 3) // 4)
            c.update(_fan(nx, c["px"]))
    if kind == "tables":
        c["bilinear"] = rng.random() < 0.5
    if kind == "mlem":
        c["n"], c["iters"] = rng.randint(1, 8), rng.randint(1, 3)
    return c


# ---- inputs ----------------------------------------------------------------------

def _problem(c):
    if "preset" in c:
        return xt.reference_problem(c["preset"])
    p = xt.reference_problem(c["nx"], c["ny"])
    p.n_src, p.n_col, p.n_row = c["views"], c["px"], 1
    p.nrg_src, p.nrg_det, p.dnrg = c["es"], c["ed"], c["dnrg"]
    p.e_src_min = p.e_det_min = 20.0
    p.e_src_max = p.e_det_max = 80.0
    p.nwt, p.nqf, p.n_mat = c["nwt"], c["nqf"], c["mats"]
    p.q_lo, p.q_hi, p.dq0 = 0.5, 4.0, 0.02 if c["nwt"] > 32 else 0.05
    return synth.scanner(p, 2.0, c["r_src"], c["r_det"], c["col"])


def _parts(c):
    """The problems of a case: one, or a batch's phantoms from half to full size."""
    n = c.get("n", 1)
    out = []
    for i in range(n):
        f = 1.0 if n == 1 else 0.5 + 0.5 * i / (n - 1)
        side = max(12, int(c["nx"] * f)) if "nx" in c else None
        d = dict(c) if n == 1 else dict(c, nx=side, ny=side, views=max(4, int(c["views"] * f)),
                                        px=max(8, int(c["px"] * f)))
        if n > 1:
            d.update(_fan(side, d["px"]))
        out.append(d)
    return out


def _inputs(c, seed):
    return [synth.make_inputs(_problem(d), 1000 * seed + i) for i, d in enumerate(_parts(c))]


def _rand(seed, shape, lo, hi):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.empty(shape, device=DEV, dtype=torch.float32).uniform_(lo, hi, generator=g)


def _counts(seed, n, mean):
    """Photon counts: Poisson noise about uneven means."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.poisson(_rand(seed + 1, n, 0.2 * mean, 1.8 * mean), generator=g)


def _model_matrix(seed, rays, K):
    """A stored model matrix with the shape of a real one: each ray a few broad
    peaks along q, over a range of magnitudes."""
    r = _rand(seed, (rays, 4), 0.0, 1.0)
    k = torch.arange(K, device=DEV, dtype=torch.float32) / K
    A = torch.zeros(rays, K, device=DEV)
    for j in range(2):
        A += torch.exp(-0.5 * ((k[None, :] - r[:, j:j + 1]) / (0.02 + 0.06 * r[:, 2:3])) ** 2)
    A *= torch.exp(-4.0 * r[:, 3:4])
    return A


def _table(p, seed):
    rng = np.random.default_rng(seed)
    q = np.linspace(0.0, 1.0, p.nq)[:, None]
    a = np.linspace(0.0, 1.0, p.na)[None, :]
    ph = rng.uniform(0, 2 * math.pi, 2)
    t = np.exp(-2.5 * q) * (0.75 + 0.2 * np.cos(2.7 * a + ph[0])) + 0.05 * np.sin(7.0 * q + ph[1]) * a
    return (255.0 * np.clip(t, 0.0, None)).astype(np.float32).flatten(order="F")


def _mlem_data(c, seed, inps):
    ys, cs, xs = [], [], []
    for i, inp in enumerate(inps):
        p = inp.problem
        ys.append(_counts(seed + 10 * i + 1, p.rays, 200.0))
        cs.append(_rand(seed + 10 * i + 3, p.rays, 0.0, 20.0))
        xs.append(_rand(seed + 10 * i + 4, p.nx * p.ny * p.nwt, 0.5, 1.5))
    return ys, cs, xs


def _matrix_data(c, seed):
    A = _model_matrix(seed, c["rays"], c["K"])
    return A, _counts(seed + 1, c["rays"], 200.0), _rand(seed + 3, c["rays"], 0.0, 20.0), \
        _rand(seed + 4, c["K"], 0.5, 1.5)


def prepare(case, seed):
    st, ctx = _stream()
    k = case["kind"]
    s = {"kind": k, "case": case}
    with torch.cuda.stream(st):
        if k == "matrix_mlem":
            s["A"], s["y"], s["c"], s["x0"] = _matrix_data(case, seed)
        elif k == "basis":
            s["C"] = _rand(seed, (case["M"], case["K"]), 0.0, 1.0)
            s["B"] = _rand(seed + 1, (case["K"], case["N"]), 0.0, 1.0)
            s["I"] = torch.empty(case["M"], case["N"], device=DEV)
        else:
            inps = _inputs(case, seed)
            inp = inps[0]
            p = s["p"] = inp.problem
            if k == "call":
                s["args"] = inp.args()[:2] + (np.asarray(inp.seg).reshape(p.nx, p.ny, order="F"),) + inp.args()[3:]
                return s
            dev = [torch.from_numpy(np.ascontiguousarray(a)).to(DEV)
                   for a in (inp.spectrum, inp.Ifine, inp.seg, inp.a1, inp.a2, inp.S2)]
            s["edges"] = (inp.q_min, inp.q_max, inp.a_min, inp.a_max)
            s["dev"] = dev
            if k in ("counts", "matrix", "tables", "ct"):
                s["N"], s["C"] = torch.empty(p.rays, device=DEV), torch.empty(p.rays, device=DEV)
            if k == "matrix":
                s["A"] = torch.empty(p.amatrix_elems, device=DEV)
            if k == "tables":
                s["S1"] = torch.from_numpy(_table(p, seed)).to(DEV)
            if k in ("op_forward", "op_adjoint", "mlem"):
                s["ops"] = [xt.Operator(i.problem, i.spectrum, i.seg, i.a1, i.a2, ctx=ctx) for i in inps]
            if k == "op_forward":
                s["x"] = _rand(seed + 1, p.nx * p.ny * p.nwt, 0.0, 1.0)
                s["y"] = torch.empty(p.rays, device=DEV)
            elif k == "op_adjoint":
                s["w"] = _rand(seed + 1, p.rays, 0.0, 2.0)
                s["g"] = torch.empty(p.nx * p.ny * p.nwt, device=DEV)
            elif k == "mlem":
                s["batch"] = xt.Batch(s["ops"], ctx=ctx)
                s["ys"], s["cs"], s["x0s"] = _mlem_data(case, seed, inps)
    st.synchronize()
    return s


def run(s):
    st, ctx = _stream()
    k = s["kind"]
    with torch.cuda.stream(st):
        if k == "call":
            return xt.Forward_XRD(*s["args"], problem=s["p"], ctx=ctx)
        if k in ("counts", "matrix"):
            d = s["dev"]
            N, C, A = xt.forward(s["p"], *d, *s["edges"], Nphotons=s["N"], Cphotons=s["C"], Amatrix=s.get("A"),
                                 want_amatrix=k == "matrix", ctx=ctx)
            return (N, C) if A is None else (N, C, A)
        if k == "tables":
            sp, _, seg, a1, a2, S2 = s["dev"]
            return xt.forward_tables(s["p"], sp, seg, a1, a2, s["S1"], S2, *s["edges"], Nphotons=s["N"],
                                     Cphotons=s["C"], bilinear=s["case"]["bilinear"], ctx=ctx)
        if k == "op_forward":
            return s["ops"][0].forward(s["x"], s["y"])
        if k == "op_adjoint":
            return s["ops"][0].adjoint(s["w"], s["g"])
        if k == "mlem":
            xs = [x.clone() for x in s["x0s"]]
            return s["batch"].mlem(s["ys"], s["cs"], xs, s["case"]["iters"])
        if k == "matrix_mlem":
            return xt.mlem_matrix(s["A"], s["y"], s["c"], s["x0"].clone(), s["case"]["iters"], ctx=ctx)
        if k == "ct":
            sp, _, _, a1, a2, _ = s["dev"]
            return xt.ct_sinogram(s["p"], sp, a1, a2, Tphotons=s["N"], gain0=s["C"], ctx=ctx)
        return xt.basis_expand(s["C"], s["B"], s["I"], ctx=ctx)


# ---- what the path cannot do without ----------------------------------------------

def work(case):
    k = case["kind"]
    if k == "basis":
        M, K, N = case["M"], case["K"], case["N"]
        return {"bytes": 4.0 * (M * K + K * N + M * N), "flops": 2.0 * M * K * N}
    if k == "matrix_mlem":
        a = 4.0 * case["rays"] * case["K"]   # the matrix once for the sensitivity and once per iteration
        return {"bytes": a * (1 + case["iters"]), "flops": a / 4 * (1 + 4 * case["iters"])}
    total = {"bytes": 0.0, "flops": 0.0}
    for d in _parts(case):
        p = _problem(d)
        pairs, E = p.n_src * p.n_det, p.nrg_src
        vox = p.nx * p.ny
        nv = 0.4 * vox                       # the phantoms fill about this much
        cells = 0.6 * max(p.nx, p.ny)        # cells a line integral crosses, 30 operations each
        rays = p.rays
        if k == "ct":
            total["bytes"] += 4.0 * (2 * vox + 2 * rays)
            total["flops"] += pairs * (2 * cells * 30.0 + p.nrg_det * (2 * p.dnrg + 1) * 6.0)
            continue
        # the line integral, the geometry, and per source energy the attenuation,
        # the wavevector transfer and the Gaussian bins; the Compton term where there is one
        bins = 8.0
        term = 25.0 + 4.0 * bins + (40.0 if k in ("call", "counts", "matrix", "tables") else 0.0)
        f = pairs * nv * (100.0 + E * term)
        b = 4.0 * (3 * vox + rays)
        if k in ("call", "counts", "matrix", "tables"):
            f += pairs * nv * cells * 30.0
            b += 4.0 * rays
        if k in ("call", "matrix"):
            b += 4.0 * p.amatrix_elems
        if k in ("op_forward", "op_adjoint"):
            b += 8.0 * pairs * nv + 4.0 * vox * p.nwt
        if k == "mlem":
            f *= 2.0 * case["iters"] + 1
            b += (8.0 * pairs * nv + 8.0 * vox * p.nwt + 8.0 * rays) * case["iters"]
        total["bytes"] += b
        total["flops"] += f
    return total


# ---- the outputs in 64 bits ----------------------------------------------------------

_LIMIT = 1.3e11    # Gaussian bins that are worth the wait
_CHUNK = 1 << 23   # (pair, voxel) elements at a time


class _Model:
    """The forward model in 64 bits on one problem, a chunk of (source, pixel)
    pairs at a time: arrays [pairs, voxels]."""

    def __init__(self, inp):
        p = self.p = inp.problem
        f64 = dict(device=DEV, dtype=torch.float64)

        def t(a):
            return torch.as_tensor(np.asarray(a), device=DEV).to(torch.float64)
        self.inp = inp
        self.a1, self.a2 = t(inp.a1).reshape(p.ny, p.nx), t(inp.a2).reshape(p.ny, p.nx)
        pad = torch.zeros(p.ny + 2, p.nx + 2, 2, **f64)
        pad[1:-1, 1:-1, 0], pad[1:-1, 1:-1, 1] = self.a1, self.a2
        self.map = pad.reshape(-1, 2)
        seg = np.asarray(inp.seg).reshape(p.ny, p.nx).T          # [x, y]: x outer, y inner
        on = np.argwhere(seg > 0)
        self.ix, self.iy = on[:, 0], on[:, 1]
        self.mat = torch.as_tensor(seg[on[:, 0], on[:, 1]] - 1, device=DEV).long()
        self.vx, self.vy = t(on[:, 0]) + 0.5, t(on[:, 1]) + 0.5
        self.nv = len(on)
        self.spec = t(inp.spectrum).reshape(p.nrg_det, p.nrg_src)    # [n, e]
        phi = np.arange(p.n_src) / p.n_src * p.src_arc + p.src_phi0
        self.sphi, self.cphi = t(np.sin(phi)), t(np.cos(phi))
        self.dEs, self.dEd = (p.e_src_max - p.e_src_min) / p.nrg_src, (p.e_det_max - p.e_det_min) / p.nrg_det
        same = p.nrg_src == p.nrg_det and p.e_src_min == p.e_det_min and p.e_src_max == p.e_det_max
        self.win = []
        for n in range(p.nrg_det):
            c = n if same else int(math.floor((p.e_det_min + (n + 0.5) * self.dEd - p.e_src_min) / self.dEs))
            lo = max(0, c - p.dnrg)
            hi = lo + 2 * p.dnrg
            if hi >= p.nrg_src:
                hi = p.nrg_src - 1
                lo = hi - 2 * p.dnrg
            self.win.append((lo, hi))
        self.e_lo, self.e_hi = min(w[0] for w in self.win), max(w[1] for w in self.win)
        self.pairs = p.n_src * p.n_det
        k = np.arange(p.nwt + 1, dtype=np.float64)
        edge = p.q_lo + k * p.dq0 + (p.q_hi - p.q_lo - p.dq0 * p.nwt) * k * k / (p.nwt * p.nwt)
        self.qk, self.dqk = 0.5 * (edge[1:] + edge[:-1]), np.diff(edge)
        # the response of detector bin n to source bin e inside its window
        self.rf = torch.zeros(p.nrg_det, p.nrg_src, **f64)
        for n, (lo, hi) in enumerate(self.win):
            self.rf[n, lo:hi + 1] = self.spec[n, lo:hi + 1]

    def compton_columns(self):
        p = self.p
        if p.quirks & 1:
            x = torch.cat([torch.zeros(1, device=DEV, dtype=torch.float64), self.vx[:-1]])
            y = torch.cat([torch.zeros(1, device=DEV, dtype=torch.float64), self.vy[:-1]])
        else:
            x, y = self.vx, self.vy
        v = self.sample(x, y)
        return v[..., 1], torch.log2(torch.abs(v[..., 0] / v[..., 1]))

    def sample(self, x, y):
        """The map at (x, y), bilinear between texel centres, 0 outside."""
        p = self.p
        x, y = x - 0.5, y - 0.5
        i, j = torch.floor(x), torch.floor(y)
        fx, fy = (x - i).unsqueeze(-1), (y - j).unsqueeze(-1)
        i = (i.long() + 1).clamp_(0, p.nx)
        o = (j.long() + 1).clamp_(0, p.ny) * (p.nx + 2) + i
        m = self.map
        lo = m[o] * (1 - fx) + m[o + 1] * fx
        o = o + (p.nx + 2)
        hi = m[o] * (1 - fx) + m[o + 1] * fx
        return lo * (1 - fy) + hi * fy

    def samples(self, L):
        p = self.p
        cap = math.ceil(math.sqrt(p.nx * p.nx + p.ny * p.ny) / (p.dq_step * p.nwt)) * p.nwt
        n = torch.floor(L / p.dq_step)
        n = torch.where((n + 1) * p.dq_step <= L, n + 1, n)
        n = torch.where(n * p.dq_step <= L, n, n - 1) + 1
        return n.clamp(max=cap).long()

    def walk(self, rx, ry, ux, uy, n):
        """DQ times the sum of the samples at r + u DQ k, k < n."""
        dq = self.p.dq_step
        acc = torch.zeros(*rx.shape, 2, device=DEV, dtype=torch.float64)
        for k in range(int(n.max()) if n.numel() else 0):
            v = self.sample(rx + ux * (dq * k), ry + uy * (dq * k))
            acc += v * (n > k).unsqueeze(-1)
        return acc * dq

    def integral(self, ex, ey, vx, vy):
        """The line integral from where the ray enters the phantom to the voxel."""
        p = self.p
        eps = float(np.float32(0.00001))
        X = [(0.0, p.nx), (p.nx, p.nx), (p.nx, 0.0), (0.0, 0.0)]
        Y = [(0.0, 0.0), (0.0, p.ny), (p.ny, p.ny), (p.ny, 0.0)]
        dx, dy = vx - ex, vy - ey
        rx = torch.full_like(dx, math.nan)
        ry = rx.clone()
        for (x3, x4), (y3, y4) in zip(X, Y):
            a, b = float(x4 - x3), float(y4 - y3)
            den = a * dy - dx * b
            ua = (a * (y3 - ey) - (x3 - ex) * b) / den
            ub = (dx * (y3 - ey) - (x3 - ex) * dy) / den
            ok = (den.abs() > eps) & (ua > -eps) & (ua < 1 + eps) & (ub > -eps) & (ub < 1 + eps) & rx.isnan()
            rx, ry = torch.where(ok, ex + dx * ua, rx), torch.where(ok, ey + dy * ua, ry)
        Lx, Ly = vx - rx, vy - ry
        L2 = Lx * Lx + Ly * Ly
        L, r = torch.sqrt(L2), 1.0 / torch.sqrt(L2)
        miss = L.isnan()
        n = torch.where(miss, torch.zeros_like(L).long(), self.samples(torch.where(miss, torch.zeros_like(L), L)))
        z = torch.zeros_like(L)
        return self.walk(torch.where(miss, z, rx), torch.where(miss, z, ry), torch.where(miss, z, Lx * r),
                         torch.where(miss, z, Ly * r), n)

    def chunks(self):
        step = max(1, _CHUNK // max(1, self.nv))
        src_side = torch.stack([self.integral(self.p.cx + self.p.r_src * self.sphi[s], self.p.cy - self.p.r_src * self.cphi[s],
                                              self.vx, self.vy) for s in range(self.p.n_src)])
        for q in range(0, self.pairs, step):
            yield torch.arange(q, min(self.pairs, q + step), device=DEV), src_side

    def geometry(self, pr, src_side):
        """What the term of (pair, voxel) needs at every energy."""
        p = self.p
        src, det = pr % p.n_src, pr // p.n_src
        col, row = det % p.n_col, det // p.n_col
        s, c = self.sphi[src][:, None], self.cphi[src][:, None]
        rdet = ((col.double() - p.n_col / 2.0 + 0.5) * p.col_pitch)[:, None]
        dx, dy = p.cx - p.r_det * s + rdet * c, p.cy + p.r_det * c + rdet * s
        dz = (p.z0 + row.double() * p.row_pitch)[:, None]
        vx, vy = self.vx[None, :], self.vy[None, :]
        ax, ay = vx - (p.cx + p.r_src * s), vy - (p.cy - p.r_src * c)
        sta, cta = math.sin(p.target_angle), math.cos(p.target_angle)
        nsx, nsy, nsz = -s * sta, c * sta, -cta
        proj = (ax * nsx + ay * nsy) / torch.sqrt(nsx * nsx + nsy * nsy)
        az, H = -proj * math.tan(p.wedge_angle / 2.0), proj * math.tan(p.wedge_angle)
        bx, by, bz = dx - vx, dy - vy, dz - az
        ab = ax * bx + ay * by + az * bz
        an, bn = ax * ax + ay * ay + az * az, bx * bx + by * by + bz * bz
        cos = ab / torch.sqrt(an) / torch.sqrt(bn)
        g = {"cos2": cos * cos, "omc": 1.0 - cos, "s": torch.sqrt(torch.abs(1.0 - cos) / 2.0)}
        S = [b - ab * a / an for a, b in ((ax, bx), (ay, by), (az, bz))]
        D = [-a + ab * b / bn for a, b in ((ax, bx), (ay, by), (az, bz))]
        V = [-(u + v) for u, v in zip(S, D)]
        Dn = D[0] * s - D[1] * c
        Sn = S[0] * nsx + S[1] * nsy + S[2] * nsz
        dD = (D[0] ** 2 + D[1] ** 2 + D[2] ** 2 - Dn * Dn) * (p.col_pitch * p.row_pitch) / 12.0
        vV = (p.vox_side ** 2 * (V[0] ** 2 + V[1] ** 2) + H * H * V[2] ** 2) / 12.0
        sS = (S[0] ** 2 + S[1] ** 2 + S[2] ** 2 - Sn * Sn) * p.focal_spot ** 2 / 12.0
        g["blur"] = (sS + vV + dD) / an / bn
        geom = (-s * ax + c * ay) / torch.sqrt(ax * ax + ay * ay) / torch.sqrt(an) * math.tan(p.wedge_angle)
        g["geom"] = geom * -(s * bx - c * by) / torch.sqrt(bn ** 3)
        g["ray"] = (1.0 + cos * cos) / 2.0
        g["Ad"] = self.integral(dx.expand_as(ab), dy.expand_as(ab), vx.expand_as(ab), vy.expand_as(ab))
        g["As"] = src_side[src]
        return g

    def energy(self, g, e):
        p = self.p
        E1 = p.e_src_min + e * self.dEs
        E2 = p.e_src_min + (e + 1) * self.dEs
        E = 0.5 * (E1 + E2)
        ein = E / p.mec2
        f1, f2 = ein ** 3, p.kn0 + p.kn1 * ein + p.kn2 * ein * ein
        t = {"E1": E1, "E2": E2, "ein": ein, "w": 2.0 * E / p.hbarc * g["s"]}
        t["s2"] = (2.0 * g["s"] / p.hbarc) ** 2 * self.dEs ** 2 / 12.0 + (E / p.hbarc) ** 2 * g["blur"] / (2.0 * g["s"]) ** 2
        Ad, As = g["Ad"], g["As"]
        t["Pin"] = torch.exp(-(Ad[..., 0] / f1 + Ad[..., 1] / f2))
        t["PP"] = t["Pin"] * torch.exp(-(As[..., 0] / f1 + As[..., 1] / f2))
        t["pref"] = t["PP"] * g["geom"] * g["ray"] * p.rsqrt2pi / torch.sqrt(t["s2"])
        return t

    def fine_sum(self, t):
        """Sum over the fine bins of Gaussian times pattern (bins beyond 9 sigma add below 1e-17 of the peak)."""
        p = self.p
        dq = (p.q_hi - p.q_lo) / p.nqf
        I = torch.as_tensor(np.asarray(self.inp.Ifine), device=DEV).double().reshape(p.n_mat, p.nqf)
        w, c = t["w"], -0.5 / t["s2"]
        H = math.ceil(9.0 * float(torch.sqrt(t["s2"].max())) / dq) + 1
        acc = torch.zeros_like(w)
        if 2 * (2 * H + 1) >= p.nqf:
            for j in range(p.nqf):
                d = w - (p.q_lo + dq * (0.5 + j))
                acc += torch.exp(d * d * c) * I[:, j][self.mat][None, :]
        else:
            pad = torch.zeros(p.n_mat, p.nqf + 2, device=DEV, dtype=torch.float64)
            pad[:, 1:-1] = I
            jc = torch.floor((w - p.q_lo) / dq)
            base = (self.mat * (p.nqf + 2))[None, :]
            for o in range(-H, H + 1):
                j = jc + o
                d = w - (p.q_lo + dq * (0.5 + j))
                acc += torch.exp(d * d * c) * pad.reshape(-1)[base + (j.clamp(-1, p.nqf).long() + 1)]
        return acc * dq

    def u8(self, S):
        p = self.p
        return torch.floor(torch.as_tensor(np.asarray(S), device=DEV).double()).clamp_(0, 255).reshape(p.na, p.nq)

    def lookup(self, S, l2w, la, bilinear):
        """A table [na, nq] at log2 coordinates [pairs, voxels] and [voxels]."""
        p, i = self.p, self.inp
        q0, q1, a0, a1 = i.q_min, i.q_max, i.a_min, i.a_max
        if not bilinear:
            jq = torch.floor((l2w - q0) / ((q1 - q0) / p.nq)).clamp_(0, p.nq - 1).long()
            ja = torch.floor((la - a0) / ((a1 - a0) / p.na)).nan_to_num_(0.0).clamp_(0, p.na - 1).long()
            return S[ja[None, :].expand_as(jq), jq]
        tq = ((l2w - q0) / ((q1 - q0) / (p.nq - 1))).clamp(0, p.nq - 1)
        ta = ((la - a0) / ((a1 - a0) / (p.na - 1))).nan_to_num(0.0).clamp(0, p.na - 1)[None, :].expand_as(tq)
        jq, ja = tq.floor().clamp_(max=p.nq - 2), ta.floor().clamp_(max=p.na - 2)
        f, g = tq - jq, ta - ja
        jq, ja = jq.long(), ja.long()
        return (1 - g) * ((1 - f) * S[ja, jq] + f * S[ja, jq + 1]) + g * ((1 - f) * S[ja + 1, jq] + f * S[ja + 1, jq + 1])

    def counts(self, S1=None, bilinear=False, matrix=False):
        """Coherent counts, Compton counts and the model matrix (or None), flat in the library's layouts."""
        p = self.p
        f64 = dict(device=DEV, dtype=torch.float64)
        a2, la = self.compton_columns()
        S2 = self.u8(self.inp.S2)
        T1 = self.u8(S1) if S1 is not None else None
        N, C = torch.zeros(p.nrg_det, self.pairs, **f64), torch.zeros(p.nrg_det, self.pairs, **f64)
        A = torch.zeros(p.nrg_det, self.pairs, p.n_mat, p.nwt, **f64) if matrix else None
        one = torch.nn.functional.one_hot(self.mat, p.n_mat).double()
        for pr, src_side in self.chunks():
            g = self.geometry(pr, src_side)
            for e in range(self.e_lo, self.e_hi + 1):
                t = self.energy(g, e)
                rf = self.rf[:, e][:, None]
                if T1 is not None:
                    s1 = self.lookup(T1, torch.log2(t["ein"] * g["s"]), la, bilinear)
                    coh = t["PP"] * g["geom"] * g["ray"] * a2[None, :] * s1
                else:
                    coh = t["pref"] * self.fine_sum(t)
                N[:, pr] += rf * coh.sum(1)[None, :]
                if matrix:
                    row = torch.stack([(t["pref"] * torch.exp(-0.5 * (t["w"] - q) ** 2 / t["s2"]) * d) @ one
                                       for q, d in zip(self.qk, self.dqk)], dim=-1)      # [pairs, mat, k]
                    for n, (lo, hi) in enumerate(self.win):
                        if lo <= e <= hi:
                            A[n, pr] += self.rf[n, e] * row
                er = 1.0 + t["ein"] * g["omc"]
                eo = t["ein"] / er
                w = t["ein"] * g["s"]
                s2 = self.lookup(S2, torch.log2(w * torch.sqrt(er + w * w) / er), la, bilinear)
                Pc = torch.exp(-(g["As"][..., 0] / eo ** 3 + g["As"][..., 1] / (p.kn0 + p.kn1 * eo + p.kn2 * eo * eo)))
                com = t["Pin"] * Pc * g["geom"] * a2[None, :] * s2 * er * er * (er + 1.0 / er - 1.0 + g["cos2"]) / 2.0
                o1, o2 = t["E1"] / er, t["E2"] / er
                com = com / (o2 - o1)
                for n, (lo, hi) in enumerate(self.win):
                    if lo <= e <= hi:
                        d1, d2 = p.e_det_min + n * self.dEd, p.e_det_min + (n + 1) * self.dEd
                        m = (torch.clamp(o2, max=d2) - torch.clamp(o1, min=d1)).clamp_(min=0.0)
                        C[n, pr] += self.rf[n, e] * (m * com).sum(1)
        return N.reshape(-1), C.reshape(-1), A.reshape(-1) if matrix else None

    def bins(self):
        return float(self.pairs) * self.nv * (self.e_hi - self.e_lo + 1)

    # one pattern per voxel: U[pair, e] = sum_{v,k} M x, and its transpose
    def vox(self, x=None, u=None):
        p = self.p
        E = range(self.e_lo, self.e_hi + 1)
        T = torch.zeros(p.nrg_src, self.pairs, device=DEV, dtype=torch.float64)
        G = torch.zeros(p.nwt, self.nv, device=DEV, dtype=torch.float64)
        for pr, src_side in self.chunks():
            g = self.geometry(pr, src_side)
            for e in E:
                t = self.energy(g, e)
                c = -0.5 / t["s2"]
                for k in range(p.nwt):
                    m = t["pref"] * torch.exp((t["w"] - self.qk[k]) ** 2 * c) * self.dqk[k]
                    if x is not None:
                        T[e, pr] += m @ x[:, k]
                    if u is not None:
                        G[k] += u[e, pr] @ m
        return T if x is not None else G.T

    def compact(self, x):
        p = self.p
        return x.double().reshape(p.ny, p.nx, p.nwt)[torch.as_tensor(self.iy), torch.as_tensor(self.ix)]

    def spread(self, g):
        p = self.p
        out = torch.zeros(p.ny, p.nx, p.nwt, device=DEV, dtype=torch.float64)
        out[torch.as_tensor(self.iy), torch.as_tensor(self.ix)] = g
        return out.reshape(-1)

    def ct(self):
        p = self.p
        pr = torch.arange(self.pairs, device=DEV)
        src, det = pr % p.n_src, pr // p.n_src
        s, c = self.sphi[src], self.cphi[src]
        rdet = ((det % p.n_col).double() - p.n_col / 2.0 + 0.5) * p.col_pitch
        sx, sy = p.cx + p.r_src * s, p.cy - p.r_src * c
        ex, ey = p.cx - p.r_det * s + rdet * c - sx, p.cy + p.r_det * c + rdet * s - sy
        t0, t1 = torch.zeros_like(ex), torch.ones_like(ex)
        for o, d, hi in ((sx, ex, p.nx), (sy, ey, p.ny)):
            z = d == 0
            ta, tb = (0.0 - o) / d, (float(hi) - o) / d
            ta, tb = torch.minimum(ta, tb), torch.maximum(ta, tb)
            t0 = torch.where(z, t0, torch.maximum(t0, ta))
            t1 = torch.where(z, torch.where((o < 0) | (o > hi), torch.full_like(t1, -1.0), t1), torch.minimum(t1, tb))
        length = torch.sqrt(ex * ex + ey * ey)
        hit = t1 > t0
        n = torch.where(hit, self.samples(torch.where(hit, (t1 - t0) * length, torch.zeros_like(t0))), 0 * det)
        A = self.walk(sx + t0 * ex, sy + t0 * ey, ex / length, ey / length, n)
        T = torch.zeros(p.nrg_det, self.pairs, device=DEV, dtype=torch.float64)
        for e in range(self.e_lo, self.e_hi + 1):
            ein = (p.e_src_min + (e + 0.5) * self.dEs) / p.mec2
            a = torch.exp(-(A[:, 0] / ein ** 3 + A[:, 1] / (p.kn0 + p.kn1 * ein + p.kn2 * ein * ein)))
            T += self.rf[:, e][:, None] * a[None, :]
        G = self.rf.sum(1)[:, None].expand_as(T)
        return T.reshape(-1), G.reshape(-1).clone()


def _fold(x, g, s):
    x = x * g / (s + 1e-7)
    return torch.where(torch.isfinite(x), x, torch.zeros_like(x)).clamp_(min=0.0)


def exact(case, seed):
    k = case["kind"]
    if k == "basis":
        return (_rand(seed, (case["M"], case["K"]), 0.0, 1.0).double()
                @ _rand(seed + 1, (case["K"], case["N"]), 0.0, 1.0).double())
    if k == "matrix_mlem":
        A, y, c, x = (v.double() for v in _matrix_data(case, seed))
        s = A.sum(0)
        for _ in range(case["iters"]):
            x = _fold(x, A.T @ (y / (A @ x + c + 1e-20)), s)
        return x
    inps = _inputs(case, seed)
    m = [_Model(i) for i in inps]
    p = m[0].p
    if k == "ct":
        return m[0].ct()
    per = {"counts": min(p.nqf, 40), "call": p.nqf + p.nwt, "matrix": p.nqf + p.nwt, "tables": 4,
           "op_forward": p.nwt, "op_adjoint": p.nwt, "mlem": 4 * p.nwt}[k]
    if sum(q.bins() for q in m) * per > _LIMIT:
        return None
    if k == "tables":
        return m[0].counts(S1=_table(p, seed), bilinear=case["bilinear"])[:2]
    if k == "counts":
        return m[0].counts()[:2]
    if k == "matrix":
        return m[0].counts(matrix=True)
    if k == "call":
        N, C, A = (v.cpu().numpy() for v in m[0].counts(matrix=True))
        shp = (p.n_src, p.n_col, p.n_row, p.nrg_det)
        return (N.reshape(shp, order="F"), C.reshape(shp, order="F"), A.reshape((p.nwt, p.n_mat) + shp, order="F"))
    if k == "op_forward":
        T = m[0].vox(x=m[0].compact(_rand(seed + 1, p.nx * p.ny * p.nwt, 0.0, 1.0)))
        return (m[0].rf @ T).reshape(-1)
    if k == "op_adjoint":
        w = _rand(seed + 1, p.rays, 0.0, 2.0).double().reshape(p.nrg_det, -1)
        return m[0].spread(m[0].vox(u=m[0].rf.T @ w))
    out = []
    for q, y, c, x in zip(m, *_mlem_data(case, seed, inps)):
        y, c, x = y.double().reshape(q.p.nrg_det, -1), c.double().reshape(q.p.nrg_det, -1), q.compact(x)
        s = q.vox(u=q.rf.T @ torch.ones_like(y))
        for _ in range(case["iters"]):
            x = _fold(x, q.vox(u=q.rf.T @ (y / (q.rf @ q.vox(x=x) + c + 1e-20))), s)
        out.append(q.spread(x))
    return out
