"""The work that users of this library have it do, as measurable cases.

Every case goes through the public Python interface of sgpp_gb300, the mirror of pysgpp's operator
interface, on synthetic data. A case is a dict of plain values:

  op         "mult", "multT", "system"  one product of an operator that the program keeps, on device
                                        vectors (multDevice, multTransposeDevice, systemApplyDevice)
             "host"      SystemMatrixLeastSquaresIdentity.mult on host vectors: what SG++'s own CG
                         loop calls in every iteration
             "predict"   a model applied to new samples: operator created on them, mult, closed
             "fit"       a mixed-precision regression fit on resident data (fitDevice)
             "request"   a fit request as the fit server handles it: operator created from host
                         data, mixed fit, alpha on the host, closed
             "fitblock"  16 regression fits that share grid and data (fitBlockDevice)
  basis      "linear" or "modlinear";  d, level: the regular sparse grid;  rounds: surplus-refinement
             rounds of 40 points each on top of it (spatially adaptive grids)
  m          data points;  data: "uniform" or "mixture" (8 Gaussian clusters clipped to the cube)
  precision  the operator's "precision" parameter: "double" (the default), "df64" or "float"

Results of the "float" products and of the fits are kept as FP32 by the program: the former are
computed in single precision, and a fit's alpha is good to its tolerance (about 1e-7 relative). The
"double" and "df64" products keep all 64 bits.
"""
import math

import numpy as np
import torch

import sgpp_gb300 as sg

LAMBDA, EPSILON = 1e-4, 1e-8
POINTS_PER_ROUND = 40
RHS = 16


def _case(name, op, d, level, m, precision="double", basis="linear", data="uniform", rounds=0):
    return {"name": name, "op": op, "d": d, "level": level, "m": m, "precision": precision,
            "basis": basis, "data": data, "rounds": rounds}


def listed():
    return [
        # a user's first script: SG++'s CG loop driving the operator on host vectors, small problem
        # (the size of the library's smoke test); launches, copies and synchronisations count
        _case("host_cg_step", "host", 5, 4, 3000),
        # the plain method at its usual size: default operator, d=5 level 6, 65,536 points
        _case("mult_double", "mult", 5, 6, 65536),
        _case("multt_double", "multT", 5, 6, 65536),
        # system product of a plain FP64 fit on a spatially adaptive grid: d=8 level 4 after six
        # refinement rounds, 2^19 points
        _case("system_adaptive", "system", 8, 4, 524288, rounds=6),
        # single-precision products on the regression workload's grid, a quarter of its points and
        # a ragged count
        _case("mult_float", "mult", 10, 5, 262147, "float", data="mixture"),
        _case("multt_float", "multT", 10, 5, 262147, "float", data="mixture"),
        # FP64-accurate float-float operator on a ModLinear grid (boundary-adjacent ramps)
        _case("system_modlinear", "system", 6, 5, 100003, "df64", "modlinear"),
        # FP64-accurate product on a large grid of the batched mix: many subspaces of many cells
        _case("mult_large_grid", "mult", 9, 6, 40961, "df64"),
        # a model with known surpluses applied to a file's worth of new samples, whole call
        _case("predict", "predict", 6, 4, 10001),
        # one request of the fit server, whole call
        _case("request", "request", 6, 5, 20011),
        # one problem of the batched mix: 16 targets on the tensor cores
        _case("fitblock", "fitblock", 7, 5, 60007),
        # the regression workload: d=10 level 5, 2^20 points, mixed-precision fit to 1e-8
        _case("fit_regression", "fit", 10, 5, 1048576, data="mixture"),
    ]


def _subspaces(c):
    return math.comb(c["d"] + c["level"] - 1, c["d"])


def _points(c):
    return sum(math.comb(c["d"] - 1 + k, k) << k for k in range(c["level"]))


def draw(rng):
    """One more case of the same operations over the size mix of the batched and serving
    configurations (d in 2..12, level in 3..7, m log-uniform), none larger than the largest above."""
    op = rng.choice(["mult", "multT", "system", "mult", "multT", "system", "host", "predict", "fit",
                     "request", "fitblock"])
    while True:
        c = {"op": op, "d": rng.randint(2, 12), "level": rng.randint(3, 7),
             "m": int(2.0 ** rng.uniform(10.0, 20.0)) | rng.randint(0, 1), "precision": "double",
             "basis": "linear", "data": rng.choice(["uniform", "mixture"]), "rounds": 0}
        if op in ("mult", "multT", "system"):
            c["precision"] = rng.choice(["double", "df64", "float"])
            c["basis"] = rng.choice(["linear", "linear", "modlinear"])
        if op in ("mult", "multT", "system") and c["level"] <= 4:
            c["rounds"] = rng.choice([0, 3, 6])
        units, dense = _subspaces(c) * c["m"], float(_points(c)) * c["m"] * c["d"]
        if _points(c) > 60000:
            continue
        if c["precision"] == "double" and op not in ("fit", "request", "fitblock"):
            if dense > 1.6e10 / (1 + 3 * (c["rounds"] > 0)):
                continue
        elif op in ("mult", "multT", "system"):
            if units > 5e8 or dense > 1e11:
                continue
        elif units > (3e8 if op == "fit" else 6e7) or dense > 3e10:
            continue
        if op in ("host", "predict", "request") and c["m"] > 200000:
            continue
        if op == "fitblock" and (c["d"] < 4 or c["level"] < 4):
            continue
        return c


def _grid(case):
    d = case["d"]
    grid = (sg.Grid.createModLinearGrid(d) if case["basis"] == "modlinear"
            else sg.Grid.createLinearGrid(d))
    grid.getGenerator().regular(case["level"])
    rng = np.random.default_rng(case["rounds"])  # the same grid for every data set
    for _ in range(case["rounds"]):
        # surpluses of a smooth target: they fall by about 4 per level
        st = grid.getStorage()
        alpha = rng.standard_normal(grid.getSize()) * 0.25 ** (st.level.sum(axis=1) - d)
        grid.getGenerator().refine(sg.SurplusRefinementFunctor(alpha, POINTS_PER_ROUND, 0.0))
    return grid


def _data(case, seed):
    """The data matrix [m x d] and a random generator for the vectors, on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    m, d = case["m"], case["d"]
    f64 = {"generator": g, "device": "cuda", "dtype": torch.float64}
    if case["data"] == "uniform":
        return torch.rand(m, d, **f64), f64
    means = 0.2 + 0.6 * torch.rand(8, d, **f64)
    comp = torch.randint(0, 8, (m,), generator=g, device="cuda")
    return (means[comp] + 0.08 * torch.randn(m, d, **f64)).clamp(0.0, 1.0), f64


def _target(x, f64):
    """A smooth function of the first coordinates plus noise."""
    y = 10.0 * torch.sin(math.pi * x[:, 0] * x[:, 1]) + 20.0 * (x[:, -1] - 0.5) ** 2
    return y + 0.1 * torch.randn(x.shape[0], **f64)


def _inputs(case, seed):
    """grid, data and the input vector (or the targets) of a case, from the seed alone."""
    grid = _grid(case)
    x, f64 = _data(case, seed)
    op = case["op"]
    if op in ("fit", "request"):
        return grid, x, _target(x, f64)
    if op == "fitblock":
        y = _target(x, f64)
        return grid, x, torch.stack([y + torch.randn(y.shape[0], **f64) for _ in range(RHS)])
    return grid, x, torch.randn(case["m"] if op == "multT" else grid.getSize(), **f64)


def _config(case):
    parameters = {"precision": case["precision"]}
    if case["op"] == "fitblock":
        parameters["algo"] = "subspace"  # the block products need the subspace form
    return sg.OperationMultipleEvalConfiguration(
        sg.OperationMultipleEvalType.STREAMING, sg.OperationMultipleEvalSubType.CUDA,
        parameters=parameters)


def prepare(case, seed):
    grid, x, v = _inputs(case, seed)
    op, n, m = case["op"], grid.getSize(), case["m"]
    s = {"op": op, "case": case, "grid": grid, "m": m, "n": n}
    if op in ("host", "predict", "request"):
        s["x"], s["v"] = x.cpu().numpy(), v.cpu().numpy()
        s["out"] = np.zeros(m if op == "predict" else n)
        if op == "host":
            s["system"] = sg.SystemMatrixLeastSquaresIdentity(grid, s["x"], LAMBDA)
        return s
    s["b"] = sg.createOperationMultipleEval(grid, x.cpu().numpy(), _config(case))
    s["v"] = v
    shape = {"mult": (m,), "fitblock": (RHS, n)}.get(op, (n,))
    s["out"] = torch.zeros(shape, dtype=torch.float64, device="cuda")
    s["narrow"] = (torch.zeros(shape, dtype=torch.float32, device="cuda")
                   if case["precision"] == "float" or op in ("fit", "fitblock") else None)
    s["stream"] = torch.cuda.Stream()
    s["b"].setStream(s["stream"].cuda_stream)
    torch.cuda.synchronize()
    return s


def run(s):
    op = s["op"]
    if op == "host":
        s["system"].mult(s["v"], s["out"])
        return s["out"]
    if op == "predict":
        b = sg.createOperationMultipleEval(s["grid"], s["x"], _config(s["case"]))
        b.mult(s["v"], s["out"])
        b.close()
        return s["out"]
    if op == "request":
        b = sg.createOperationMultipleEval(s["grid"], s["x"], _config(s["case"]))
        alpha, _, _ = b.fit(s["v"], LAMBDA, 100000, EPSILON, mode=sg.SGMEV_SOLVE_MIXED)
        b.close()
        return alpha.astype(np.float32)
    b, v, out = s["b"], s["v"].data_ptr(), s["out"].data_ptr()
    if op == "mult":
        b.multDevice(v, out)
    elif op == "multT":
        b.multTransposeDevice(v, out)
    elif op == "system":
        b.systemApplyDevice(v, out, LAMBDA * s["m"])
    elif op == "fit":
        b.fitDevice(v, out, LAMBDA, 100000, EPSILON, mode=sg.SGMEV_SOLVE_MIXED)
    else:
        b.fitBlockDevice(v, out, LAMBDA, 100000, EPSILON)
    if s["narrow"] is None:
        return s["out"]
    with torch.cuda.stream(s["stream"]):
        return s["narrow"].copy_(s["out"])


def work(case):
    """Every input read once and every output written once; per data point and subspace (one basis
    function of it is not zero) a multiply-add, in both products of each CG iteration of a fit."""
    m, n, op = case["m"], _points(case), case["op"]
    units = float(_subspaces(case)) * m
    if op in ("fit", "request", "fitblock"):
        k = RHS if op == "fitblock" else 1
        return {"bytes": 8.0 * (m * case["d"] + k * (m + n)), "flops": 4.0 * units * 75 * k}
    both = op in ("system", "host")
    return {"bytes": 8.0 * (m * case["d"] + (2 * n if both else m + n)),
            "flops": (4.0 if both else 2.0) * units}


# ---- the same results in 64 bits, by plain torch -------------------------------------------------
class _Exact:
    """B in FP64: per subspace the value of its one basis function at every point, and the grid
    point that it belongs to (grid points of one level vector have disjoint supports)."""

    def __init__(self, grid, x, keep):
        st = grid.getStorage()
        level, index = np.asarray(st.level), np.asarray(st.index)
        self.x, self.n, self.mod = x, level.shape[0], grid.getType() == sg.GridType.ModLinear
        rows, which = np.unique(level, axis=0, return_inverse=True)
        which = np.asarray(which).reshape(-1)
        order = np.argsort(which, kind="stable")
        cut = np.searchsorted(which[order], np.arange(rows.shape[0] + 1))
        self.sub = []
        for k in range(rows.shape[0]):
            g = order[cut[k]:cut[k + 1]]
            size = 1 << (rows[k] - 1)
            flat = np.zeros(g.size, np.int64)
            for t in range(rows.shape[1]):
                flat = flat * size[t] + (index[g, t] - 1) // 2
            table = np.full(int(np.prod(size)), -1, np.int64)
            table[flat] = g
            self.sub.append((rows[k], torch.from_numpy(table).cuda()))
        self.spread = torch.arange(x.shape[0], device="cuda") % 128
        self.kept = [self._column(*s) for s in self.sub] if keep else None

    def _column(self, lev, table):
        m = self.x.shape[0]
        val = torch.ones(m, dtype=torch.float64, device="cuda")
        cell = torch.zeros(m, dtype=torch.int64, device="cuda")
        for t, l in enumerate(lev.tolist()):
            x, scale, last = self.x[:, t], float(1 << l), (1 << (l - 1)) - 1
            k = (x * (scale / 2)).floor().clamp(0, last)
            cell = cell * (last + 1) + k.to(torch.int64)
            if self.mod and l == 1:
                continue
            h = 1.0 - (x * scale - (2.0 * k + 1.0)).abs()
            if self.mod:
                h = torch.where(k == 0, 2.0 - x * scale, h)
                h = torch.where(k == last, x * scale - (2.0 * last), h)
            val = val * h.clamp(min=0.0)
        g = table[cell]
        return (torch.where(g >= 0, val, torch.zeros_like(val)), g.clamp(min=0), cell.to(torch.int32))

    def _columns(self):
        for k, s in enumerate(self.sub):
            yield s[1], (self.kept[k] if self.kept is not None else self._column(*s))

    def mult(self, a):
        out = torch.zeros(a.shape[:-1] + (self.x.shape[0],), dtype=torch.float64, device="cuda")
        for _, (val, g, _) in self._columns():
            out += a[..., g] * val
        return out

    def mult_transpose(self, v):
        out = torch.zeros(v.shape[:-1] + (self.n,), dtype=torch.float64, device="cuda")
        for table, (val, _, cell) in self._columns():
            # spread over 128 bins per cell, so that the additions do not queue at one address
            bins = torch.zeros(v.shape[:-1] + (table.numel() * 128,), dtype=torch.float64,
                               device="cuda")
            bins.index_add_(-1, cell.to(torch.int64) * 128 + self.spread, v * val)
            sums = bins.view(v.shape[:-1] + (table.numel(), 128)).sum(-1)
            real = table >= 0
            out[..., table[real]] = sums[..., real]
        return out

    def fit(self, y, lam_m):
        """Conjugate gradients to a relative residual of 1e-13, every column by itself."""
        b = self.mult_transpose(y)
        x, r = torch.zeros_like(b), b.clone()
        p, rr = r.clone(), (r * r).sum(-1, keepdim=True)
        stop = rr * 1e-26
        for _ in range(1000):
            if bool((rr <= stop).all()):
                break
            q = self.mult_transpose(self.mult(p)) + lam_m * p
            step = torch.where(rr > stop, rr / (p * q).sum(-1, keepdim=True), torch.zeros_like(rr))
            x += step * p
            r -= step * q
            new = (r * r).sum(-1, keepdim=True)
            p = r + torch.where(rr > stop, new / rr, torch.zeros_like(rr)) * p
            rr = new
        return x


def exact(case, seed):
    op = case["op"]
    fits = op in ("fit", "request", "fitblock")
    columns = RHS if op == "fitblock" else 1
    if fits and float(_subspaces(case)) * case["m"] * columns > 5e8:
        return None  # the regression workload: 45 seconds
    grid, x, v = _inputs(case, seed)
    e = _Exact(grid, x, keep=fits)
    if op in ("mult", "predict"):
        return e.mult(v)
    if op == "multT":
        return e.mult_transpose(v)
    if op in ("system", "host"):
        return e.mult_transpose(e.mult(v)) + LAMBDA * case["m"] * v
    return e.fit(v, LAMBDA * case["m"])
