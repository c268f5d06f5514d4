"""The workloads this framework is timed on, through its public entry points.

``listed()`` names them, ``draw()`` gives more of the same ranges,
``prepare()`` makes what a program holds before the call (inputs from a seed,
buffers, stencils, operators), ``run()`` is one pass, ``work()`` its
compulsory bytes and operations and ``exact()`` its result in plain 64-bit
torch, without the library.

Kinds of pass:

* ``operator``  stencil search, then the fixed-width assembly of a node set's
                weights, inputs and outputs on the device
* ``knn``       the stencil search alone
* ``uneven``    the assembly of a ragged CSR batch of mixed sizes and degrees
* ``host``      search and assembly from host arrays to host arrays
* ``spmv``      an assembled operator applied to a field, with boundary rows
* ``solve``     BiCGSTAB on an assembled Laplacian with Dirichlet rows
* ``lbm``       a semi-Lagrangian lattice Boltzmann step through assembled
                interpolation operators
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "gpu-assembly_b200"))

import rbf_b200 as R  # noqa: E402
from rbf_b200 import nodesets as NS  # noqa: E402

OMEGA = 1.5  # relaxation rate of the lattice Boltzmann step
TOL = 1e-10  # relative residual of a solve that runs to convergence


def listed():
    return [
        # the smallest node set of the test-suite: a call dominated by launches
        dict(name="operator_small", kind="operator", geometry="square", n=4761, k=21, degree=2,
             precision="fp64", nrhs=3),
        # a node set of the size one solver subdomain has, odd count, Laplacian only
        dict(name="operator_disk_60k", kind="operator", geometry="disk", n=60013, k=28, degree=3,
             precision="fp64", nrhs=1),
        # the benchmark's workload: one large periodic node set
        dict(name="operator_periodic_1m", kind="operator", geometry="periodic", n=1048576, k=35,
             degree=3, precision="fp64", nrhs=3),
        # the refined form (FP32 factors, FP64 refinement)
        dict(name="operator_refined_250k", kind="operator", geometry="periodic", n=250000, k=35,
             degree=3, precision="fp32_ir", nrhs=3),
        # high order: variable density, large ill-conditioned systems
        dict(name="operator_bump_150k", kind="operator", geometry="bump", n=150001, k=64, degree=4,
             precision="fp64", nrhs=3),
        # the search alone, on the open plane (renewed stencils of moving nodes)
        dict(name="knn_disk_1m", kind="knn", geometry="disk", n=1000003, k=21),
        # boundary-refined stencils: mixed sizes and degrees in one batch
        dict(name="uneven_disk_500k", kind="uneven", n=500009),
        # a program whose arrays live on the host
        dict(name="host_periodic_250k", kind="host", n=250000, k=35, degree=3, nrhs=3),
        # the operator applied to a field, as a time step does
        dict(name="spmv_disk_1m", kind="spmv", n=1000003, k=35, degree=3),
        # a Poisson problem solved to convergence; every vector fits in L2
        dict(name="solve_disk_32k", kind="solve", n=32000, ragged=False, maxit=20000),
        # a fixed budget of iterations on a large ragged operator
        dict(name="solve_uneven_1m", kind="solve", n=1000003, ragged=True, maxit=48),
        # a lattice Boltzmann time step, FP64 populations
        dict(name="lbm_1m", kind="lbm", n=1048576, k=21, degree=2, populations="fp64"),
    ]


def _log_size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _stencil(rng):
    """Stencil size and degree: the usual pairs and the sizes around them."""
    degree = rng.choice([2, 3, 3, 4])
    k = {2: lambda: rng.randint(15, 26), 3: lambda: rng.randint(25, 37),
         4: lambda: rng.randint(45, 64)}[degree]()
    return k, degree


def draw(rng):
    kind = rng.choice(["operator", "operator", "operator", "knn", "uneven", "host", "spmv",
                       "solve", "lbm"])
    if kind == "operator":
        geometry = rng.choice(["square", "disk", "periodic", "bump"])
        precision = rng.choice(["fp64", "fp64", "fp32_ir"])
        k, degree = _stencil(rng)
        if precision == "fp32_ir" and degree == 4:
            k, degree = 35, 3  # the refined form does not pay at degree 4
        n = _log_size(rng, 2000, 150000 if degree == 4 else 700000)
        return dict(kind=kind, geometry=geometry, n=n, k=k, degree=degree, precision=precision,
                    nrhs=rng.choice([1, 2, 3, 3]))
    if kind == "knn":
        return dict(kind=kind, geometry=rng.choice(["square", "disk", "periodic", "bump"]),
                    n=_log_size(rng, 2000, 1000000), k=rng.randint(12, 64))
    if kind == "uneven":
        return dict(kind=kind, n=_log_size(rng, 5000, 500000))
    if kind == "host":
        k, degree = rng.choice([(21, 2), (28, 3), (35, 3)])
        return dict(kind=kind, n=_log_size(rng, 4000, 250000), k=k, degree=degree,
                    nrhs=rng.choice([1, 3]))
    if kind == "spmv":
        k, degree = _stencil(rng)
        return dict(kind=kind, n=_log_size(rng, 4000, 150000 if degree == 4 else 1000000), k=k,
                    degree=degree)
    if kind == "solve":
        ragged = rng.random() < 0.5
        if rng.random() < 0.5:
            return dict(kind=kind, n=_log_size(rng, 3000, 30000), ragged=False, maxit=20000)
        return dict(kind=kind, n=_log_size(rng, 30000, 1000000), ragged=ragged,
                    maxit=rng.randint(8, 48))
    return dict(kind="lbm", n=_log_size(rng, 10000, 1000000), k=rng.choice([15, 18, 21, 21, 24]),
                degree=2, populations=rng.choice(["fp64", "fp32"]))


# ---- inputs -----------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _context():
    """The program's one library context."""
    return R.Context(0)


def _side(n):
    return int(math.ceil(math.sqrt(n)))


def _nodes(geometry, n, seed):
    """(x, y, boundary flags, period) of n nodes, float64 on the host."""
    if geometry in ("square", "periodic"):
        m = _side(n)
        x, y, flag = NS.jittered_grid(m, 0.3, seed, periodic=geometry == "periodic")
        return x[:n], y[:n], flag[:n], (1.0, 1.0) if geometry == "periodic" else None
    if geometry == "disk":
        x, y, flag = NS.unit_disk(n, nb=_boundary(n), seed=seed)
        return x, y, flag, None
    x, y, flag = NS.gaussian_bump(n, seed)
    return x, y, flag, None


def _boundary(n):
    """Boundary nodes of an n-node disk: about the interior's spacing."""
    return max(16, int(3.5 * math.sqrt(n)))


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda")


def _ops(nrhs):
    return {1: R.OP_LAPLACE, 2: R.OP_DX | R.OP_DY, 3: R.DEFAULT_OPS}[nrhs]


def _op_names(nrhs):
    return {1: ["L"], 2: ["x", "y"], 3: ["L", "x", "y"]}[nrhs]


def _empty(n, dtype=torch.float64):
    return torch.empty(n, dtype=dtype, device="cuda")


def _uneven(n, seed):
    """The ragged disk batch: boundary stencils of 48-64 nodes at degree 4,
    interior ones of 21, 28 or 35 at degree 2 or 3."""
    x, y, flag = NS.unit_disk(n, nb=_boundary(n), seed=seed)
    nb = int(flag.sum())
    rng = np.random.default_rng(seed + 1000)
    kvec = np.concatenate([rng.permutation(np.resize(np.arange(48, 65, dtype=np.int32), nb)),
                           rng.permutation(np.resize(np.array([21, 28, 35], np.int32), n - nb))])
    degree = np.where(kvec < 28, 2, 3).astype(np.int8)
    degree[:nb] = 4
    xd, yd, kd = _dev(x), _dev(y), _dev(kvec)
    kmax = int(kvec.max())
    ja = _empty(n * kmax, torch.int32)
    _context().knn_stencils(xd, yd, kmax, ja)
    keep = torch.arange(kmax, device="cuda")[None, :] < kd[:, None]
    ia = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    ia[1:] = torch.cumsum(kd, 0)
    return dict(x=xd, y=yd, ia=ia, ja=ja.view(n, kmax)[keep].contiguous(), degree=_dev(degree),
                kvec=kd, bnd=_dev(np.flatnonzero(flag).astype(np.int32)))


def _u_exact(x, y):
    return torch.exp(x) * torch.sin(2.0 * y) + x * x


def _poisson_rhs(x, y, bnd):
    f = -3.0 * torch.exp(x) * torch.sin(2.0 * y) + 2.0
    f[bnd.long()] = _u_exact(x, y)[bnd.long()]
    return f


def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    ctx = _context()
    if kind in ("operator", "knn"):
        x, y, _, period = _nodes(case["geometry"], n, seed)
        s = dict(kind=kind, k=case["k"], period=period, x=_dev(x), y=_dev(y),
                 ja=_empty(n * case["k"], torch.int32))
        if kind == "operator":
            s["values"] = [_empty(n * case["k"]) for _ in range(case["nrhs"])]
            s["info"] = _empty(n, torch.int32)
            s["desc"] = R.make_desc(case["degree"], 0, _ops(case["nrhs"]),
                                    R.FP64 if case["precision"] == "fp64" else R.FP32_IR, True,
                                    period=period)
        return s
    if kind == "uneven":
        s = _uneven(n, seed)
        s.update(kind=kind, desc=R.make_desc(3, 0, R.DEFAULT_OPS, R.FP64, True),
                 values=[_empty(s["ja"].numel()) for _ in range(3)], info=_empty(n, torch.int32))
        return s
    if kind == "host":
        x, y, _, period = _nodes("periodic", n, seed)
        k = case["k"]
        return dict(kind=kind, k=k, x=torch.as_tensor(x.copy()).pin_memory(),
                    y=torch.as_tensor(y.copy()).pin_memory(),
                    ja=torch.empty(n * k, dtype=torch.int32, pin_memory=True),
                    values=[torch.empty(n * k, dtype=torch.float64, pin_memory=True)
                            for _ in range(case["nrhs"])],
                    desc=R.make_desc(case["degree"], 0, _ops(case["nrhs"]), R.FP64, True,
                                     period=period))
    if kind == "spmv":
        x, y, flag, _ = _nodes("disk", n, seed)
        s = dict(kind=kind, n=n, k=case["k"], x=_dev(x), y=_dev(y),
                 ja=_empty(n * case["k"], torch.int32), L=_empty(n * case["k"]), out=_empty(n),
                 bnd=_dev(np.flatnonzero(flag).astype(np.int32)))
        ctx.knn_stencils(s["x"], s["y"], s["k"], s["ja"])
        ctx.assemble(R.make_desc(case["degree"], 0, R.OP_LAPLACE), s["x"], s["y"], s["k"], s["ja"],
                     [s["L"]])
        s["u"] = _u_exact(s["x"], s["y"])
        return s
    if kind == "solve":
        if case["ragged"]:
            s = _uneven(n, seed)
            s["L"] = _empty(s["ja"].numel())
            ctx.assemble_csr(R.make_desc(3, 0, R.OP_LAPLACE), s["x"], s["y"], s["ia"], s["ja"],
                             [s["L"]], degree=s["degree"])
            s["k"] = None
        else:
            x, y, flag, _ = _nodes("disk", n, seed)
            s = dict(k=21, ia=None, x=_dev(x), y=_dev(y), ja=_empty(n * 21, torch.int32),
                     L=_empty(n * 21), bnd=_dev(np.flatnonzero(flag).astype(np.int32)))
            ctx.knn_stencils(s["x"], s["y"], 21, s["ja"])
            ctx.assemble(R.make_desc(2, 0, R.OP_LAPLACE), s["x"], s["y"], 21, s["ja"], [s["L"]])
        s.update(kind=kind, maxit=case["maxit"], u=_empty(n),
                 f=_poisson_rhs(s["x"], s["y"], s["bnd"]))
        return s
    # lbm: the operators of the 8 departure points half a grid spacing away
    x, y, _, period = _nodes("periodic", n, seed)
    k = case["k"]
    xd, yd = _dev(x), _dev(y)
    s = dict(kind=kind, k=k, ja=_empty(n * k, torch.int32), W=_empty(8 * n * k))
    ctx.knn_stencils(xd, yd, k, s["ja"], period=period)
    xc, yc = (_dev(a) for a in R.lbm_departure_points(0.5 / _side(n)))
    ctx.assemble(R.make_desc(case["degree"], 0, R.OP_INTERP, R.FP64, True, period=period, xc=xc,
                             yc=yc, nc=8), xd, yd, k, s["ja"], list(s["W"].split(n * k)))
    dt = torch.float64 if case["populations"] == "fp64" else torch.float32
    rho, ux, uy = _flow(xd, yd, dt)
    s.update(pdf=_empty(9 * n, dt), out=_empty(9 * n, dt), rho=rho, ux=ux, uy=uy)
    R.lbm_feq(rho, ux, uy, s["pdf"])
    torch.cuda.synchronize()  # xc and yc are read by the assembly above
    return s


def _flow(x, y, dt):
    """Density and velocity of a smooth periodic flow."""
    t = 2.0 * math.pi
    return ((1.0 + 0.02 * torch.sin(t * x)).to(dt), (0.03 * torch.cos(t * y)).to(dt),
            (0.01 * torch.sin(t * (x + y))).to(dt))


# ---- one pass ---------------------------------------------------------------

def run(s):
    kind, ctx = s["kind"], _context()
    if kind == "operator":
        ctx.knn_stencils(s["x"], s["y"], s["k"], s["ja"], period=s["period"])
        ctx.assemble(s["desc"], s["x"], s["y"], s["k"], s["ja"], s["values"], s["info"])
        return {"ja": s["ja"], "values": s["values"], "info": s["info"]}
    if kind == "knn":
        ctx.knn_stencils(s["x"], s["y"], s["k"], s["ja"], period=s["period"])
        return {"ja": s["ja"]}
    if kind == "uneven":
        ctx.assemble_csr(s["desc"], s["x"], s["y"], s["ia"], s["ja"], s["values"],
                         degree=s["degree"], info=s["info"])
        return {"values": s["values"], "info": s["info"]}
    if kind == "host":
        ctx.assemble_host(s["desc"], s["x"], s["y"], s["k"], s["values"], ja_out_h=s["ja"])
        return {"ja": s["ja"], "values": s["values"]}
    if kind == "spmv":
        R.spmv(s["n"], s["k"], s["ja"], s["L"], s["u"], s["out"], s["bnd"])
        return {"out": s["out"]}
    if kind == "solve":
        s["u"].zero_()
        status, iters, _ = ctx.solve_bicgstab(s["L"], s["ja"], s["f"], s["u"], k=s["k"],
                                              ia=s["ia"], bnd=s["bnd"], tol=TOL,
                                              maxit=s["maxit"])
        return {"u": s["u"], "status": status, "iters": iters}
    R.lbm_stream_collide(s["k"], s["ja"], s["W"], OMEGA, s["pdf"], s["out"], s["rho"], s["ux"],
                         s["uy"])
    return {"pdf": s["out"], "rho": s["rho"], "ux": s["ux"], "uy": s["uy"]}


# ---- compulsory work --------------------------------------------------------

def _npoly(degree):
    return (degree + 1) * (degree + 2) // 2


def _lu_flops(k, degree, nrhs):
    m = k + _npoly(degree)
    return 2.0 / 3.0 * m ** 3 + 2.0 * m * m * nrhs


def work(case):
    kind, n = case["kind"], case["n"]
    k = case.get("k")
    if kind in ("operator", "host"):
        b = n * (16 + 4 * k + 8 * k * case["nrhs"] + (4 if kind == "operator" else 0))
        return {"bytes": b, "flops": n * (_lu_flops(k, case["degree"], case["nrhs"]) + 5 * k)}
    if kind == "knn":
        return {"bytes": n * (16 + 4 * k), "flops": n * 5 * k}
    nb = _boundary(n)
    if kind == "uneven" or case.get("ragged"):
        nnz = 28 * (n - nb) + 56 * nb  # means of the sizes in _uneven
    else:
        nnz = n * (k or 21)
    if kind == "uneven":
        f = (n - nb) / 3.0 * (_lu_flops(21, 2, 3) + _lu_flops(28, 3, 3) + _lu_flops(35, 3, 3))
        return {"bytes": 16 * n + 5 * n + nnz * (4 + 24) + 4 * n,
                "flops": f + nb * _lu_flops(56, 4, 3)}
    if kind == "spmv":
        return {"bytes": 12 * nnz + 16 * n + 20 * nb, "flops": 2 * nnz}
    if kind == "solve":
        # two operator passes and the vector updates of every iteration; a solve
        # to convergence takes about 9 sqrt(n) iterations on this problem
        iters = case["maxit"] if case["maxit"] < 1000 else 9 * math.sqrt(n)
        return {"bytes": iters * (24 * nnz + 162 * n), "flops": iters * (4 * nnz + 24 * n)}
    es = 8 if case["populations"] == "fp64" else 4
    return {"bytes": n * (8 * 8 * k + 4 * k + 21 * es), "flops": n * (16 * k + 90)}


# ---- the same results in plain 64-bit torch ---------------------------------

def _wrap(d, L):
    return d - L * torch.round(d / L) if L else d


def _neighbours(x, y, k, period):
    """k nearest nodes of every node by (distance, index): candidates from the
    cells around each node, more rings until the k-th lies inside them."""
    n = x.numel()
    L = period[0] if period else 0.0
    x0, y0 = (x.new_tensor(0.0),) * 2 if period else (x.min(), y.min())
    c = max(1, int(math.sqrt(n / 4)))
    hx = L / c if period else float(x.max() - x0) / c * (1 + 1e-12)
    hy = L / c if period else float(y.max() - y0) / c * (1 + 1e-12)
    cx = ((x - x0) / hx).long().clamp(0, c - 1)
    cy = ((y - y0) / hy).long().clamp(0, c - 1)
    cell = cy * c + cx
    order = torch.argsort(cell, stable=True)
    count = torch.bincount(cell, minlength=c * c)
    first = torch.cumsum(count, 0) - count
    cap = int(count.max())
    table = torch.full((c * c, cap), -1, dtype=torch.int64, device=x.device)
    table[cell[order], torch.arange(n, device=x.device) - first[cell[order]]] = order
    out = torch.empty((n, k), dtype=torch.int64, device=x.device)
    todo = torch.arange(n, device=x.device)
    ring = 2
    while todo.numel():
        ring = min(ring, c)
        whole = 2 * ring + 1 >= c
        off = torch.arange(-ring, ring + 1, device=x.device)
        if whole and period:
            off = torch.arange(0, c, device=x.device)
        oy, ox = (g.reshape(-1) for g in torch.meshgrid(off, off, indexing="ij"))
        left = []
        step = max(1, int(4e7 // (oy.numel() * cap)))
        for q in todo.split(step):
            gy, gx = cy[q][:, None] + oy, cx[q][:, None] + ox
            if period:
                gy, gx = gy % c, gx % c
                ok = torch.ones_like(gy, dtype=torch.bool)
            else:
                ok = (gy >= 0) & (gy < c) & (gx >= 0) & (gx < c)
            cand = table[(gy * c + gx).clamp(0, c * c - 1)]
            cand = torch.where(ok[..., None], cand, -1).reshape(q.numel(), -1)
            cand = cand.sort(dim=1).values
            dx = _wrap(x[q][:, None] - x[cand.clamp_min(0)], L)
            dy = _wrap(y[q][:, None] - y[cand.clamp_min(0)], L)
            d2 = torch.where(cand < 0, math.inf, dx * dx + dy * dy)
            d2, at = d2.sort(dim=1, stable=True)
            if d2.shape[1] < k:
                left.append(q)
                continue
            far = d2[:, k - 1].sqrt()
            good = (far < ring * min(hx, hy) * (1 - 1e-9)) | (ring >= c)
            if whole and period:
                good = torch.ones_like(good)
            out[q[good]] = cand.gather(1, at[:, :k])[good]
            left.append(q[~good])
        todo = torch.cat(left) if left else todo[:0]
        ring += max(1, ring // 2)
    return out


def _weights(x, y, ja, degree, rows, period):
    """Weights of the right-hand sides `rows` ("L", "x", "y" or a point) of the
    fixed-width stencils ja: the PHS + polynomial system of every stencil."""
    n, k = ja.shape
    npol, q = _npoly(degree), 2 * degree - 1
    L = period[0] if period else 0.0
    out = [torch.empty((n, k), dtype=torch.float64, device=x.device) for _ in rows]
    m = k + npol
    for s in torch.arange(n, device=x.device).split(max(1, int(1.5e8 // (m * m)))):
        X = _wrap(x[ja[s]] - x[ja[s][:, :1]], L)
        Y = _wrap(y[ja[s]] - y[ja[s][:, :1]], L)
        h = torch.sqrt(X * X + Y * Y).amax(1, keepdim=True)
        X, Y = X / h, Y / h
        r2 = (X[:, :, None] - X[:, None, :]) ** 2 + (Y[:, :, None] - Y[:, None, :]) ** 2
        A = torch.zeros((s.numel(), m, m), dtype=torch.float64, device=x.device)
        A[:, :k, :k] = r2 ** (q // 2) * torch.sqrt(r2)
        mono = [(d - j, j) for d in range(degree + 1) for j in range(d + 1)]
        for i, (a, b) in enumerate(mono):
            A[:, :k, k + i] = A[:, k + i, :k] = X ** a * Y ** b
        B = torch.zeros((s.numel(), m, len(rows)), dtype=torch.float64, device=x.device)
        R2 = X * X + Y * Y
        rq2 = R2 ** ((q - 2) // 2) * torch.sqrt(R2)  # r^(q - 2)
        for c, op in enumerate(rows):
            if op == "L":
                B[:, :k, c] = q * q * rq2
                B[:, k + mono.index((2, 0)), c] = B[:, k + mono.index((0, 2)), c] = 2.0
            elif op == "x":
                B[:, :k, c] = -q * rq2 * X
                B[:, k + mono.index((1, 0)), c] = 1.0
            elif op == "y":
                B[:, :k, c] = -q * rq2 * Y
                B[:, k + mono.index((0, 1)), c] = 1.0
            else:
                px, py = op[0] / h, op[1] / h
                e2 = (X - px) ** 2 + (Y - py) ** 2
                B[:, :k, c] = e2 ** (q // 2) * torch.sqrt(e2)
                for i, (a, b) in enumerate(mono):
                    B[:, k + i, c] = (px ** a * py ** b)[:, 0]
        W = torch.linalg.solve(A, B)[:, :k]
        for c, op in enumerate(rows):
            order = {"L": 2, "x": 1, "y": 1}.get(op if isinstance(op, str) else "", 0)
            out[c][s] = W[:, :, c] / h ** order
    return out


def _uneven_weights(s, rows):
    """The ragged batch's weights in CSR order, one stencil size at a time."""
    kvec, ia, ja = s["kvec"], s["ia"].long(), s["ja"].long()
    out = [torch.empty(ja.numel(), dtype=torch.float64, device="cuda") for _ in rows]
    for k in kvec.unique().tolist():
        at = torch.nonzero(kvec == k)[:, 0]
        pos = ia[at][:, None] + torch.arange(k, device="cuda")
        degree = 2 if k < 28 else 3 if k < 48 else 4
        for o, w in zip(out, _weights(s["x"], s["y"], ja[pos], degree, rows, None)):
            o[pos] = w
    return out


def _ragged_stencils(s):
    """The CSR stencils of the ragged batch from the plain search."""
    kmax = int(s["kvec"].max())
    near = _neighbours(s["x"], s["y"], kmax, None)
    keep = torch.arange(kmax, device="cuda")[None, :] < s["kvec"][:, None]
    return near[keep]


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    if kind == "knn":
        return None  # whole numbers
    if kind == "solve" and (case["ragged"] or case["maxit"] < 1000):
        return None  # not run to convergence
    if kind == "uneven":
        s = _uneven(n, seed)
        s["ja"] = _ragged_stencils(s)
        return {"values": _uneven_weights(s, ["L", "x", "y"]), "info": None}
    geometry = {"host": "periodic", "spmv": "disk", "solve": "disk", "lbm": "periodic"}
    x, y, flag, period = _nodes(case.get("geometry") or geometry[kind], n, seed)
    x, y = _dev(x), _dev(y)
    k, degree = case.get("k", 21), case.get("degree", 2)
    near = _neighbours(x, y, k, period)
    if kind in ("operator", "host"):
        values = [w.reshape(-1) for w in
                  _weights(x, y, near, degree, _op_names(case["nrhs"]), period)]
        return {"ja": None, "values": values} | ({"info": None} if kind == "operator" else {})
    bnd = torch.as_tensor(np.flatnonzero(flag), device="cuda")
    if kind == "spmv":
        u = _u_exact(x, y)
        out = (_weights(x, y, near, degree, ["L"], None)[0] * u[near]).sum(1)
        out[bnd] = u[bnd]
        return {"out": out}
    if kind == "solve":
        A = torch.zeros((n, n), dtype=torch.float64, device="cuda")
        A.scatter_(1, near, _weights(x, y, near, degree, ["L"], None)[0])
        A[bnd] = 0.0
        A[bnd, bnd] = 1.0
        u = torch.linalg.solve(A, _poisson_rhs(x, y, bnd))
        return {"u": u, "status": None, "iters": None}
    xc, yc = R.lbm_departure_points(0.5 / _side(n))
    W = _weights(x, y, near, degree, list(zip(xc.tolist(), yc.tolist())), period)
    dt = torch.float64 if case["populations"] == "fp64" else torch.float32
    rho, ux, uy = (v.double() for v in _flow(x, y, dt))
    cv = np.array(R.LBM_C, np.float64)
    w = [4 / 9] + [1 / 9] * 4 + [1 / 36] * 4

    def equilibrium(rho, ux, uy):
        cu = [cx * ux + cy * uy for cx, cy in cv]
        return [w[a] * rho * (1 + 3 * cu[a] + 4.5 * cu[a] ** 2 - 1.5 * (ux * ux + uy * uy))
                for a in range(9)]
    f = equilibrium(rho, ux, uy)
    f = [f[0]] + [(W[a - 1] * f[a][near]).sum(1) for a in range(1, 9)]
    rho = sum(f)
    ux = sum(c[0] * g for c, g in zip(cv, f)) / rho
    uy = sum(c[1] * g for c, g in zip(cv, f)) / rho
    out = [(1 - OMEGA) * g + OMEGA * e for g, e in zip(f, equilibrium(rho, ux, uy))]
    return {"pdf": torch.cat(out), "rho": rho, "ux": ux, "uy": uy}
