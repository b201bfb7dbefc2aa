"""The work that programs have this library do, as cases to be timed.

Every case goes through the public Python entry points (bcm-problems_b200/bsg.py)
and stands for one thing a user's program does: a product inside its own loop,
the preconditioner, a factorisation in a time step, a whole driver call on host
arrays, a batch of problems, a homogenisation cell, the learned stage and its
training.  Sizes are those of the benchmark's configurations (32^3, 48^3, 64^3,
128^3 grids, batches of 2-D problems of side 32 to 256) and of the tests (12^3),
and odd ones between them.

The systems are made here, on the GPU, from the seed: the cell-centred 7-point
(5-point in 2-D) finite-volume heat operator with lognormal conductivity,
optionally with upwind convection, and trilinear (Q1) linear elasticity in 3x3
blocks, periodic with stiff inclusions or clamped at the bottom.  Storage is the
library's: 0-based CSR, each row's diagonal first, then ascending columns;
blocks column-major.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "bcm-problems_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

TAU = 1e-3  # dropping threshold of every factor (tau1 = tau2), as in the benchmark


def listed():
    return [
        # The smallest system of the tests: a caller's own loop around the
        # product, where the call and the launch are all there is.
        dict(name="product 12^3", kind="product", nx=12, ny=12, nz=12, block=False, nrhs=1),
        # The product of the benchmark's largest system (2.1M rows).
        dict(name="product 128^3", kind="product", nx=128, ny=128, nz=128, block=False, nrhs=1),
        # Elasticity, all six load cases of a homogenisation cell in one call.
        dict(name="block product 6 vectors", kind="product", nx=45, ny=37, nz=41, block=True, nrhs=6),
        # The default preconditioner: FP64 factor, exact forward and backward
        # solve (the reference's SolveL / SolveU).
        dict(name="exact solves", kind="precond", nx=47, ny=40, nz=33, sigma=1.0, fp32=False, sweeps=0),
        # The fast preconditioner of the benchmark's system: FP32 factor values,
        # six Jacobi sweeps each way.
        dict(name="sweeps fp32 128^3", kind="precond", nx=128, ny=128, nz=128, sigma=1.5, fp32=True, sweeps=6),
        # A time step with new coefficients: the matrix's IC2 factor, turned
        # to FP32, and its first application.
        dict(name="factor 80x72x65", kind="factor", nx=80, ny=72, nz=65, sigma=1.5, ilu=False, fp32=True),
        # The symmetric host driver at the benchmark's first configuration:
        # 32^3, unit conductivity, FP64, exact solves, PCG to 1e-10.
        dict(name="driver 32^3", kind="driver", nx=32, ny=32, nz=32, sigma=0.0, wind=0.0, sweeps=0, eps=1e-10),
        # The nonsymmetric host driver on convection-diffusion: ILU2, two-sided Lanczos.
        dict(name="driver convection", kind="driver", nx=28, ny=21, nz=24, sigma=0.5, wind=0.5, sweeps=0, eps=1e-10),
        # The benchmark's headline solve: learned FGMRES(30) on a factor in hand.
        dict(name="learned fgmres 128^3", kind="krylov", nx=128, ny=128, nz=128, sigma=1.5, method="learned", eps=1e-8),
        # A batch of the learned stage's training at its training size.
        dict(name="unet training 64^3", kind="train", nx=64, ny=64, nz=64, samples=2),
        # Many small independent 2-D problems of uneven sizes, from host arrays
        # to solutions in one go.
        dict(name="batch of 2-D problems", kind="batch", count=96, smin=32, smax=160, sigma=1.0),
        # A homogenisation cell: block IC2 of the periodic elastic cell and PCG
        # on its six load cases.
        dict(name="elastic cell 20^3", kind="elastic", n=20, periodic=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["product", "product", "precond", "precond", "factor", "driver", "krylov", "unet", "train",
                       "batch", "elastic"])

    def grid(lo, hi):
        s = _log(rng, lo, hi)
        return dict(nx=s, ny=max(lo, min(hi, s + rng.randint(-s // 4, s // 4))),
                    nz=max(lo, min(hi, s + rng.randint(-s // 4, s // 4))))

    if kind == "product":
        if rng.random() < 0.4:
            return dict(kind=kind, block=True, nrhs=rng.randint(1, 8), **grid(6, 46))
        return dict(kind=kind, block=False, nrhs=rng.choice([1, 1, 2, 5, 8]), **grid(10, 112))
    if kind == "precond":
        if rng.random() < 0.5:
            return dict(kind=kind, sigma=round(rng.uniform(0, 1.5), 2), fp32=rng.random() < 0.3, sweeps=0, **grid(10, 44))
        return dict(kind=kind, sigma=round(rng.uniform(0, 1.5), 2), fp32=rng.random() < 0.7, sweeps=rng.randint(2, 8),
                    **grid(12, 110))
    if kind == "factor":
        return dict(kind=kind, sigma=round(rng.uniform(0, 1.5), 2), ilu=rng.random() < 0.4, fp32=rng.random() < 0.6,
                    **grid(12, 84))
    if kind == "driver":
        wind = rng.choice([0.0, 0.0, 0.3, 0.6])
        return dict(kind=kind, sigma=round(rng.uniform(0, 1.0), 2), wind=wind, sweeps=0 if wind else rng.choice([0, 6]),
                    eps=1e-10, **grid(8, 24 if wind else 36))
    if kind == "krylov":
        return dict(kind=kind, sigma=round(rng.uniform(0.5, 1.5), 2), eps=1e-8,
                    method=rng.choice(["pcg", "pcg64", "fgmres"]), **grid(20, 100))
    if kind == "unet":
        return dict(kind=kind, nx=rng.choice([16, 24, 32, 64, 96, 128]), ny=8 * rng.randint(2, 14),
                    nz=8 * rng.randint(2, 14))
    if kind == "train":
        s = 8 * rng.randint(2, 8)
        return dict(kind=kind, nx=s, ny=s, nz=8 * rng.randint(2, 8), samples=rng.randint(1, 4))
    if kind == "batch":
        smin = _log(rng, 24, 64)
        return dict(kind=kind, count=_log(rng, 4, 96), smin=smin, smax=min(160, _log(rng, smin, 160) + 8),
                    sigma=round(rng.uniform(0.3, 1.2), 2))
    return dict(kind="elastic", n=_log(rng, 7, 20), periodic=rng.random() < 0.5)


# ---- inputs ----------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) + 1)
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _csr(cols, vals, keep):
    """CSR of the kept slots of [rows, slots] columns and values, in slot order."""
    ia = torch.zeros(keep.shape[0] + 1, dtype=torch.int64, device=keep.device)
    torch.cumsum(keep.sum(1), 0, out=ia[1:])
    return ia.to(torch.int32), cols[keep].to(torch.int32), vals[keep]


def _heat(g, nx, ny, nz, sigma, wind=0.0):
    """[rows, 7] columns and values (diagonal, -z, -y, -x, +x, +y, +z) of the
    heat operator and which of them are inside the grid; wind: upwind
    convection along (1, 0.5, 0.25) times the mean conductance."""
    k = torch.exp(sigma * _randn(g, nz, ny, nx)) if sigma > 0 else torch.ones(nz, ny, nx, dtype=torch.float64, device="cuda")
    n = nx * ny * nz
    row = torch.arange(n, device="cuda").view(nz, ny, nx)
    dirs = [(0, -1, nx * ny), (1, -1, nx), (2, -1, 1), (2, 1, 1), (1, 1, nx), (0, 1, nx * ny)]
    if nz == 1:
        dirs = dirs[1:5]
    vel = {2: wind, 1: 0.5 * wind, 0: 0.25 * wind}
    diag = torch.zeros_like(k)
    cols, vals, keep = [row.reshape(-1)], [None], [torch.ones(n, dtype=torch.bool, device="cuda")]
    for d, sgn, stride in dirs:
        inside = torch.ones(nz, ny, nx, dtype=torch.bool, device="cuda")
        inside.select(d, 0 if sgn < 0 else k.shape[d] - 1).fill_(False)
        other = torch.roll(k, -sgn, d)
        c = torch.where(inside, 2 * k * other / (k + other), k)
        up = vel[d] if sgn < 0 else 0.0  # the wind blows towards larger coordinates
        diag += c + up
        cols.append((row + sgn * stride).reshape(-1))
        vals.append((-c - up).reshape(-1))
        keep.append(inside.reshape(-1))
    vals[0] = diag.reshape(-1)
    return torch.stack(cols, 1), torch.stack(vals, 1), torch.stack(keep, 1)


def _upper(cols, vals, keep):
    return _csr(cols, vals, keep & (cols >= cols[:, :1]))


def _heat2d_batch(g, count, smin, smax, sigma):
    """`count` square 2-D problems on the diagonal, sides from smin to smax
    evenly over the logarithm and in no order, and their row offsets."""
    u = np.random.RandomState(count).permutation(count) / max(1, count - 1)
    sides = np.floor(np.exp(math.log(smin) + u * (math.log(smax) - math.log(smin))) + 0.5).astype(int)
    off = np.concatenate([[0], np.cumsum(sides * sides)]).astype(np.int32)
    parts = []
    for s, o in zip(sides, off):
        cols, vals, keep = _heat(g, int(s), int(s), 1, sigma)
        parts.append((cols + int(o), vals, keep))
    return [torch.cat(t) for t in zip(*parts)], off


def _hexahedron(nu, h):
    """Stiffness [24, 24] and unit-strain loads [6, 24] of the trilinear cube
    element, E = 1, 2x2x2 Gauss points, Voigt order xx yy zz yz xz xy."""
    lam, mu = nu / ((1 + nu) * (1 - 2 * nu)), 1 / (2 * (1 + nu))
    C = np.zeros((6, 6))
    C[:3, :3] = lam
    C[range(3), range(3)] += 2 * mu
    C[range(3, 6), range(3, 6)] = mu
    corner = np.array([[2 * (a & 1) - 1, (a & 2) - 1, (a & 4) // 2 - 1] for a in range(8)], float)
    K, F = np.zeros((24, 24)), np.zeros((6, 24))
    for q in corner / math.sqrt(3.0):
        f = 1 + q * corner
        dN = corner * np.stack([f[:, 1] * f[:, 2], f[:, 0] * f[:, 2], f[:, 0] * f[:, 1]], 1) / 8 * (2 / h)
        B = np.zeros((6, 8, 3))
        B[0, :, 0], B[1, :, 1], B[2, :, 2] = dN[:, 0], dN[:, 1], dN[:, 2]
        B[3, :, 1], B[3, :, 2] = dN[:, 2], dN[:, 1]
        B[4, :, 0], B[4, :, 2] = dN[:, 2], dN[:, 0]
        B[5, :, 0], B[5, :, 1] = dN[:, 1], dN[:, 0]
        B = B.reshape(6, 24)
        K += B.T @ C @ B * (h / 2) ** 3
        F -= C @ B * (h / 2) ** 3
    return K, F


def _elastic(g, nx, ny, nz, periodic):
    """Q1 elasticity on nx x ny x nz nodes: [rows, 27] block columns, [rows,
    27, 9] column-major blocks, which exist, and right-hand sides [nrhs, 3
    rows].  periodic: stiff spheres (contrast 100) in about 30% of the cell,
    node 0 pinned, six unit strains; else lognormal stiffness, the z = 0 nodes
    clamped, a unit body force."""
    h = 1.0 / max(nx, ny, nz)
    K, F = _hexahedron(0.3, h)
    K = torch.as_tensor(K, device="cuda").view(8, 3, 8, 3)
    F = torch.as_tensor(F, device="cuda").view(6, 8, 3)
    n = nx * ny * nz
    node = torch.arange(n, device="cuda").view(nz, ny, nx)
    ax = [torch.arange(m, device="cuda", dtype=torch.float64) + 0.5 for m in (nz, ny, nx)]
    if periodic:
        E = torch.ones(nz, ny, nx, dtype=torch.float64, device="cuda")
        size = torch.tensor([nz, ny, nx], device="cuda", dtype=torch.float64)
        for c, r in zip(_rand(g, 8, 3) * size, (0.16 + 0.10 * _rand(g, 8)) * min(nx, ny, nz)):
            d2 = 0
            for i, shape in enumerate(((-1, 1, 1), (1, -1, 1), (1, 1, -1))):
                d = (ax[i] - c[i]).abs()
                d2 = d2 + torch.minimum(d, size[i] - d).square().view(shape)
            E = torch.where(d2 <= r * r, torch.full_like(E, 100.0), E)
        fixed = node == 0
    else:
        E = torch.exp(_randn(g, nz, ny, nx))
        E[-1], E[:, -1], E[:, :, -1] = 0, 0, 0  # the cells beyond the last nodes do not exist
        fixed = (node // (nx * ny)) == 0
    W = torch.zeros(27, n, 3, 3, dtype=torch.float64, device="cuda")
    load = torch.zeros(6 if periodic else 1, n, 3, dtype=torch.float64, device="cuda")
    for a in range(8):
        ca = ((a >> 2) & 1, (a >> 1) & 1, a & 1)
        e = torch.roll(E, ca, (0, 1, 2)).reshape(-1)  # stiffness of the cell whose corner a this node is
        for b in range(8):
            cb = ((b >> 2) & 1, (b >> 1) & 1, b & 1)
            o = [cb[i] - ca[i] + 1 for i in range(3)]
            W[9 * o[0] + 3 * o[1] + o[2]] += e[:, None, None] * K[a, :, b, :]
        if periodic:
            load += e[None, :, None] * F[:, a, None, :]
        else:
            load[0, :, 2] -= (e > 0) * h ** 3 / 8
    cols, keep = [], []
    for o in range(27):
        d = (o // 9 - 1, o // 3 % 3 - 1, o % 3 - 1)
        cols.append(torch.roll(node, [-v for v in d], (0, 1, 2)).reshape(-1))
        inside = torch.ones(nz, ny, nx, dtype=torch.bool, device="cuda")
        if not periodic:
            for i in range(3):
                if d[i]:
                    inside.select(i, 0 if d[i] < 0 else inside.shape[i] - 1).fill_(False)
        keep.append(inside.reshape(-1))
    cols, keep, W = torch.stack(cols, 1), torch.stack(keep, 1), W.permute(1, 0, 2, 3).contiguous()
    fixed = fixed.reshape(-1)
    keep &= ~(fixed[:, None] | fixed[cols])
    keep[:, 13] = True
    W[fixed, 13] = torch.eye(3, dtype=torch.float64, device="cuda")
    load[:, fixed] = 0
    key = cols.clone()
    key[:, 13] = -1  # the diagonal block first, then ascending columns
    order = key.argsort(1)
    cols, keep = cols.gather(1, order), keep.gather(1, order)
    W = W.gather(1, order[:, :, None, None].expand_as(W))
    return cols, W.transpose(2, 3).reshape(n, 27, 9), keep, load.view(load.shape[0], 3 * n)


def _host(*ts):
    return [t.cpu().numpy() for t in ts]


def _weights():
    return np.load(os.path.join(PKG, "weights", "unet_heat64.npz"))["w"].astype(np.float32)


def _param(bsg, **kw):
    base = dict(ordtype=0, fcttyp=2, tau1=TAU, tau2=TAU, theta=0.1, memory=20.0, ittype=0, sttype=1, niter=3000,
                true_residual=1)
    base.update(kw)
    return bsg.default_param(**base)


def _inputs(case, seed):
    """The system and vectors of a case: what prepare() hands to the library
    and exact() computes with."""
    g = _generator(seed)
    kind, d = case["kind"], {}
    if kind == "batch":
        (cols, vals, keep), d["seg"] = _heat2d_batch(g, case["count"], case["smin"], case["smax"], case["sigma"])
    elif kind == "elastic" or case.get("block"):
        dims = (case["n"],) * 3 if kind == "elastic" else (case["nx"], case["ny"], case["nz"])
        cols, vals, keep, d["load"] = _elastic(g, *dims, kind == "elastic" and case["periodic"])
    else:
        cols, vals, keep = _heat(g, case["nx"], case["ny"], case["nz"], case.get("sigma", 1.0), case.get("wind", 0.0))
    n = cols.shape[0]
    d.update(n=n, cols=cols, vals=vals, keep=keep)
    if kind == "product":
        d["x"] = _randn(g, case["nrhs"], n * (3 if case["block"] else 1))
    elif kind in ("unet", "train"):
        d["r"] = _randn(g, case.get("samples", 1), n)
        if kind == "train":
            # errors are smoother than the residuals they leave
            t = d["r"].view(-1, case["nz"], case["ny"], case["nx"])
            for i in (1, 2, 3):
                t = t + 0.9 * torch.roll(t, 1, i)
            d["t"] = (t + 0.3 * _randn(g, *t.shape)).reshape(-1, n).contiguous()
    elif kind != "elastic":
        d["b"] = 2 * _rand(g, n) - 1
    return d


def prepare(case, seed):
    import bsg
    d = _inputs(case, seed)
    kind = case["kind"]
    ctx = bsg.Context(0)
    s = dict(kind=kind, case=case, bsg=bsg, ctx=ctx)

    def matrix(symm):
        ia, ja, a = _host(*(_upper if symm else _csr)(d["cols"], d["vals"], d["keep"]))
        return bsg.Matrix(ctx, d["n"], ia, ja, a.reshape(-1), 3 if case.get("block") else 1, symm)

    if kind == "product":
        s["m"], s["x"], s["y"] = matrix(False), d["x"], torch.empty_like(d["x"])
    elif kind == "precond":
        s["m"] = matrix(True)
        s["p"] = _param(bsg, precision=int(case["fp32"]))
        s["f"] = bsg.Factor(ctx, s["m"], "ich2", s["p"])
        s["x"], s["t"], s["y"] = d["b"], torch.empty_like(d["b"]), torch.empty_like(d["b"])
    elif kind == "factor":
        s["m"] = matrix(not case["ilu"])
        s["x"], s["t"], s["y"] = d["b"], torch.empty_like(d["b"]), torch.empty_like(d["b"])
    elif kind == "driver":
        s["symm"] = case["wind"] == 0
        s["n"] = d["n"]
        s["ia"], s["ja"], s["a"] = _host(*(_upper if s["symm"] else _csr)(d["cols"], d["vals"], d["keep"]))
        s["b"] = d["b"].cpu().numpy()
    elif kind == "krylov":
        s["m"], s["b"], s["x"] = matrix(True), d["b"], torch.empty_like(d["b"])
        full64 = case["method"] == "pcg64"
        s["p"] = _param(bsg, precision=0 if full64 else 1, trisolve=1, nsweeps=6, eps=case["eps"], restart=30,
                        krylov=0 if case["method"] in ("pcg", "pcg64") else 2)
        s["f"] = bsg.Factor(ctx, s["m"], "ich2", s["p"])
        if case["method"] == "learned":
            s["net"] = bsg.UNet(ctx, case["nx"], case["ny"], case["nz"])
            s["net"].set_weights(_weights())
            s["p"].learned = s["net"].h.value
    elif kind in ("unet", "train"):
        s["net"] = bsg.UNet(ctx, case["nx"], case["ny"], case["nz"], train=kind == "train")
        s["net"].set_weights(_weights())
        s["diag"] = d["vals"][:, 0].contiguous()
        s["r"], s["y"], s["t"] = d["r"], torch.empty_like(d["r"][0]), d.get("t")
        s["net"].set_diag(s["diag"])
    elif kind == "batch":
        s["n"], s["seg"] = d["n"], d["seg"]
        s["ia"], s["ja"], s["a"] = _host(*_upper(d["cols"], d["vals"], d["keep"]))
        s["b"], s["x"] = d["b"][None], torch.empty_like(d["b"][None])
    elif kind == "elastic":
        s["n"], s["b"] = d["n"], d["load"].contiguous()
        s["ia"], s["ja"], s["a"] = _host(*(_upper if case["periodic"] else _csr)(d["cols"], d["vals"], d["keep"]))
        s["x"] = torch.empty_like(s["b"])
    return s


def run(s):
    bsg, ctx, case, kind = s["bsg"], s["ctx"], s["case"], s["kind"]
    if kind == "product":
        if case["nrhs"] == 1:
            s["m"].mvm(s["x"], s["y"])
        else:
            s["m"].mvm_multi(s["x"], s["y"])
        return s["y"]
    if kind == "precond":
        mode = dict(mode=1, nsweeps=case["sweeps"]) if case["sweeps"] else dict(mode=0)
        s["f"].solve_l(s["x"], s["t"], **mode)
        s["f"].solve_u(s["t"], s["y"], **mode)
        return s["y"]
    if kind == "factor":
        p = _param(bsg, precision=int(case["fp32"]))
        f = bsg.Factor(ctx, s["m"], "ilu2" if case["ilu"] else "ich2", p)
        f.solve_l(s["x"], s["t"], mode=1, nsweeps=6)
        f.solve_u(s["t"], s["y"], mode=1, nsweeps=6)
        return dict(y=s["y"], entries=f.info()["nnz"], density=p.density)
    if kind == "driver":
        solve = bsg.solve_symm if s["symm"] else bsg.solver
        p = _param(bsg, eps=case["eps"], trisolve=1 if case["sweeps"] else 0, nsweeps=max(1, case["sweeps"]))
        return solve(ctx, s["n"], s["ia"], s["ja"], s["a"], s["b"], p)
    if kind == "krylov":
        s["x"].zero_()
        (bsg.pcg if s["p"].krylov == 0 else bsg.gmres)(ctx, s["m"], s["f"], s["b"], s["x"], s["p"])
        return s["x"]
    if kind == "unet":
        s["net"].forward(s["r"][0], s["y"])
        return s["y"]
    if kind == "train":
        s["net"].zero_grads()
        for r, t in zip(s["r"], s["t"]):
            s["net"].set_diag(s["diag"])
            s["net"].train_sample(r, t)
        return s["net"].grads()
    if kind == "batch":
        p = _param(bsg, eps=1e-8, precision=1, trisolve=1, nsweeps=6)
        m = bsg.Matrix(ctx, s["n"], s["ia"], s["ja"], s["a"], 1, True)
        f = bsg.Factor(ctx, m, "ich2", p)
        s["x"].zero_()
        bsg.pcg_batch(ctx, m, f, s["b"], s["x"], p, s["seg"])
        return s["x"]
    p = _param(bsg, eps=1e-10, trisolve=1, nsweeps=6, restart=50, krylov=0 if case["periodic"] else 1)
    m = bsg.Matrix(ctx, s["n"], s["ia"], s["ja"], s["a"].reshape(-1), 3, case["periodic"])
    f = bsg.Factor(ctx, m, "ich2" if case["periodic"] else "ilu2", p)
    s["x"].zero_()
    if case["periodic"]:
        bsg.pcg_batch(ctx, m, f, s["b"], s["x"], p)
    else:
        bsg.gmres(ctx, m, f, s["b"][0], s["x"][0], p)
    return s["x"]


_CHANNELS = ((16, 16), (16, 32), (32, 64), (64, 64), (128, 32), (64, 16), (32, 16))


def work(case):
    kind = case["kind"]
    if kind == "batch":
        ls, lb = math.log(case["smin"]), math.log(case["smax"])
        n = case["count"] * (math.exp(2 * lb) - math.exp(2 * ls)) / (2 * (lb - ls)) if lb > ls else case["count"] * math.exp(2 * ls)
        return dict(bytes=n * (4 + 3 * 12 + 16), flops=2 * n * 5)  # the upper triangle in, b in, x out
    if kind == "elastic":
        n, nv = case["n"] ** 3, 6 if case["periodic"] else 1
        return dict(bytes=n * (4 + (14 if case["periodic"] else 27) * 76 + 48 * nv), flops=2 * n * 243 * nv)
    n = case["nx"] * case["ny"] * case["nz"]
    if kind == "product":
        entry, row, width = (27, 76, 3) if case["block"] else (7, 12, 1)
        return dict(bytes=n * (4 + entry * row + 16 * width * case["nrhs"]),
                    flops=2 * n * entry * width * width * case["nrhs"])
    if kind == "precond":
        # about 24 strict factor entries a row at these thresholds, read once
        # by an exact solve and once by each dependent sweep after the first
        passes = max(1, case["sweeps"] - 1)
        return dict(bytes=2 * n * (passes * 24 * (8 if case["fp32"] else 12) + 24), flops=2 * 2 * 24 * n * passes)
    if kind == "factor":
        return dict(bytes=n * (4 + 4 * 12 + 16 + 24 * 12), flops=2 * 24 * 24 * n / 2)  # the matrix in, the factor out
    if kind in ("driver", "krylov"):
        return dict(bytes=n * (4 + 7 * 12 + 16), flops=2 * 7 * n)
    level = (0, 1, 2, 3, 2, 1, 0)
    flops = sum(2 * 27 * ci * co * n / 8 ** l for l, (ci, co) in zip(level, _CHANNELS))
    if kind == "train":
        return dict(bytes=24 * n * case["samples"], flops=3 * flops * case["samples"])
    return dict(bytes=24 * n, flops=flops)


# ---- the same in 64 bits -----------------------------------------------------

def _sparse(d):
    """Point matrix of a case in torch CSR, float64."""
    cols, vals, keep = d["cols"], d["vals"], d["keep"]
    n = cols.shape[0]
    rows = torch.arange(n, device="cuda")[:, None].expand_as(cols)[keep]
    c, v, bs = cols[keep], vals[keep], 1
    if v.dim() == 2:
        bs = 3
        i = torch.arange(9, device="cuda")
        rows = (3 * rows[:, None] + i % 3).reshape(-1)
        c = (3 * c[:, None] + i // 3).reshape(-1)
        v = v.reshape(-1)
    order = (rows * (n * bs) + c).argsort()
    rows, c, v = rows[order], c[order], v[order]
    ia = torch.zeros(n * bs + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(torch.bincount(rows, minlength=n * bs), 0, out=ia[1:])
    return torch.sparse_csr_tensor(ia, c, v, size=(n * bs, n * bs)), rows, c, v


def _cg(A, diag, b):
    """Jacobi-preconditioned CG to the last bits, restarted once from the true residual."""
    x = torch.zeros_like(b)
    for _ in range(2):
        r = b - (A @ x[:, None])[:, 0]
        z = r / diag
        p, rz, goal = z.clone(), r @ z, 1e-30 * (b @ (b / diag))
        for it in range(20000):
            q = (A @ p[:, None])[:, 0]
            a = rz / (p @ q)
            x += a * p
            r -= a * q
            z = r / diag
            new = r @ z
            if it % 50 == 0 and not float(new) > float(goal):
                break
            p = z + (new / rz) * p
            rz = new
    return x


def _unet(x0, w, shape):
    """The network in float64: channels 16-32-64-64 down, 32-16-16 up with the
    skip connections, 3x3x3 convolutions, ReLU, mean pooling, nearest upsampling."""
    import torch.nn.functional as nnf
    W, o = [], 0
    for ci, co in _CHANNELS:
        k = w[o:o + 27 * ci * co].view(3, 3, 3, co, ci).permute(3, 4, 0, 1, 2)
        W.append(k)
        o += 27 * ci * co
    head = w[o:o + 16]

    def conv(x, k):
        with torch.backends.cudnn.flags(enabled=False):
            return torch.relu(nnf.conv3d(x, k, padding=1))

    def up(x):
        return x.repeat_interleave(2, 2).repeat_interleave(2, 3).repeat_interleave(2, 4)

    e0 = conv(x0, W[0][:, :2])
    e1 = conv(nnf.avg_pool3d(e0, 2), W[1])
    e2 = conv(nnf.avg_pool3d(e1, 2), W[2])
    e3 = conv(nnf.avg_pool3d(e2, 2), W[3])
    d2 = conv(torch.cat([up(e3), e2], 1), W[4])
    d1 = conv(torch.cat([up(d2), e1], 1), W[5])
    d0 = conv(torch.cat([up(d1), e0], 1), W[6])
    return (d0 * head.view(1, 16, 1, 1, 1)).sum(1).reshape(shape)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("precond", "factor"):
        return None  # a threshold factor is a row-by-row recurrence: hours in plain torch
    d = _inputs(case, seed)
    if kind == "product":
        A = _sparse(d)[0]
        y = (A @ d["x"].T.contiguous()).T.contiguous()
        return y
    if kind in ("unet", "train"):
        shape = (case["nz"], case["ny"], case["nx"])
        ld = torch.log(d["vals"][:, 0])
        ld = (ld - ld.mean()) / ld.std(unbiased=False)
        w = torch.as_tensor(_weights(), device="cuda").bfloat16().double().requires_grad_(kind == "train")
        for i in range(d["r"].shape[0]):
            nr = d["r"][i].norm()
            x0 = torch.stack([d["r"][i] / nr, ld]).view(1, 2, *shape)
            y = _unet(x0, w, (-1,))
            if kind == "unet":
                return y
            t = d["t"][i]
            (1 - (y @ t) ** 2 / ((y @ y) * (t @ t))).backward()
        return w.grad.cpu().numpy()
    A, rows, cols, vals = _sparse(d)
    if kind == "driver" and case["wind"]:
        dense = torch.zeros(d["n"], d["n"], dtype=torch.float64, device="cuda")
        dense[rows, cols] = vals
        return torch.linalg.solve(dense, d["b"]).cpu().numpy()
    diag = torch.zeros(A.shape[0], dtype=torch.float64, device="cuda")
    diag[rows[rows == cols]] = vals[rows == cols]
    if kind == "elastic":
        return torch.stack([_cg(A, diag, b) for b in d["load"]])
    x = _cg(A, diag, d["b"])
    return x.cpu().numpy() if kind == "driver" else x[None] if kind == "batch" else x
