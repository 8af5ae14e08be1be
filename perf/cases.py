"""The work that users of the library have it do, as measurable cases.

Every case goes through the public Python binding (Solver, Batch) with host
arrays in and host arrays out.  The element matrices are formed in prepare(),
as a program that solves several load vectors on one mesh holds them; the
`job` case forms them in the measured call.

The stopping tolerances are a few digits tighter than the 1e-5 .. 1e-8 of
everyday runs.  The fields returned are then set by the equations and not by
where the iteration happened to stop, so two builds can be compared to many
digits.  Iteration counts are not returned: they move by some per cent with
the rounding of any one operation.
"""
import math

import numpy as np
import torch

import parafem_gb300 as P

# Node positions of the 20-node brick (-1, 0, 1 along x, y, z) in Smith-Griffiths order.
_XI = np.array([-1, -1, -1, 0, 1, 1, 1, 0, -1, -1, 1, 1, -1, -1, -1, 0, 1, 1, 1, 0])
_ETA = np.array([-1] * 8 + [0] * 4 + [1] * 8)
_ZETA = np.array([-1, 0, 1, 1, 1, 0, -1, -1, -1, 1, 1, -1, -1, 0, 1, 1, 1, 0, -1, -1])
# and of the 8-node brick
_XI8 = np.array([-1, -1, 1, 1, -1, -1, 1, 1])
_ETA8 = np.array([-1, -1, -1, -1, 1, 1, 1, 1])
_ZETA8 = np.array([-1, 1, 1, -1, -1, 1, 1, -1])

_MODES = {"p121": P.MODE_P121, "fp64": P.MODE_FP64_RES, "mixed": P.MODE_MIXED, "mixed16": P.MODE_MIXED16}


def listed():
    return [
        # The smallest drop-in run: a 10^3 cube, FP64, p121's own stopping test.  Launch latency.
        dict(name="p121_10", kind="solve", mode="p121", nx=10, ny=10, nz=10, nip=27, hetero=False, bend=0.0, tol=1e-12),
        # The book's p121 deck: 40^3 elements, 2x2x2 points, the FP64 drop-in.
        dict(name="p121_book40", kind="solve", mode="p121", nx=40, ny=40, nz=40, nip=8, hetero=False, bend=0.0, tol=1e-12),
        # FP64 to a residual on an odd-sized, distorted mesh with a material of its own in every element.
        dict(name="fp64_odd", kind="solve", mode="fp64", nx=23, ny=17, nz=31, nip=27, hetero=True, bend=0.06, tol=1e-11),
        # A small mesh in the mixed mode: latency of the inner iterations and of the corrections.
        dict(name="mixed_12", kind="solve", mode="mixed", nx=12, ny=11, nz=9, nip=27, hetero=False, bend=0.05, tol=1e-11),
        # The headline path (mixed, one material) at a size that streams far more than L2 holds.
        dict(name="mixed_64", kind="solve", mode="mixed", nx=64, ny=64, nz=64, nip=27, hetero=False, bend=0.0, tol=1e-10),
        # FP16 element matrices on a heterogeneous mesh.
        dict(name="mixed16_33", kind="solve", mode="mixed16", nx=33, ny=36, nz=31, nip=27, hetero=True, bend=0.03, tol=1e-10),
        # One element matrix for the whole mesh (PCG_KM), tensor-core products.
        dict(name="pcg_km_64", kind="shared", mode="mixed", nx=64, ny=64, nz=64, nip=27, tol=1e-11),
        # Sixteen load cases of one mesh together.
        dict(name="loads_28x16", kind="multi", nx=28, ny=28, nz=28, nip=27, k=16, tol=1e-11),
        # A whole job from host arrays: mesh tables, storkm, solve, stresses of every element.
        dict(name="job_36", kind="job", mode="mixed", nx=37, ny=36, nz=35, nip=27, hetero=False, bend=0.05, tol=1e-11),
        # p122: a load increment of a Mohr-Coulomb solid, many short warm-started FP64 solves.
        dict(name="p122_10", kind="plastic", nx=10, ny=10, nz=10, nip=8),
        # p123: Laplace's equation on 8-node bricks, half the book's edge.
        dict(name="p123_100", kind="laplace", nx=100, ny=100, nz=100, tol=1e-12),
        # The serving engine: a queue of independent meshes of mixed sizes, solved as one batch.
        dict(name="serving_24", kind="serving", requests=24, lo=4, hi=18, nip=27, prec=32, tol=1e-10),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo, hi):
    n = _log_int(rng, lo, hi)
    return dict(zip(("nx", "ny", "nz"), (min(hi, max(3, int(round(n * rng.uniform(0.75, 1.25))))) for _ in range(3))))


def draw(rng):
    kind = rng.choice(["fp64", "fp64", "mixed", "mixed", "mixed16", "shared", "multi", "job", "plastic", "laplace",
                       "serving"])
    nip = rng.choice([8, 27, 27])
    if kind == "fp64":
        hetero = rng.random() < 0.4
        return dict(kind="solve", mode=rng.choice(["p121", "fp64"]), nip=27 if hetero else nip, hetero=hetero,
                    bend=rng.choice([0.0, 0.05]), tol=1e-11 if hetero else 1e-12, **_box(rng, 6, 24 if hetero else 40))
    if kind in ("mixed", "mixed16"):
        hetero = rng.random() < 0.4
        return dict(kind="solve", mode=kind, nip=27, hetero=hetero, bend=rng.choice([0.0, 0.05]),
                    tol=1e-10, **_box(rng, 8, 34 if hetero else 64))
    if kind == "shared":
        return dict(kind="shared", mode=rng.choice(["mixed", "mixed", "fp64"]), nip=nip, tol=1e-11, **_box(rng, 9, 48))
    if kind == "multi":
        return dict(kind="multi", nip=27, k=8 * rng.randint(1, 4), tol=1e-11, **_box(rng, 7, 26))
    if kind == "job":
        return dict(kind="job", mode=rng.choice(["p121", "mixed"]), nip=27, hetero=False, bend=rng.choice([0.0, 0.05]),
                    tol=1e-11, **_box(rng, 8, 34))
    if kind == "plastic":
        return dict(kind="plastic", nip=8, **_box(rng, 4, 10))
    if kind == "laplace":
        return dict(kind="laplace", tol=1e-12, **_box(rng, 16, 100))
    return dict(kind="serving", requests=rng.randint(5, 24), lo=rng.randint(3, 6), hi=rng.randint(8, 18), nip=27,
                prec=rng.choice([32, 32, 16, 64]), tol=1e-10)


# ---------------------------------------------------------------------------
# inputs
def _mesh(nx, ny, nz, xi, eta, zeta):
    """Bricks of the given local nodes: g_num (nels, nod), coords (nn, 3).  Elements run x fastest, then z, then
    y, and nodes are numbered plane by plane in y, as the reference's box geometries are."""
    gx, gy, gz = 2 * nx + 1, 2 * ny + 1, 2 * nz + 1
    iy, iz, ix = np.meshgrid(np.arange(ny), np.arange(nz), np.arange(nx), indexing="ij")
    iy, iz, ix = (a.reshape(-1, 1) for a in (iy, iz, ix))
    cell = ((2 * iy + 1 + eta) * gz + (2 * iz + 1 + zeta)) * gx + (2 * ix + 1 + xi)
    used = np.zeros(gx * gy * gz, bool)
    used[cell.ravel()] = True
    at = np.flatnonzero(used)
    number = np.cumsum(used, dtype=np.int32)
    coords = 0.5 * np.stack([at % gx, at // (gx * gz), (at // gx) % gz], axis=1)
    return number[cell], coords


def _bent(coords, amount, top):
    """A smooth distortion of the box that keeps its base and its top plane."""
    if not amount:
        return coords
    w = np.sin(math.pi * coords[:, 2] / top)
    shift = np.stack([np.sin(1.3 * coords[:, 1]), np.cos(0.9 * coords[:, 0]), np.sin(0.7 * coords[:, 0])], axis=1)
    return coords + amount * w[:, None] * shift


def _solid(c, seed):
    """Mesh, numbering, material and loads of a box of 20-node bricks on a fixed base."""
    rng = np.random.default_rng([seed, c["nx"], c["ny"], c["nz"]])
    g_num, coords = _mesh(c["nx"], c["ny"], c["nz"], _XI, _ETA, _ZETA)
    coords = _bent(coords, c.get("bend", 0.0), float(c["nz"]))
    nn, nels = coords.shape[0], g_num.shape[0]
    free = np.repeat((coords[:, 2] > 1e-9)[:, None], 3, axis=1)
    eq = np.where(free, np.cumsum(free.ravel(), dtype=np.int32).reshape(nn, 3), 0).astype(np.int32)
    neq = int(free.sum())
    if c.get("hetero"):
        e, v = np.exp(rng.uniform(0.0, math.log(1000.0), nels)), rng.uniform(0.2, 0.35, nels)
    else:
        e, v = np.array([100.0 * rng.uniform(0.5, 2.0)]), np.array([rng.uniform(0.25, 0.32)])
    top = np.flatnonzero(coords[:, 2] > c["nz"] - 1e-9)

    def loads(k):
        r = np.zeros((neq, k), order="F")
        r[eq[top, 2] - 1] = -rng.uniform(0.5, 1.5, (top.size, k)) / top.size
        r[eq[top, 0] - 1] = rng.uniform(-0.2, 0.2, (top.size, k)) / top.size
        return r

    return dict(g_num=g_num, g_g=eq[g_num - 1].reshape(nels, 60),
                g_coord=np.ascontiguousarray(coords[g_num - 1].transpose(0, 2, 1)), nn=nn, neq=neq, e=e, v=v,
                loads=loads, eq=eq, coords=coords)


def _potential(c, seed):
    """A box of 8-node bricks, potential 0 on the base, sources and sinks on the top face."""
    rng = np.random.default_rng([seed, c["nx"], c["ny"], c["nz"]])
    g_num, coords = _mesh(c["nx"], c["ny"], c["nz"], _XI8, _ETA8, _ZETA8)
    coords = 0.1 * coords
    free = coords[:, 2] > 1e-9
    eq = np.where(free, np.cumsum(free, dtype=np.int32), 0).astype(np.int32)
    neq = int(free.sum())
    top = np.flatnonzero(coords[:, 2] > 0.1 * c["nz"] - 1e-9)
    r = np.zeros(neq)
    r[eq[top] - 1] = rng.uniform(-1.0, 3.0, top.size)
    return dict(g_num=g_num, g_g=eq[g_num - 1], g_coord=np.ascontiguousarray(coords[g_num - 1].transpose(0, 2, 1)),
                nn=coords.shape[0], neq=neq, r=r, k=(2.0, 1.0, 3.0))


def _requests(c, seed):
    """The served meshes: the sizes from the case, materials and loads from the seed."""
    size = np.random.default_rng([c["requests"], c["lo"], c["hi"]])
    out = []
    for i in range(c["requests"]):
        nx, ny, nz = (int(n) for n in size.integers(c["lo"], c["hi"] + 1, 3))
        m = _solid(dict(nx=nx, ny=ny, nz=nz), seed * 64 + i)
        m["r"] = np.ascontiguousarray(m["loads"](1)[:, 0])
        out.append(m)
    return out


_PLASTIC = dict(phi=20.0, c=30.0, psi=5.0, e=1.0e4, v=0.3, qinc=[200.0, 60.0], plasits=60, cjits=3000, plastol=1e-3,
                cjtol=1e-12)


def _plastic(c, seed):
    """A footing: the middle of the top face loaded downwards, yielding from the first increment."""
    m = _solid(dict(c, bend=0.0), seed)
    rng = np.random.default_rng([seed, 122])
    x, y, z = m["coords"].T
    patch = (z > c["nz"] - 1e-9) & (np.abs(x - 0.5 * c["nx"]) < 0.26 * c["nx"]) & (np.abs(y - 0.5 * c["ny"]) < 0.26 * c["ny"])
    m["r"] = np.zeros(m["neq"])
    m["r"][m["eq"][patch, 2] - 1] = -rng.uniform(0.9, 1.1, int(patch.sum())) / 6.0
    return m


# ---------------------------------------------------------------------------
def _solver(m, nip, form=True):
    s = P.Solver()
    s.setup(m["g_num"], m["g_g"], m["g_coord"], m["nn"], m["neq"])
    s.set_material(m["e"], m["v"])
    if form:
        s.form_storkm(nip)
    return s


def prepare(case, seed):
    kind = case["kind"]
    if kind == "laplace":
        m = _potential(case, seed)
        s = P.Solver()
        s.setup_scalar8(m["g_num"], m["g_g"], m["g_coord"], m["nn"], m["neq"])
        s.form_storkc(8, *m["k"])
        return dict(case=case, s=s, r=m["r"])
    if kind == "serving":
        reqs = _requests(case, seed)
        need = sum(60_000 * q["g_num"].shape[0] for q in reqs) + (1 << 28)
        return dict(case=case, b=P.Batch(need, 64, prec=case["prec"]), reqs=reqs, cap=max(q["neq"] for q in reqs))
    if kind == "plastic":
        m = _plastic(case, seed)
        m["e"], m["v"] = np.array([_PLASTIC["e"]]), np.array([_PLASTIC["v"]])
        return dict(case=case, s=_solver(m, case["nip"]), r=m["r"])
    m = _solid(case, seed)
    if kind == "job":
        m["r"] = np.ascontiguousarray(m["loads"](1)[:, 0])
        return dict(case=case, s=P.Solver(), m=m)
    if kind == "shared":
        s = _solver(m, case["nip"], form=False)
        s.set_shared_km(s.form_km(1, case["nip"]))
    else:
        s = _solver(m, case["nip"])
    r = m["loads"](case.get("k", 1))
    return dict(case=case, s=s, r=r if kind == "multi" else np.ascontiguousarray(r[:, 0]))


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind in ("solve", "shared"):
        return state["s"].solve(state["r"], c["tol"], 30000, _MODES[c["mode"]])[0]
    if kind == "multi":
        return state["s"].solve_multi(state["r"], c["tol"], 30000, 16)[0]
    if kind == "laplace":
        return state["s"].solve(state["r"], c["tol"], 30000, P.MODE_P121)[0]
    if kind == "plastic":
        p = _PLASTIC
        res, totd = state["s"].p122_solve(c["nip"], p["phi"], p["c"], p["psi"], p["qinc"], p["plasits"], p["cjits"],
                                          p["plastol"], p["cjtol"], state["r"], keep_totd=True)
        return res[:, :4].copy(), totd
    if kind == "serving":
        b, ids = state["b"], []
        for q in state["reqs"]:
            ids.append(b.admit(q["g_num"], q["g_g"], q["g_coord"], q["nn"], q["neq"], q["e"], q["v"], q["r"],
                               tol=c["tol"], nip=c["nip"]))
        done = b.run_all(state["cap"])
        return [done[i][2] for i in ids]
    s, m = state["s"], state["m"]
    s.setup(m["g_num"], m["g_g"], m["g_coord"], m["nn"], m["neq"])
    s.set_material(m["e"], m["v"])
    s.form_storkm(c["nip"])
    x = s.solve(m["r"], c["tol"], 30000, _MODES[c["mode"]])[0]
    return x, s.element_stresses(x)


# ---------------------------------------------------------------------------
def _iterations(c, n):
    """PCG iterations of a box with n elements along its longest edge, near what the solver takes to the tolerance."""
    per = 28.0 if c.get("hetero") is not True else 120.0
    return per * n + 20.0


def work(case):
    """Bytes and operations per pass.  An iteration reads every distinct element-matrix entry once (packed symmetric,
    in the precision of the products), the connectivity, and moves eleven vector streams in FP64."""
    kind = case["kind"]
    if kind == "serving":
        size = np.random.default_rng([case["requests"], case["lo"], case["hi"]])
        b = f = 0.0
        for _ in range(case["requests"]):
            nx, ny, nz = (int(n) for n in size.integers(case["lo"], case["hi"] + 1, 3))
            w = work(dict(kind="job", mode={64: "fp64", 32: "mixed", 16: "mixed16"}[case["prec"]], nx=nx, ny=ny, nz=nz,
                          nip=case["nip"], tol=case["tol"]))
            b, f = b + w["bytes"], f + w["flops"]
        return {"bytes": b, "flops": f}
    nels = case["nx"] * case["ny"] * case["nz"]
    its = _iterations(case, max(case["nx"], case["ny"], case["nz"]))
    if kind == "laplace":
        nn = (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)
        its = 4.0 * max(case["nx"], case["ny"], case["nz"]) + 20.0
        return {"bytes": its * (nels * (36 * 8 + 32) + 88.0 * nn) + 16.0 * nn, "flops": its * (128.0 * nels + 14.0 * nn)}
    neq = 3 * (4 * nels + 3 * (case["nx"] * case["ny"] + case["ny"] * case["nz"] + case["nx"] * case["nz"]))
    k = case.get("k", 1)
    per = {"p121": 8, "fp64": 8, "mixed": 4, "mixed16": 2}.get(case.get("mode"), 4 if kind == "multi" else 8)
    matrix = 0 if kind == "shared" else 1830 * per
    if kind == "plastic":
        its *= 15.0 * len(_PLASTIC["qinc"])
    b = its * (nels * (matrix + 80.0) + 88.0 * neq * k) + 16.0 * neq * k
    f = its * k * (7200.0 * nels + 14.0 * neq)
    if kind == "job":
        b += nels * (80.0 + 240.0 + 480.0 + 1830 * 8.0 + 48.0)
        f += nels * case["nip"] * 210 * 18.0
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# 64-bit values of the results: element matrices, assembled products and a conjugate-gradient solve in plain torch
def _gauss(nip):
    """Points and weights of SAMPLE; its 27-point rule takes 5./9. and 8./9. in single precision for one factor."""
    if nip == 8:
        r = 1.0 / math.sqrt(3.0)
        return [((sx * r, sy * r, sz * r), 1.0) for sx in (-1, 1) for sy in (-1, 1) for sz in (-1, 1)]
    r, w = 0.2 * math.sqrt(15.0), (5.0 / 9.0, 8.0 / 9.0, 5.0 / 9.0)
    f = (float(np.float32(5.0) / np.float32(9.0)), float(np.float32(8.0) / np.float32(9.0)))
    pts = []
    for j, eta in enumerate((-r, 0.0, r)):
        for i, xi in enumerate((-r, 0.0, r)):
            for k, zeta in enumerate((-r, 0.0, r)):
                pts.append(((xi, eta, zeta), w[i] * w[k] * f[1 if j == 1 else 0]))
    return pts


def _shape_der(p, nod):
    """d N / d(xi, eta, zeta) of the serendipity brick (20) or the trilinear brick (8) at p: (3, nod)."""
    x, y, z = (torch.tensor(v, dtype=torch.float64, requires_grad=True) for v in p)
    if nod == 8:
        a, b, c = (torch.tensor(v, dtype=torch.float64) for v in (_XI8, _ETA8, _ZETA8))
        n = (1 + a * x) * (1 + b * y) * (1 + c * z) / 8
    else:
        a, b, c = (torch.tensor(v, dtype=torch.float64) for v in (_XI, _ETA, _ZETA))
        fx, fy, fz = 1 + a * x, 1 + b * y, 1 + c * z
        corner = fx * fy * fz * (a * x + b * y + c * z - 2) / 8
        n = torch.where(a == 0, (1 - x * x) * fy * fz / 4,
                        torch.where(b == 0, (1 - y * y) * fx * fz / 4,
                                    torch.where(c == 0, (1 - z * z) * fx * fy / 4, corner)))
    rows = [torch.stack(torch.autograd.grad(n[i], (x, y, z), retain_graph=True)) for i in range(nod)]
    return torch.stack(rows, dim=1).detach()


def _matrices(coord, nip, e=None, v=None, k=None):
    """Element matrices (nels, nd, nd): B'DB for a solid, grad' diag(k) grad for a potential.  coord (nels, 3, nod)."""
    nels, _, nod = coord.shape
    out = torch.zeros(nels, *((nod, nod) if k else (3 * nod, 3 * nod)), dtype=torch.float64, device=coord.device)
    pts = [(_shape_der(p, nod).to(coord.device), w) for p, w in _gauss(nip)]
    for at in range(0, nels, 20000):
        co = coord[at:at + 20000]
        for der, w in pts:
            jac = torch.einsum("dn,ejn->edj", der, co)
            det = torch.linalg.det(jac)
            g = torch.linalg.solve(jac, der.expand(co.shape[0], 3, nod))
            wd = (det * w)[:, None, None]
            if k:
                kd = torch.tensor(k, dtype=torch.float64, device=co.device)[None, :, None]
                out[at:at + 20000] += torch.bmm(g.transpose(1, 2), g * kd * wd)
                continue
            ee, vv = (t[at:at + 20000] if t.numel() > 1 else t for t in (e, v))
            lam, mu = ee * vv / ((1 + vv) * (1 - 2 * vv)), ee / (2 * (1 + vv))
            gg = torch.einsum("ian,ibm->inamb", g, g) * wd[..., None, None]   # g_a(n) g_b(m)
            tr = gg.diagonal(dim1=2, dim2=4).sum(-1)
            block = lam.view(-1, 1, 1, 1, 1) * gg + mu.view(-1, 1, 1, 1, 1) * gg.transpose(2, 4)
            block += (mu.view(-1, 1, 1) * tr)[:, :, None, :, None] * torch.eye(3, dtype=torch.float64, device=co.device)[None, None, :, None, :]
            out[at:at + 20000] += block.reshape(co.shape[0], 3 * nod, 3 * nod)
    return out


def _solution(km, g_g, neq, r):
    """K x = r by Jacobi-preconditioned conjugate gradients in 64 bits, restarted once on the true residual."""
    dev, k = km.device, r.shape[1]
    idx = torch.from_numpy(np.ascontiguousarray(g_g)).to(dev).long()
    one = km.shape[0] == 1

    def product(p):
        full = torch.cat([torch.zeros(1, k, dtype=torch.float64, device=dev), p])
        pe = full[idx]
        ue = torch.matmul(km[0], pe) if one else torch.bmm(km, pe)
        return torch.zeros_like(full).index_add_(0, idx.reshape(-1), ue.reshape(-1, k))[1:]

    kd = km.diagonal(dim1=1, dim2=2).expand(idx.shape[0], idx.shape[1])
    dinv = 1.0 / torch.zeros(neq + 1, dtype=torch.float64, device=dev).index_add_(0, idx.reshape(-1), kd.reshape(-1))[1:, None]
    f = torch.from_numpy(np.ascontiguousarray(r)).to(dev)
    x = torch.zeros_like(f)
    for stop in (1e-12, 1e-5):
        res = f - product(x)
        start = res.norm(dim=0)
        c, z = torch.zeros_like(f), dinv * res
        p, up = z.clone(), (res * z).sum(0)
        for it in range(30000):
            u = product(p)
            alpha = up / (p * u).sum(0)
            c += alpha * p
            res -= alpha * u
            if it % 50 == 49 and bool((res.norm(dim=0) <= stop * start).all()):
                break
            z = dinv * res
            new = (res * z).sum(0)
            p = z + (new / up) * p
            up = new
        x = x + c
    return x


def _stresses(m, x, dev):
    """D B u at the centroid of every element, ordered sx, sy, sz, txy, tyz, tzx."""
    der = _shape_der((0.0, 0.0, 0.0), 20).to(dev)
    co = torch.from_numpy(m["g_coord"]).to(dev)
    g = torch.linalg.solve(torch.einsum("dn,ejn->edj", der, co), der.expand(co.shape[0], 3, 20))
    full = torch.cat([torch.zeros(1, dtype=torch.float64, device=dev), x])
    ue = full[torch.from_numpy(m["g_g"]).to(dev).long()].reshape(-1, 20, 3)
    grad = torch.einsum("edn,enj->ejd", g, ue)
    e, v = (torch.from_numpy(m[q]).to(dev).view(-1, 1, 1) for q in ("e", "v"))
    eps = 0.5 * (grad + grad.transpose(1, 2))
    lam, mu = e * v / ((1 + v) * (1 - 2 * v)), e / (2 * (1 + v))
    sig = 2 * mu * eps + lam * eps.diagonal(dim1=1, dim2=2).sum(-1)[:, None, None] * torch.eye(3, dtype=torch.float64, device=dev)
    return torch.stack([sig[:, 0, 0], sig[:, 1, 1], sig[:, 2, 2], sig[:, 0, 1], sig[:, 1, 2], sig[:, 2, 0]], dim=1)


def exact(case, seed):
    kind = case["kind"]
    nels = 0 if kind == "serving" else case["nx"] * case["ny"] * case["nz"]
    if kind == "plastic" or kind == "multi" and nels * case["k"] > 600_000 or case.get("hetero") and nels > 40_000:
        return None   # no closed form, or too long in plain torch
    dev = torch.device("cuda")
    on = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    if kind == "laplace":
        m = _potential(case, seed)
        km = _matrices(on(m["g_coord"]), 8, k=m["k"])
        return _solution(km, m["g_g"], m["neq"], m["r"][:, None])[:, 0].cpu().numpy()
    if kind == "serving":
        out = []
        for m in _requests(case, seed)[:6]:
            km = _matrices(on(m["g_coord"]), case["nip"], on(m["e"]), on(m["v"]))
            out.append(_solution(km, m["g_g"], m["neq"], m["r"][:, None])[:, 0].cpu().numpy())
        return out + [None] * (case["requests"] - len(out))
    m = _solid(case, seed)
    if kind == "shared":
        m["g_coord"] = m["g_coord"][:1]
    r = m["loads"](case.get("k", 1))
    km = _matrices(on(m["g_coord"]), case["nip"], on(m["e"]), on(m["v"]))
    x = _solution(km, m["g_g"], m["neq"], r)
    if kind == "multi":
        return x.cpu().numpy()
    if kind == "job":
        return x[:, 0].cpu().numpy(), _stresses(m, x[:, 0], dev).cpu().numpy()
    return x[:, 0].cpu().numpy()
