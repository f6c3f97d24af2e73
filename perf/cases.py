"""The work that users of this package have it do, as cases to be timed.

A structural designer's program goes through these steps: voxelise a mesh and
mark its supports and loads, map spline coefficients to densities, set up the
multigrid operators of the density, solve for displacements, search the worst
case load, form the sensitivities and the overhang constraint, and let MMA
move the coefficients.  Each kind below is one of these steps, or the whole
objective with its gradient, called as such a program calls it: with device
tensors through the package's public entry points (the mesh input takes host
arrays).  Sizes run from small studies, which are bound by launches, over odd
boxes that fit no tile, to the 256^3 box.
"""
import math

import numpy as np
import torch

import robustoptspline3d_b200 as R
from robustoptspline3d_b200 import boundary as B
from robustoptspline3d_b200.autograd import worst_case_objective
from robustoptspline3d_b200.voxelize import voxelize

DEV = "cuda"
ORDER = 4  # tricubic splines


def listed():
    return [
        # the whole objective and its gradient: one design iteration of the 256^3 design with 32^3 coefficients
        dict(name="objective_256", kind="objective", ex=256, ey=256, ez=256, parts=28, points=0),
        # the same in a coarse study on an odd box, with the overhang constraint at sampled surface points
        dict(name="objective_odd_small", kind="objective", ex=49, ey=38, ez=56, parts=7, points=5000),
        # compliance analysis of a small cantilever in plain FP64, displacement and sensitivity
        dict(name="solve_cantilever_fp64", kind="solve", shape="cantilever", ex=64, ey=32, ez=32, precision="fp64",
             smoother="jacobi", factor=2, levels=4),
        # an ellipsoidal part in its box, smoothed by coloured Gauss-Seidel as in the reference method
        dict(name="solve_ellipsoid_gs", kind="solve", shape="ellipsoid", ex=128, ey=64, ez=64, precision="fp64",
             smoother="gs", factor=4, levels=0),
        # one load case of the largest box in mixed precision
        dict(name="solve_256_mixed", kind="solve", shape="top", ex=256, ey=256, ez=256, precision="mixed",
             smoother="chebyshev", factor=4, levels=0),
        # the same on an odd box with the package's default smoother
        dict(name="solve_odd_mixed", kind="solve", shape="cantilever", ex=93, ey=71, ez=85, precision="mixed",
             smoother="jacobi", factor=4, levels=0),
        # new density -> coarse operators, coarsest factor and smoother bounds
        dict(name="operators_256", kind="operators", ex=256, ey=256, ez=256),
        # design variables -> density and the chain back, with the sensitivity filter
        dict(name="map_256", kind="map", ex=256, ey=256, ez=256, order=4, parts=28, radius=2.0, shell=False),
        # the same on an odd box with shell elements, quadratic spline and a wider filter
        dict(name="map_odd_shell", kind="map", ex=87, ey=61, ez=75, order=3, parts=11, radius=3.5, shell=True),
        # overhang constraint on every element and its coefficient gradient
        dict(name="overhang_256", kind="overhang", ex=256, ey=256, ez=256, parts=28, mode=4),
        # one MMA step on 32^3 coefficients under volume and overhang constraints
        dict(name="mma_32768", kind="mma", n=32768, m=2),
        # mesh input: voxels, shell, support and load node masks, normals at the load nodes
        dict(name="mesh_256", kind="mesh", resolution=200, nu=512, nv=256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng, lo, hi):
    """A box whose edges lie within a factor of about two of one another."""
    n = _log(rng, lo, hi)
    return dict(zip(("ex", "ey", "ez"), (max(lo, min(hi, int(n * rng.uniform(0.7, 1.4)))) for _ in range(3))))


def draw(rng):
    kind = rng.choice(["objective", "solve", "solve", "operators", "map", "map", "overhang", "mma", "mesh"])
    if kind == "objective":
        return dict(kind=kind, **_dims(rng, 32, 176), parts=rng.randint(4, 20),
                    points=rng.choice([0, 0, _log(rng, 2000, 100000)]))
    if kind == "solve":
        precision = rng.choice(["mixed", "mixed", "fp64"])
        smoother = rng.choice(["chebyshev", "jacobi"] + (["gs"] if precision == "fp64" else []))
        return dict(kind=kind, shape=rng.choice(["cantilever", "ellipsoid", "top"]),
                    **_dims(rng, 32, 224 if precision == "mixed" else 112), precision=precision, smoother=smoother,
                    factor=4, levels=0)
    if kind == "operators":
        return dict(kind=kind, **_dims(rng, 32, 240))
    if kind == "map":
        return dict(kind=kind, **_dims(rng, 32, 240), order=rng.choice([3, 4, 4]), parts=rng.randint(4, 28),
                    radius=rng.choice([1.5, 2.0, 2.5, 3.5]), shell=rng.choice([False, True]))
    if kind == "overhang":
        return dict(kind=kind, **_dims(rng, 32, 240), parts=rng.randint(4, 28), mode=rng.choice([4, 4, 5]))
    if kind == "mma":
        return dict(kind=kind, n=_log(rng, 512, 262144), m=rng.choice([1, 2, 2]))
    nu = _log(rng, 32, 512)
    return dict(kind=kind, resolution=_log(rng, 24, 200), nu=nu, nv=max(16, nu // rng.choice([2, 3])))


# ------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(1000003 * (seed % 1000003) + 17)


def _uniform(shape, lo, hi, gen):
    return lo + (hi - lo) * torch.rand(shape, generator=gen, device=DEV, dtype=torch.float32)


def _density(shape, gen):
    """i.i.d. U[0.2, 1], then one 3x3x3 mean over the neighbours in the box."""
    rho = _uniform(shape, 0.2, 1.0, gen)
    return torch.nn.functional.avg_pool3d(rho[None, None], 3, 1, 1, count_include_pad=False)[0, 0].contiguous()


def _coefficients(n, gen):
    return (0.5 + 0.15 * torch.randn(n, generator=gen, device=DEV, dtype=torch.float32)).clamp_(0, 1)


def _box(c, shape):
    """(element mask, fixed node area, load node area) of the box problems."""
    ex, ey, ez = c["ex"], c["ey"], c["ez"]
    em = np.ones((ez, ey, ex), np.uint8)
    fa = np.zeros((ez + 1, ey + 1, ex + 1), np.uint8)
    la = np.zeros_like(fa)
    if shape == "cantilever":  # x = 0 clamped, load on the mid-height line of the other end
        fa[:, :, 0] = 1
        la[ez // 2, :, ex] = 1
    elif shape == "top":  # bottom clamped, load on the top face
        fa[0] = 1
        la[ez] = 1
    else:  # ellipsoid in the box, its lowest nodes clamped, load on the rest of its skin
        z, y, x = np.ogrid[:ez, :ey, :ex]
        h = [(n / 2 - 2) for n in (ex, ey, ez)]
        d = [((t + 0.5 - n / 2) / r) ** 2 for t, n, r in zip((x, y, z), (ex, ey, ez), h)]
        em[d[0] + d[1] + d[2] > 1] = 0
        low = int(np.flatnonzero(em.any(axis=(1, 2)))[0])
        fa[: low + 1] = 1
        la[ez // 2:] = 1
    return em, fa, la


def _config(c, precision="mixed", smoother="chebyshev"):
    sm = {"gs": R.rso.SMOOTH_GS, "jacobi": R.rso.SMOOTH_JACOBI, "chebyshev": R.rso.SMOOTH_CHEBYSHEV}[smoother]
    return R.Config(precision=R.rso.MIXED if precision == "mixed" else R.rso.FP64, smoother=sm, omega=0.8,
                    cheb_lower=0.07, first_factor=c.get("factor", 4), n_levels=c.get("levels", 0))


def _load(grid, shape, gen):
    """A load on the load nodes: downwards with some scatter, or of random directions."""
    nodes = torch.as_tensor(grid.load_nodes(), device=DEV).long()
    f = torch.zeros(3, grid.nn, dtype=torch.float64, device=DEV)
    if shape == "cantilever":
        f[2, nodes] = -1.0
    w = torch.randn(3, len(nodes), generator=gen, device=DEV, dtype=torch.float64)
    f[:, nodes] += w * (0.1 if shape == "cantilever" else 1.0)
    return (f / len(nodes)).reshape(-1)


def _torus(nu, nv, tilt):
    a = np.arange(nu) * (2 * np.pi / nu)
    b = np.arange(nv) * (2 * np.pi / nv)
    a, b = np.meshgrid(a, b, indexing="ij")
    v = np.stack([(2 + 0.7 * np.cos(b)) * np.cos(a), (2 + 0.7 * np.cos(b)) * np.sin(a), 0.7 * np.sin(b)], -1)
    c, s = np.cos(tilt), np.sin(tilt)
    v = v.reshape(-1, 3) @ np.array([[1, 0, 0], [0, c, -s], [0, s, c]])
    i, j = np.meshgrid(np.arange(nu), np.arange(nv), indexing="ij")
    p, q = i * nv + j, ((i + 1) % nu) * nv + j
    p1, q1 = i * nv + (j + 1) % nv, ((i + 1) % nu) * nv + (j + 1) % nv
    f = np.stack([np.stack([p, q, q1], -1), np.stack([p, q1, p1], -1)], 2).reshape(-1, 3)
    return v.astype(np.float32), f.astype(np.int32)


def _mesh(c, seed):
    rng = np.random.default_rng(seed)
    v, f = _torus(c["nu"], c["nv"], rng.uniform(0.05, 0.45))
    # points of a grid of the voxels' spacing along the mesh: where the load nodes lie
    h = float(np.ptp(v, axis=0).max()) / c["resolution"]
    near = v[rng.permutation(len(v))[: len(v) // 8]].astype(np.float64)
    return v, f, np.round(near / h) * h


def prepare(case, seed):
    c, gen, kind = case, _gen(seed), case["kind"]
    s = {"case": c}
    if kind == "mma":
        n, m = c["n"], c["m"]
        s["mma"] = R.MMA(n, m, 0.0, 1.0)
        s["x"] = _coefficients(n, gen).double()
        noise = torch.randn(m + 1, n, generator=gen, device=DEV, dtype=torch.float64)
        s["df"] = -torch.exp(noise[0])
        s["dg"] = (1e3 / n) * torch.stack([1 + 0.2 * noise[1]] + [noise[2]] * (m - 1))
        s["g"] = np.array([200.0] + [30.0] * (m - 1))
        s["mma"].set_x(s["x"])
        return s
    if kind == "mesh":
        s["v"], s["f"], s["points"] = _mesh(c, seed)
        s["fix"] = [B.halfspace(0, 0, -1, -0.5, closed=True), B.sphere((2, 0, 0), 0.5)]
        s["load"] = [B.halfspace(0, 0, 1, -0.5)]
        return s
    shape = c.get("shape", "top")
    em, fa, la = _box(c, shape)
    cfg = _config(c, c.get("precision", "mixed"), c.get("smoother", "chebyshev"))
    s["grid"] = g = R.HierarchyGrid(em, fa, la, None, cfg)
    if kind in ("objective", "map", "overhang"):
        n = g.set_spline_partition(c["parts"], c["parts"], c["parts"], c.get("order", ORDER))
        s["coeff"] = _coefficients(n, gen)
    if kind == "objective":
        s["coeff"].requires_grad_()
        s["weights"] = torch.tensor([1.0, 1.0, 0.01], dtype=torch.float64, device=DEV)
        s["params"] = R.IterParams(ss_points=c["points"], ss_mc_res=64)
    elif kind == "map":
        s["g"] = -torch.exp(torch.randn(em.shape, generator=gen, device=DEV))
        s["shell"] = None
        if c["shell"]:  # the outermost layer of elements stays solid
            s["shell"] = np.ones(em.shape, np.uint8)
            s["shell"][1:-1, 1:-1, 1:-1] = 0
    else:
        rho = _uniform(em.shape, 0.35, 0.45, gen) if shape == "ellipsoid" else _density(em.shape, gen)
        s["rho"] = (rho * torch.as_tensor(em, device=DEV)).reshape(-1)
        if kind == "operators":
            s["u"], s["f"] = [], []
            for level in range(1, g.n_levels()):
                nn = int(np.prod(g.level_dims(level)[3:]))
                s["u"].append(torch.randn(3 * nn, generator=gen, device=DEV, dtype=torch.float64))
                s["f"].append(torch.randn(3 * nn, generator=gen, device=DEV, dtype=torch.float64))
        else:
            g.set_density(s["rho"])
            g.update_stencil()
            s["f"] = _load(g, shape, gen)
    return s


# ------------------------------------------------------------------ one pass
def run(s):
    c, kind = s["case"], s["case"]["kind"]
    if kind == "mma":
        s["mma"].set_x(s["x"])
        s["mma"].update(s["df"], s["dg"], s["g"])
        return dict(zip(("x", "L", "U", "alpha", "beta"), s["mma"].get()))
    if kind == "mesh":
        solid, res, box = voxelize(s["v"], s["f"], c["resolution"])
        shell = B.shell_elements(s["v"], s["f"], box, res, 3.0, solid)
        origin, h = B.node_grid(box, res)
        fixed = B.region_mask(s["fix"], origin, h, (res + 1,) * 3)
        load = B.region_mask(s["load"], origin, h, (res + 1,) * 3)
        return {"solid": solid, "shell": shell, "fixed": fixed, "load": load, "box": box,
                "normals": B.mesh_normals(s["v"], s["f"], s["points"])}
    g = s["grid"]
    if kind == "objective":
        s["coeff"].grad = None
        values = worst_case_objective(s["coeff"], g, s["params"])
        (values @ s["weights"]).backward()
        return {"values": values.detach(), "grad": s["coeff"].grad}
    if kind == "solve":
        u = g.solve(s["f"], tol=1e-10, max_iter=400)[0]
        return {"u": u, "compliance": g.compliance(s["f"], u), "sensitivity": g.computeSensitivity(u)}
    if kind == "operators":
        g.set_density(s["rho"])
        g.update_stencil()
        return [g.coarse_residual(k + 1, u, f) for k, (u, f) in enumerate(zip(s["u"], s["f"]))]
    if kind == "map":
        rho_hat = g.coeff2density(s["coeff"], s["shell"])
        rho = g.projectDensities(rho_hat, 8.0, s["shell"])
        sens = g.filterSensitivity(c["radius"], g.projectSensitivity(rho_hat, 8.0, s["g"]))
        return {"rho_hat": rho_hat, "rho": rho, "volume": g.volumeRatio(rho), "sens": sens,
                "dc": g.ddensity2dcoeff(sens, s["shell"])}
    value, per, dc, count, probe = g.deal_background_points(s["coeff"], 8.0, c["mode"])
    return {"value": value, "per": per, "dc": dc, "count": count, "probe": probe}


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    c, kind = case, case["kind"]
    if kind == "mma":  # x, the two asymptotes and limits, and the m + 1 gradients; some 40 Newton steps in FP64
        return {"bytes": 8.0 * c["n"] * (c["m"] + 12), "flops": 40.0 * c["n"] * (60 + 20 * c["m"])}
    if kind == "mesh":
        r = 1 << c["resolution"].bit_length()
        return {"bytes": 3.0 * r ** 3 + 2.0 * (r + 1) ** 3 + 72.0 * c["nu"] * c["nv"], "flops": 8.0 * r ** 3}
    ne = float(c["ex"] * c["ey"] * c["ez"])
    nn = float((c["ex"] + 1) * (c["ey"] + 1) * (c["ez"] + 1))
    # one application of the operator: about 200 additions and multiplications per node
    apply_k = 200.0 * nn
    if kind == "objective":  # 20 Lanczos steps of about a dozen iterations, each some six applications
        return {"bytes": 8.0 * ne + 48.0 * nn, "flops": 20 * 12 * 6 * apply_k}
    if kind == "solve":  # the load in and the displacement out; some twenty iterations
        return {"bytes": 4.0 * ne + 48.0 * nn, "flops": 20 * 6 * apply_k}
    if kind == "operators":  # the stencil of every coarse level: 243 values a node, two types
        fac = (c.get("factor", 4)) ** 3
        return {"bytes": 4.0 * ne + 1.15 * 243 * 12 * nn / fac, "flops": 2.0 * 576 * ne + 10.0 * ne}
    o = c.get("order", ORDER)
    coeff = 4.0 * (c["parts"] + o) ** 3
    if kind == "map":
        taps = 4.2 * c["radius"] ** 3
        return {"bytes": 16.0 * ne + 2 * coeff, "flops": ne * (2.0 * o * o + 2 * taps + 4 * o + 30)}
    return {"bytes": 4.0 * ne + 2 * coeff, "flops": ne * (16.0 * o * o + 60)}


# ------------------------------------------------------------------ the same in plain 64-bit torch
def _corner(t, a, dims):
    """Corner a's entries of a nodal field (..., nz, ny, nx), one per element."""
    ex, ey, ez = dims
    dx, dy, dz = a & 1, (a >> 1) & 1, a >> 2
    return t[..., dz:dz + ez, dy:dy + ey, dx:dx + ex]


def _element_matrix(nu=0.3, E=1e6):
    """Trilinear unit cube, 2x2x2 Gauss points, isotropic; degrees of freedom by node, then axis."""
    c = E / ((1 + nu) * (1 - 2 * nu))
    D = np.zeros((6, 6))
    D[:3, :3] = c * nu
    D[range(3), range(3)] = c * (1 - nu)
    D[range(3, 6), range(3, 6)] = c * (1 - 2 * nu) / 2
    K = np.zeros((24, 24))
    for q in range(8):
        gp = [0.5 + (0.5 if q >> k & 1 else -0.5) / math.sqrt(3) for k in range(3)]
        Bm = np.zeros((6, 24))
        for a in range(8):
            r = [gp[k] if a >> k & 1 else 1 - gp[k] for k in range(3)]
            d = [(1 if a >> k & 1 else -1) * r[(k + 1) % 3] * r[(k + 2) % 3] for k in range(3)]
            for k in range(3):
                Bm[k, 3 * a + k] = d[k]
            for row, (p, q2) in enumerate(((1, 2), (0, 2), (0, 1)), 3):
                Bm[row, 3 * a + p], Bm[row, 3 * a + q2] = d[q2], d[p]
        K += Bm.T @ D @ Bm / 8
    return torch.as_tensor(K, device=DEV)


def _gather(u, dims):
    return torch.stack([_corner(u[i], a, dims).reshape(-1) for a in range(8) for i in range(3)])


def _scatter(fe, dims):
    ex, ey, ez = dims
    out = torch.zeros(3, ez + 1, ey + 1, ex + 1, dtype=torch.float64, device=DEV)
    for a in range(8):
        for i in range(3):
            _corner(out[i], a, dims).add_(fe[3 * a + i].view(ez, ey, ex))
    return out


def _support(em, fa, dims):
    """Clamped nodes: surface nodes of the solid in the fixed area."""
    return torch.as_tensor(B.surface_nodes(em) & (fa > 0), device=DEV)


def _exact_solve(c, s, em, fa):
    dims = (c["ex"], c["ey"], c["ez"])
    K0 = _element_matrix()
    rp = s["rho"].double() ** 3
    free = (~_support(em, fa, dims)).double()
    diag = _scatter(K0.diagonal()[:, None] * rp, dims) * free
    inv = torch.where(diag > 0, 1 / diag.clamp_min(1e-300), 0.0)

    def apply(u):
        return _scatter(K0 @ _gather(u, dims) * rp, dims) * free

    # conjugate gradients with the diagonal, well below the case's tolerance
    r = s["f"].view(3, c["ez"] + 1, c["ey"] + 1, c["ex"] + 1) * free
    u, z = torch.zeros_like(r), inv * r
    p, rz, stop = z, torch.sum(r * z), 1e-13 * float(r.norm())
    for it in range(20000):
        q = apply(p)
        a = rz / torch.sum(p * q)
        u, r = u + a * p, r - a * q
        if it % 25 == 24 and float(r.norm()) < stop:
            break
        z = inv * r
        rz, old = torch.sum(r * z), rz
        p = z + (rz / old) * p
    ue = _gather(u, dims)
    sens = -3 * s["rho"].double() ** 2 * torch.sum(ue * (K0 @ ue), 0) * torch.as_tensor(em, device=DEV).reshape(-1)
    return {"u": u.reshape(-1), "compliance": float(torch.sum(s["f"] * u.reshape(-1))), "sensitivity": sens}


def _exact_operators(c, s, em, fa):
    """f - R K P u on every coarse level: u interpolated to the fine nodes, the element
    products with 1e6 on the clamped entries, and the transposed interpolation."""
    K0, grid, out = _element_matrix(), s["grid"], []
    fixed_fine = _support(em, fa, (c["ex"], c["ey"], c["ez"]))
    for k, (u, f) in enumerate(zip(s["u"], s["f"])):
        ce = [int(v) for v in grid.level_dims(k + 1)[:3]]
        fac = 4 << k
        dims = tuple(e * fac for e in ce)
        rp = torch.zeros(dims[::-1], dtype=torch.float64, device=DEV)
        rp[: c["ez"], : c["ey"], : c["ex"]] = s["rho"].double().view(em.shape) ** 3
        fixed = torch.zeros([d + 1 for d in dims[::-1]], dtype=torch.bool, device=DEV)
        fixed[: c["ez"] + 1, : c["ey"] + 1, : c["ex"] + 1] = fixed_fine
        P = []
        for e, d in zip(ce, dims):
            x = torch.arange(d + 1, device=DEV, dtype=torch.float64)
            P.append((1 - (x[:, None] / fac - torch.arange(e + 1, device=DEV)).abs()).clamp_min(0))
        uc = u.view(3, ce[2] + 1, ce[1] + 1, ce[0] + 1)
        uf = torch.einsum("ckji,zk,yj,xi->czyx", uc, P[2], P[1], P[0])
        free = (~fixed).double()
        r = _scatter(K0 @ _gather(uf * free, dims) * rp.reshape(-1), dims) * free
        solid = (rp > 0).double()
        touching = torch.zeros_like(free)
        for a in range(8):
            _corner(touching, a, dims).add_(solid)
        r += 1e6 * touching * fixed * uf
        rc = torch.einsum("czyx,zk,yj,xi->ckji", r, P[2], P[1], P[0])
        out.append(f - rc.reshape(-1))
        del uf, r
    return out


def _basis(n, parts, order):
    """(n, order + parts) values and derivatives of the spline basis at the element centres."""
    f32 = np.float32
    d = f32(2) * f32(n) / f32(parts + 1)
    lo, hi = f32(0) - d, f32(n) + d
    step = (hi - lo) / f32(parts + 1)
    knots, t = [lo] * order, lo
    for _ in range(parts):
        t = f32(t + step)
        knots.append(t)
    knots = np.array(knots + [hi] * order, np.float64)
    x = np.arange(n) + 0.5
    span = ((x.astype(f32) - lo) / step).astype(np.int64) + order - 1
    N = np.zeros((n, len(knots) - 1))
    N[np.arange(n), span] = 1.0
    prev = N
    for p in range(1, order):
        prev, N = N, np.zeros((n, len(knots) - 1 - p))
        for j in range(N.shape[1]):
            a, b = knots[j + p] - knots[j], knots[j + p + 1] - knots[j + 1]
            N[:, j] += (x - knots[j]) / a * prev[:, j] if a else 0
            N[:, j] += (knots[j + p + 1] - x) / b * prev[:, j + 1] if b else 0
    p, D = order - 1, np.zeros_like(N)
    for j in range(N.shape[1]):
        a, b = knots[j + p] - knots[j], knots[j + p + 1] - knots[j + 1]
        D[:, j] = (p / a * prev[:, j] if a else 0) - (p / b * prev[:, j + 1] if b else 0)
    return torch.as_tensor(N, device=DEV), torch.as_tensor(D, device=DEV)


def _spline(coeff, bx, by, bz):
    c = coeff.double().view(bz.shape[1], by.shape[1], bx.shape[1])
    return torch.einsum("kji,zk,yj,xi->zyx", c, bz, by, bx)


def _spline_t(g, bx, by, bz):
    return torch.einsum("zyx,zk,yj,xi->kji", g, bz, by, bx).reshape(-1)


def _tanh_step(r, beta):
    return (math.tanh(beta / 2) + torch.tanh(beta * (r - 0.5))) / (2 * math.tanh(beta / 2))


def _exact_map(c, s):
    N = [_basis(c[e], c["parts"], c["order"])[0] for e in ("ex", "ey", "ez")]
    rho_hat = _spline(s["coeff"], *N).clamp(1e-3, 1)
    shell = torch.zeros(rho_hat.shape, dtype=torch.bool, device=DEV)
    if s["shell"] is not None:
        shell = torch.as_tensor(s["shell"], device=DEV) > 0
    rho_hat = torch.where(shell, 1.0, rho_hat)
    rho = torch.where(shell, 1.0, _tanh_step(rho_hat, 8.0).clamp(1e-3, 1))
    t = torch.tanh(8.0 * (rho_hat - 0.5))
    g = s["g"].double() * 8.0 * (1 - t * t) / (2 * math.tanh(4.0))
    rad = c["radius"]
    k = int(rad + 0.5)
    num, den = torch.zeros_like(g), torch.zeros_like(g)
    pad = torch.nn.functional.pad
    gp, one = pad(g, (k,) * 6), pad(torch.ones_like(g), (k,) * 6)
    for dz in range(-k, k + 1):
        for dy in range(-k, k + 1):
            for dx in range(-k, k + 1):
                r = math.sqrt(dx * dx + dy * dy + dz * dz) / rad
                if r <= 1:
                    w = 1 - 6 * r * r + 8 * r ** 3 - 3 * r ** 4
                    at = tuple(slice(k + d, k + d + n) for d, n in zip((dz, dy, dx), g.shape))
                    num += w * gp[at]
                    den += w * one[at]
    sens = num / den
    # the volume is over the element count padded to 32 per colour, which this file does not restate
    return {"rho_hat": rho_hat.reshape(-1), "rho": rho.reshape(-1), "volume": None, "sens": sens.reshape(-1),
            "dc": _spline_t(torch.where(shell, 0.0, sens), *N)}


def _exact_overhang(c, s):
    (Nx, Dx), (Ny, Dy), (Nz, Dz) = (_basis(c[e], c["parts"], ORDER) for e in ("ex", "ey", "ez"))
    f = _spline(s["coeff"], Nx, Ny, Nz)
    gx, gy, gz = _spline(s["coeff"], Dx, Ny, Nz), _spline(s["coeff"], Nx, Dy, Nz), _spline(s["coeff"], Nx, Ny, Dz)
    # outward is against the gradient: the density grows along a short probe of it
    sign = -1.0
    nn = torch.sqrt(gx * gx + gy * gy + gz * gz)
    cosang = math.cos(0.75 * math.pi)
    inner = sign * gz / nn / cosang
    down = sign * gz < 0
    mid = math.cos(math.pi) / cosang
    sc = (mid - 1) / math.log(1 / 0.004 - 1)
    near = torch.exp(-200.0 * (f - 0.5) ** 2)
    e = torch.exp(-(inner - mid) / sc)
    over, d_over = 2 / (1 + e), 2 / (1 + e) ** 2 / sc * e
    lin, d_lin = torch.where(inner > 1, 15 * (inner - 1) + 1, 1.0), torch.where(inner > 1, 15.0, 1.0)
    on = down if c["mode"] % 2 == 0 else torch.ones_like(down)
    per = torch.where(on, near * over * lin, 0.0)
    A = torch.where(on, -400.0 * (f - 0.5) * near * over * lin, 0.0)
    Bw = torch.where(on, near * (d_over * lin + over * d_lin), 0.0)
    count = float(on.sum())
    den = sign * nn * nn * cosang
    dc = _spline_t(A, Nx, Ny, Nz) + _spline_t(Bw * (nn - gz * gz / nn) / den, Nx, Ny, Dz)
    dc += _spline_t(-Bw * gz * gx / nn / den, Dx, Ny, Nz) + _spline_t(-Bw * gz * gy / nn / den, Nx, Dy, Nz)
    return {"value": float(per.sum()) / count, "per": per.reshape(-1), "dc": dc / count, "count": count, "probe": None}


def _exact_normals(v, f, points):
    """Unit vector from the closest point of the mesh, turned to the face's side, by trying all faces."""
    V = torch.as_tensor(v, device=DEV).double()[torch.as_tensor(f, device=DEV).long()]
    a, b, c = V[:, 0], V[:, 1], V[:, 2]
    out = []
    for p in torch.as_tensor(points, device=DEV).split(max(1, 12_000_000 // len(V))):
        best_d = torch.full((len(p), len(V)), math.inf, dtype=torch.float64, device=DEV)
        best_q = torch.zeros(len(p), len(V), 3, dtype=torch.float64, device=DEV)
        n = torch.linalg.cross(b - a, c - a)
        t = ((p[:, None] - a) * n).sum(-1) / (n * n).sum(-1)
        q = p[:, None] - t[..., None] * n
        inside = torch.ones_like(t, dtype=torch.bool)
        for x, y in ((a, b), (b, c), (c, a)):
            inside &= (torch.linalg.cross((y - x).expand_as(q), q - x) * n).sum(-1) >= 0
            w = ((p[:, None] - x) * (y - x)).sum(-1) / ((y - x) ** 2).sum(-1)
            e = x + w.clamp(0, 1)[..., None] * (y - x)
            d = ((p[:, None] - e) ** 2).sum(-1)
            near = d < best_d
            best_d, best_q = torch.where(near, d, best_d), torch.where(near[..., None], e, best_q)
        best_d = torch.where(inside, ((p[:, None] - q) ** 2).sum(-1), best_d)
        best_q = torch.where(inside[..., None], q, best_q)
        d, k = best_d.min(1)
        r = torch.arange(len(p), device=DEV)
        dvec = best_q[r, k] - p
        t = torch.linalg.cross(a[k] - c[k], b[k] - c[k])
        dvec = torch.where(((dvec * t).sum(-1) < 0)[:, None], -dvec, dvec)
        dvec = torch.where((d.sqrt() < 1e-6)[:, None], t, dvec)
        out.append(dvec / dvec.norm(dim=1, keepdim=True))
    return torch.cat(out)


def exact(case, seed):
    c, kind = case, case["kind"]
    size = c["ex"] * c["ey"] * c["ez"] if "ex" in c else 0
    if kind in ("mma", "objective"):
        return None  # an inner iteration's last iterate; 20 solves of the whole system
    if kind == "solve" and size > 600_000:
        return None
    if kind == "mesh":
        v, f, points = _mesh(c, seed)
        if len(f) * len(points) > 400_000_000:
            return None
        return {"solid": None, "shell": None, "fixed": None, "load": None, "box": None,
                "normals": _exact_normals(v, f, points)}
    s = prepare(case, seed)
    if kind == "map":
        return _exact_map(c, s)
    if kind == "overhang":
        return _exact_overhang(c, s)
    em, fa, _ = _box(c, c.get("shape", "top"))
    return (_exact_operators if kind == "operators" else _exact_solve)(c, s, em, fa)
