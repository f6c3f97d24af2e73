"""Kernels and dispatch rules at the sizes where they can go wrong (edges of tiles and chunks,
remainders, the smallest and largest of a range), against the FP64 oracle."""
import numpy as np
import pytest

import mesh_shapes as M
import problems as P
from test_gpu_00_parity import make, rel, t

pytestmark = pytest.mark.gpu


# node boxes one short of, on and one past the 31 x 7 tile, and depths that give z chunks of
# 2, 4, 8, 16 and 32 planes with full and ragged last chunks
@pytest.mark.parametrize("dims", [(3, 2, 1), (30, 6, 1), (31, 7, 2), (29, 5, 41), (62, 41, 70), (93, 97, 65),
                                  (130, 118, 96)])
def test_fine_fp64_chunks(oracle, cuda, dims):
    """FP64 K u, residual and damped Jacobi step; 1e-12 relative, the bound of the FP64 operator pieces."""
    g, o = make(oracle, P.cantilever(*dims), n_levels=2 if dims[0] < 40 else 0, first_factor=2 if dims[0] < 40 else 4)
    rng = np.random.default_rng(7)
    fix = np.tile((o.node_class() & 4) > 0, 3)
    u, f = (np.where(fix, 0.0, rng.standard_normal(3 * o.nn)) for _ in range(2))
    assert rel(g.applyK(t(u, cuda)).cpu().numpy(), o.apply_K(u)) < 1e-12
    assert rel(g.update_residual(t(u, cuda), t(f, cuda)).cpu().numpy(), o.residual(u, f)) < 1e-12
    g.update_stencil()
    jac = g.gs_relax(0, t(u, cuda), t(f, cuda), kind=1, omega=0.3).cpu().numpy()
    assert rel(jac, o.smooth(0, u, f, kind=1, omega=0.3, sweeps=1)) < 1e-12


# the packed FP32 kernel's tiles (31 nodes by 3, 7 or 15): one short of, on and past a tile edge in x
# and y, where a thread's second column or its right neighbour is missing
@pytest.mark.parametrize("rows", [2, 4, 8])
@pytest.mark.parametrize("dims", [(6, 4, 3), (29, 13, 9), (30, 14, 10), (31, 15, 17), (33, 6, 12)])
def test_fine_fp32_tile_edges(oracle, cuda, dims, rows):
    """FP32 K u, residual and Chebyshev step; 2e-5 relative, the bound of the FP32 operator pieces."""
    g, o = make(oracle, P.cantilever(*dims), n_levels=2, first_factor=2)
    g.set_launch_shapes(fine_rows=rows)
    rng = np.random.default_rng(9)
    cls = o.node_class()
    fix = np.tile(((cls & 4) > 0) | ((cls & 1) == 0), 3)
    u, f, up = (np.where(fix, 0.0, rng.standard_normal(3 * o.nn)) for _ in range(3))
    assert rel(g.fine_sweep_fp32(1, t(u, cuda)).cpu().numpy(), o.apply_K(u)) < 2e-5
    assert rel(g.fine_sweep_fp32(0, t(u, cuda), t(f, cuda)).cpu().numpy(), o.residual(u, f)) < 2e-5
    step = o.smooth(0, u, f, kind=1, omega=0.3, sweeps=1) + 0.7 * (u - up)
    assert rel(g.fine_sweep_fp32(2, t(u, cuda), t(f, cuda), t(up, cuda), omega=0.3, c1=0.7).cpu().numpy(), step) < 2e-5


# coarse levels of 2 to 17 nodes an edge: colours of one node, of fewer and of more than the 32 a CTA
# takes, with a ragged last CTA; the ellipsoid leaves inactive nodes inside the box
@pytest.mark.parametrize("gen", [lambda: P.cantilever(6, 4, 3), lambda: P.cantilever(30, 21, 13),
                                 lambda: P.ellipsoid(40, 24, 20)])
@pytest.mark.parametrize("reverse", [0, 1])
def test_coarse_gauss_seidel(oracle, cuda, gen, reverse):
    """FP64 coloured sweeps on every coarse level; 1e-12 relative, the bound of the FP64 operator pieces."""
    g, o = make(oracle, gen(), n_levels=3, first_factor=2)
    g.update_stencil()
    o.update_stencil()
    rng = np.random.default_rng(11)
    for lvl in range(1, o.n_levels()):
        mask = np.tile(o.level_masks(lvl)[1], 3)
        u, f = (rng.standard_normal(mask.size) * mask for _ in range(2))
        got = g.gs_relax(lvl, t(u, cuda), t(f, cuda), sweeps=2, reverse=reverse).cpu().numpy()
        assert rel(got, o.smooth(lvl, u, f, kind=0, omega=1.0, sweeps=2, reverse=reverse)) < 1e-12, lvl


# bottoms whose levels all fit in shared memory (one tile and a ragged last one, several levels), and
# one whose first level has more stencil tiles than the GPU has SMs and is streamed
@pytest.mark.parametrize("dims", [(17, 9, 13), (64, 64, 64), (93, 71, 85), (128, 128, 64)])
@pytest.mark.parametrize("pre,post", [(2, 2), (1, 3)])
def test_bottom_kernel_levels(cuda, dims, pre, post):
    """Mixed solves with the persistent bottom kernel against per-level launches, one system and a
    batch: the same solution to 1e-8 and iterations within one, as for every launch shape."""
    from robustoptspline3d_b200 import Config, HierarchyGrid
    prob = P.cantilever(*dims)
    g = HierarchyGrid(prob["emask"], prob["fixed"], prob["load"], None,
                      Config(poisson_ratio=0.4, pre=pre, post=post, smoother=2, first_factor=2 if dims[0] < 32 else 4,
                             n_levels=3 if dims[0] < 32 else 0))
    g.set_density(prob["rho"].astype(np.float32).ravel())
    g.update_stencil()
    f = t(prob["f"], cuda)
    F = cuda.stack([f, 0.5 * f.flip(0)])
    assert g.n_levels() > 2
    g.set_launch_shapes(4, 1)
    got = [g.solve(f, tol=1e-10) for _ in range(3)]  # plain launches, the capture, a replay
    batch, infos = g.solve_batch(F, tol=1e-10)
    g.set_launch_shapes(4, -1)
    want, it, _, _ = g.solve(f, tol=1e-10)
    for u, k, _, _ in got:
        assert rel(u.cpu().numpy(), want.cpu().numpy()) < 1e-8 and abs(k - it) <= 1
    assert rel(batch[0].cpu().numpy(), want.cpu().numpy()) < 1e-8 and abs(infos[0][0] - it) <= 1


# boxes below, on and past the 32 x 8 tile and the 128-element row segment; radii on both sides of
# every reach the tiled filter is built for and past the last one (the general kernel)
@pytest.mark.parametrize("dims,radius", [((33, 9, 10), 1.0), ((33, 9, 10), 1.9), ((32, 8, 64), 2.0), ((70, 5, 3), 2.99),
                                         ((40, 24, 24), 3.5), ((31, 17, 20), 4.99), ((31, 17, 20), 5.0), ((9, 8, 8), 0.7)])
@pytest.mark.parametrize("gen", [P.cantilever, lambda *d: P.voids_box(*d, nvoids=1)])
def test_filter_tiles(oracle, cuda, gen, dims, radius):
    """FP64 sums rounded to FP32 once: 1e-6 relative (half an FP32 ulp is 6e-8); in place as well."""
    small = min(dims) < 8
    g, o = make(oracle, gen(*dims), n_levels=2 if small else 0, first_factor=2 if small else 4)
    x = np.random.default_rng(3).standard_normal(o.ne).astype(np.float32)
    want = o.filter(radius, x.astype(np.float64))
    assert rel(g.filterSensitivity(radius, x).cpu().numpy(), want) < 1e-6
    assert rel(g.densityFilter(radius, x, adjoint=True).cpu().numpy(),
               o.density_filter_adjoint(radius, x.astype(np.float64))) < 1e-6
    buf = t(x, cuda)
    assert g.lib.rso_filter(g.h, radius, buf.data_ptr(), buf.data_ptr()) == 0
    assert rel(buf.cpu().numpy(), want) < 1e-6


# orders 2 to 5 (2 and 5 outside the probe bound's C1 splines and at its end), one to many knots per
# element row segment, rows longer than a segment; amplitudes for which the probe's sign is known
# (1), unknown for many (30) and for all elements (3000)
@pytest.mark.parametrize("dims,order,parts", [((20, 12, 9), 2, (3, 3, 2)), ((150, 11, 7), 3, (40, 0, 3)),
                                              ((129, 9, 13), 4, (9, 4, 5)), ((24, 18, 20), 5, (4, 3, 6)),
                                              ((12, 10, 8), 4, (30, 1, 9))])
@pytest.mark.parametrize("amplitude", [1.0, 30.0, 3000.0])
def test_spline_rows_and_overhang(oracle, cuda, dims, order, parts, amplitude):
    """Density map and adjoint 1e-6, constraint value 1e-5 and gradient 1e-4 relative, counts and
    probe sums equal: the bounds of these maps in the parity tests."""
    g, o = make(oracle, P.voids_box(*dims, nvoids=1), n_levels=2, first_factor=2)
    n = o.spline_setup(order, parts)
    assert g.set_spline_partition(*parts, order) == n
    rng = np.random.default_rng(19)
    c = (amplitude * rng.normal(0.5, 0.15, n)).astype(np.float32)
    x = rng.standard_normal(o.ne).astype(np.float32)
    assert rel(g.coeff2density(c).cpu().numpy(), o.coeff2density(c.astype(np.float64))) < 1e-6
    assert rel(g.ddensity2dcoeff(x).cpu().numpy(), o.density2coeff_adjoint(x.astype(np.float64))) < 1e-6
    for mode in (4, 5):
        v, per, dc, cnt, ds = g.deal_background_points(c, 8.0, mode)
        vo, pero, dco, cnto, dso = o.selfsupport(c.astype(np.float64), 8.0, mode)
        assert cnt == cnto and ds == dso
        assert abs(v - vo) <= 1e-5 * max(abs(vo), 1e-12)
        assert rel(per.cpu().numpy(), pero) < 1e-5
        assert rel(dc.cpu().numpy(), dco) < 1e-4


@pytest.mark.parametrize("penal", [1.0, 2.0, 3.0, 3.5])
@pytest.mark.parametrize("dims", [(33, 9, 5), (30, 18, 12)])
def test_sensitivity_modes(oracle, cuda, dims, penal):
    """u^T K0 u summed in the sum/difference basis in FP64, rounded to FP32: 1e-6 relative."""
    from robustoptspline3d_b200 import Config, HierarchyGrid, element_matrix
    prob = P.voids_box(*dims)
    g = HierarchyGrid(prob["emask"], prob["fixed"], prob["load"], prob["normals"], Config(penal=penal, n_levels=2,
                                                                                          first_factor=2))
    rho = prob["rho"].astype(np.float32)
    g.set_density(rho.ravel())
    u = np.random.default_rng(4).standard_normal((3, dims[2] + 1, dims[1] + 1, dims[0] + 1))
    cls = g.node_class().reshape(u.shape[1:])
    u[:, (cls & 4 > 0) | (cls & 1 == 0)] = 0
    ue = np.stack([u[i, k >> 2:(k >> 2) + dims[2], (k >> 1 & 1):(k >> 1 & 1) + dims[1], (k & 1):(k & 1) + dims[0]]
                   for k in range(8) for i in range(3)]).reshape(24, -1)
    q = np.einsum("ie,ij,je->e", ue, element_matrix(), ue)
    r = rho.astype(np.float64).ravel() * prob["emask"].ravel()
    on = prob["emask"].ravel() > 0
    want = np.where(on, -penal * np.where(on, r, 1.0) ** (penal - 1) * q, 0.0)
    assert rel(g.computeSensitivity(t(u.ravel(), cuda)).cpu().numpy(), want) < 1e-6
    assert rel(g.elementCompliance(t(u.ravel(), cuda)).cpu().numpy(), np.where(on, r ** penal * q, 0.0)) < 1e-6


# one CTA (no grid barrier) with a part and exactly its 512 threads, one variable more, a ragged last
# CTA, and more variables than the GPU's threads; every number of constraints an update is built for
@pytest.mark.parametrize("n,m", [(1, 1), (512, 2), (513, 1), (5000, 3), (5000, 4), (5000, 5), (80001, 2)])
def test_mma_update_sizes(oracle, cuda, n, m):
    """Three updates against the oracle, 1e-8 relative and 1e-10 absolute as in the parity test."""
    from robustoptspline3d_b200 import MMA
    rng = np.random.default_rng(23)
    o, g = oracle.MMA(n, m, 0.0, 1.0), MMA(n, m, 0.0, 1.0)
    x0 = rng.uniform(0.2, 0.8, n)
    o.set_x(x0)
    g.set_x(x0)
    for k in range(3):
        x = o.get()[0]
        df = -np.exp(-x) * (1 + rng.uniform(0, 0.1, n))
        dg = np.stack([np.full(n, 1.0 / n)] + [rng.standard_normal(n) * 0.1 for _ in range(m - 1)])
        gval = np.array([x.mean() - 0.4] + [0.05 * np.sin(k + j) for j in range(m - 1)])
        o.update(df, dg, gval)
        g.update(t(df, cuda), t(dg, cuda), gval)
        for a, b in zip(g.get(), o.get()):
            assert np.allclose(a, b, rtol=1e-8, atol=1e-10)


# boxes whose edges are multiples of the coarsening factors and not, with voids and clamped faces, both
# first factors
@pytest.mark.parametrize("dims,levels,factor", [((12, 8, 8), 2, 4), ((21, 13, 9), 3, 2), ((33, 18, 22), 3, 4)])
def test_galerkin_operators(oracle, cuda, dims, levels, factor):
    """Products with the assembled stencils, 1e-12 relative, as the FP64 operator pieces."""
    g, o = make(oracle, P.voids_box(*dims, nvoids=1), n_levels=levels, first_factor=factor, smoother=1)
    g.update_stencil()
    o.update_stencil()
    rng = np.random.default_rng(29)
    for lvl in range(1, o.n_levels()):
        mask = np.tile(o.level_masks(lvl)[1], 3)
        u, f = (rng.standard_normal(mask.size) * mask for _ in range(2))
        assert rel(g.coarse_residual(lvl, t(u, cuda), t(f, cuda)).cpu().numpy(), o.coarse_residual(lvl, u, f)) < 1e-12


# coarsest systems of part of a 32-wide tile, of tiles and a remainder (N = 105, 417, 2175), and past
# the size up to which the inversion is the blocked Gauss-Jordan kernel (N = 4707)
@pytest.mark.parametrize("dims,levels,factor", [((12, 8, 8), 2, 4), ((21, 13, 9), 3, 2), ((16, 16, 16), 2, 2),
                                                ((24, 20, 20), 2, 2)])
def test_coarsest_inverse(cuda, dims, levels, factor):
    """K x = f on the coarsest level, residual 1e-9 relative, as the coarsest solve's parity test."""
    from robustoptspline3d_b200 import Config, HierarchyGrid
    prob = P.voids_box(*dims, nvoids=1)
    g = HierarchyGrid(prob["emask"], prob["fixed"], prob["load"], prob["normals"],
                      Config(n_levels=levels, first_factor=factor))
    g.set_density(prob["rho"].astype(np.float32).ravel())
    g.update_stencil()
    last = g.n_levels() - 1
    mask = np.tile(g.level_masks(last)[1], 3)
    f = np.random.default_rng(31).standard_normal(mask.size) * mask
    x = g.solve_coarsest(t(f, cuda))
    r = g.coarse_residual(last, x, t(f, cuda)).cpu().numpy()
    assert np.linalg.norm(r) < 1e-9 * np.linalg.norm(f)


@pytest.mark.parametrize("precision", [0, 1])
def test_batch_on_used_memory(cuda, precision):
    """The batch's slabs come from memory that held NaN before: its padding must not reach the solution."""
    from robustoptspline3d_b200 import Config, HierarchyGrid
    prob = P.cantilever(20, 12, 12)
    g = HierarchyGrid(prob["emask"], prob["fixed"], prob["load"], None,
                      Config(poisson_ratio=0.4, precision=precision, smoother=1, n_levels=3, first_factor=2))
    g.set_density(prob["rho"].astype(np.float32).ravel())
    g.update_stencil()
    used = [cuda.full((1 << 20,), float("nan"), dtype=cuda.float64, device="cuda") for _ in range(64)]
    cuda.cuda.synchronize()
    del used
    cuda.cuda.empty_cache()
    f = t(prob["f"], cuda)
    U, infos = g.solve_batch(cuda.stack([f, 2 * f]), tol=1e-10)
    u, it, _, _ = g.solve(f, tol=1e-10)
    assert rel(U[0].cpu().numpy(), u.cpu().numpy()) < 1e-8 and abs(infos[0][0] - it) <= 1


@pytest.mark.parametrize("gen,smoother", [(lambda: P.cantilever(48, 24, 24), 2), (lambda: P.ellipsoid(40, 24, 24), 1),
                                          (lambda: P.cantilever(33, 18, 20), 0)])
def test_fp64_vcycle_graphs_and_bottom(cuda, gen, smoother):
    """FP64 solves: replayed V-cycles bit-identical to plain launches; with the persistent bottom kernel
    (nine threads per node) and without, the same solution to 1e-8 and iterations within one."""
    from robustoptspline3d_b200 import Config, HierarchyGrid
    prob = gen()
    g = HierarchyGrid(prob["emask"], prob["fixed"], prob["load"], prob["normals"],
                      Config(precision=0, smoother=smoother, poisson_ratio=0.4, n_levels=3, first_factor=2, pre=2, post=2))
    g.set_density(prob["rho"].astype(np.float32).ravel())
    g.update_stencil()
    ln = g.load_nodes()
    f = np.zeros(3 * g.nn)
    f[2 * g.nn + ln] = np.random.default_rng(37).standard_normal(len(ln))
    g.set_vcycle_graphs(False)
    plain, it, _, _ = g.solve(t(f, cuda), tol=1e-9)
    g.set_vcycle_graphs(True)
    for _ in range(3):
        u, k, _, _ = g.solve(t(f, cuda), tol=1e-9)
        assert k == it and np.array_equal(u.cpu().numpy(), plain.cpu().numpy())
    g.set_launch_shapes(4, -1)
    u, k, _, _ = g.solve(t(f, cuda), tol=1e-9)
    assert abs(k - it) <= 1 and rel(u.cpu().numpy(), plain.cpu().numpy()) < 1e-8


# grids of 2, 4 and 8 voxels (several columns to a word or a warp), of one warp's words a column (128)
# and of more (256)
@pytest.mark.parametrize("pref", [1, 2, 6, 100, 130])
def test_voxel_columns(cuda, pref):
    """Solid voxels of every column layout of the parity scan; the same bytes."""
    from oracle import voxel
    from robustoptspline3d_b200.voxelize import voxelize
    v, f = M.icosphere(1, 5.0, rotation_seed=3)
    got, R, _ = voxelize(v, f, pref)
    want, Ro, _ = voxel.voxelize(v, f, pref)
    assert R == Ro and np.array_equal(got, want), int(np.sum(got != want))


# boxes of more rows than a warp takes (the cube), rows that are no multiple of eight bytes, and slivers
# whose closest points are too inexact for the bounding-box test (the flattened sphere)
@pytest.mark.parametrize("shape,R,width,flat", [("cube", 71, 3.5, 1.0), ("icosphere", 37, 2.2, 1.0),
                                                ("icosphere", 24, 1.3, 1e-7), ("icosphere", 8, 9.0, 1.0)])
def test_shell_rows(cuda, shape, R, width, flat):
    """Shell elements for any non-zero solid byte; the same bytes."""
    from oracle import boundary as OB
    from robustoptspline3d_b200 import boundary as B
    v, f = M.cube(4.0) if shape == "cube" else M.icosphere(2, 4.0, rotation_seed=2)
    v = (np.asarray(v, np.float64) * [1.0, 1.0, flat]).astype(np.float32)
    lo, size = v.min(0), 1.1 * float(np.ptp(v, axis=0).max())
    lo = (0.5 * (v.min(0) + v.max(0)) - 0.5 * size).astype(np.float32)
    box = np.concatenate([lo, lo + np.float32(size)]).astype(np.float32)
    solid = np.random.default_rng(1).choice(np.array([0, 1, 2, 255], np.uint8), size=(R, R, R))
    got = B.shell_elements(v, f, box, R, width, solid)
    want = OB.shell_elements(v, f, box, R, width, (solid > 0).astype(np.uint8))
    assert np.array_equal(got, want), int(np.sum(got != want))
    assert got.sum() > 0


@pytest.mark.parametrize("flat", [1.0, 0.0])
def test_normals_rings(cuda, flat):
    """Normals at points in the mesh's box, far outside it (many rings) and on vertices (ties), of a
    sphere and of a flat disc; 1e-12, the bound of the normals test."""
    from oracle import boundary as OB
    from robustoptspline3d_b200 import boundary as B
    v, f = M.icosphere(3, 1.0, rotation_seed=5)
    v = (np.asarray(v, np.float64) * [1.0, 1.0, flat]).astype(np.float32)
    rng = np.random.default_rng(8)
    P = np.concatenate([rng.uniform(-1.2, 1.2, (301, 3)), rng.uniform(-40, 40, (70, 3)), v[:33].astype(np.float64)])
    if flat == 0.0:
        P = P[:371]  # both layers of the disc tie at a vertex and have opposite planes
    got, want = B.mesh_normals(v, f, P), OB.mesh_normals(v, f, P)
    assert np.max(np.abs(got - want)) <= 1e-12


@pytest.mark.parametrize("dims", [(1, 5, 3), (31, 3, 2), (33, 7, 5), (257, 2, 3)])
def test_region_rows(cuda, dims):
    """Region masks on rows shorter than, equal to and longer than a warp; the same bytes."""
    from robustoptspline3d_b200 import boundary as B
    r = [B.sphere((0.4, 0.3, 0.2), 0.9), B.halfspace(1, 0.5, -1, -9.0)]
    got = B.region_mask(r, (-0.5, -0.4, -0.3), 0.2, dims)
    z, y, x = np.meshgrid(*(np.arange(n) for n in dims[::-1]), indexing="ij")
    x, y, z = -0.5 + x * 0.2, -0.4 + y * 0.2, -0.3 + z * 0.2
    want = ((x - 0.4) ** 2 + (y - 0.3) ** 2 + (z - 0.2) ** 2 < 0.9 ** 2) | (x + 0.5 * y - z - 9.0 > 0)
    assert np.array_equal(got, want.astype(np.uint8))


@pytest.mark.parametrize("sweeps", [1, 2, 3, 4])
def test_chebyshev_sweeps(oracle, cuda, sweeps):
    """FP64 Chebyshev smoothing of a single level (two sweeps take the factored form, others the
    recurrence) against the recurrence on the oracle's operator; 1e-11 relative, ten times the bound of
    the operator pieces for up to four of them in a row."""
    g, o = make(oracle, P.cantilever(9, 6, 5), n_levels=1, smoother=2)
    g.update_stencil()
    rng = np.random.default_rng(21)
    cls = o.node_class()
    fix = np.tile(((cls & 4) > 0) | ((cls & 1) == 0), 3)
    u, f = (np.where(fix, 0.0, rng.standard_normal(3 * o.nn)) for _ in range(2))
    got, _ = g.v_cycle(t(u, cuda), t(f, cuda), pre=sweeps, post=0)
    lam, lower = g.level_lambda(0), 0.25
    theta, delta = 0.5 * lam * (1 + lower), 0.5 * lam * (1 - lower)
    rho, step = delta / theta, 0.0
    for k in range(sweeps):
        d = o.smooth(0, u, f, kind=1, omega=1.0, sweeps=1) - u  # D^-1 (f - K u)
        if k == 0:
            step = d / theta
        else:
            new = 1.0 / (2.0 * theta / delta - rho)
            step = new * rho * step + 2.0 * new / delta * d
            rho = new
        u = u + step
    assert rel(got.cpu().numpy(), u) < 1e-11


# boxes whose planes, rows and groups of four do not divide by the coarsening, one to three coarse columns wide
@pytest.mark.parametrize("dims,factor", [((7, 5, 3), 2), ((13, 9, 6), 4), ((21, 10, 7), 2), ((33, 18, 11), 4)])
def test_prolongation_and_first_step_fp32(oracle, cuda, dims, factor):
    """FP32 prolongation and the fine level's step from zero; 2e-5 relative, the bound of the FP32 pieces."""
    g, o = make(oracle, P.cantilever(*dims), n_levels=2, first_factor=factor)
    g.update_stencil()
    rng = np.random.default_rng(13)
    cls = o.node_class()
    fix = np.tile(((cls & 4) > 0) | ((cls & 1) == 0), 3)
    _, vm = o.level_masks(1)
    uc = rng.standard_normal(3 * vm.size) * np.tile(vm, 3)
    uf = np.where(fix, 0.0, rng.standard_normal(3 * o.nn))
    want = np.where(fix, 0.0, o.prolong(1, uc, uf))
    assert rel(g.prolong_fp32(1, t(uc, cuda), t(uf, cuda)).cpu().numpy(), want) < 2e-5
    z = np.zeros(3 * o.nn)
    got = g.fine_sweep_fp32(3, t(z, cuda), t(uf, cuda), omega=0.3).cpu().numpy()
    assert rel(got, o.smooth(0, z, uf, kind=1, omega=0.3, sweeps=1)) < 2e-5


@pytest.mark.parametrize("threads", [1, 3])
@pytest.mark.parametrize("dims", [(160, 162, 161), (160, 163, 162), (256, 256, 257)])
def test_large_masks_to_host(cuda, dims, threads):
    """Results of 4 MB (just under and over the size that takes the pinned ring) and 17 MB (each slot of it
    refilled) in ordinary memory, from one caller and from several at once; the same bytes."""
    from concurrent.futures import ThreadPoolExecutor
    from robustoptspline3d_b200 import boundary as B
    z, y, x = np.meshgrid(*(np.arange(n) for n in dims[::-1]), indexing="ij", sparse=True)
    want = ((x * 0.5 + y * 0.25 - z * 0.125 - 20.0) > 0).astype(np.uint8)
    with ThreadPoolExecutor(threads) as pool:
        got = list(pool.map(lambda _: B.region_mask([B.halfspace(0.5, 0.25, -0.125, -20.0)], (0, 0, 0), 1.0, dims),
                            range(2 * threads)))
    assert all(np.array_equal(m, want) for m in got)


@pytest.mark.parametrize("order", [2, 3, 4, 5])
def test_probe_past_the_integers(oracle, cuda, order):
    """Probes and surface points at coordinates past the integers lie outside the knots: probe sums and
    counts equal to the oracle's for finite coefficients, and no error, with the same results
    afterwards, for infinite ones and points."""
    g, o = make(oracle, P.voids_box(12, 10, 8, nvoids=1), n_levels=2, first_factor=2)
    n = o.spline_setup(order, (3, 2, 4))
    assert g.set_spline_partition(3, 2, 4, order) == n
    c = np.random.default_rng(41).normal(0.5, 0.15, n).astype(np.float32)
    big = (np.float32(1e15) * (c - np.float32(0.5))).astype(np.float32)
    _, _, _, cnt, ds = g.deal_background_points(big, 8.0, 4)
    _, _, _, cnto, dso = o.selfsupport(big.astype(np.float64), 8.0, 4)
    assert cnt == cnto and ds == dso
    before = g.deal_background_points(c, 8.0, 4)
    inf = c.copy()
    inf[n // 2] = np.inf
    inf[n // 3] = -np.inf
    g.deal_background_points(inf, 8.0, 4)
    after = g.deal_background_points(c, 8.0, 4)
    assert all(cuda.equal(a, b) if isinstance(a, cuda.Tensor) else a == b for a, b in zip(before, after))
    pts = np.random.default_rng(43).uniform(1, 7, (3, 40)).astype(np.float32)
    g.uploadSurfacePoints(pts)
    want = g.deal_surface_points(c, 8.0, 5)[1]
    g.uploadSurfacePoints(np.concatenate([pts, np.array([[1e12, 3e38, np.inf], [2, -np.inf, 3], [3, 2, 1e12]], np.float32)], 1))
    assert cuda.equal(g.deal_surface_points(c, 8.0, 5)[1][:40], want)


@pytest.mark.parametrize("precision", [0, 1])
def test_barrier_that_gave_up_is_reported(cuda, precision):
    """Every entry point that runs the persistent kernels reports a grid-barrier wait that gave up, once,
    and computes the same as before on its next call."""
    from robustoptspline3d_b200 import Config, HierarchyGrid
    from robustoptspline3d_b200.rso import RSOError
    prob = P.cantilever(32, 16, 16)
    g = HierarchyGrid(prob["emask"], prob["fixed"], prob["load"], None,
                      Config(poisson_ratio=0.4, precision=precision, n_levels=3, first_factor=2))
    g.set_density(prob["rho"].astype(np.float32).ravel())
    g.update_stencil()
    f = t(prob["f"], cuda)
    z = cuda.zeros_like(f)
    calls = [lambda: g.v_cycle(z, f, 2, 2)[0], lambda: g.solve(f, tol=1e-8)[0],
             lambda: g.solve(f, tol=1e-3, max_iter=100, method=0)[0],
             lambda: g.solve_batch(cuda.stack([f, 2 * f]), tol=1e-8)[0], lambda: g.modifiedPM(0, max_itn=5)[2],
             lambda: (g.update_stencil(), g.stencil(1))[1]]
    for i, call in enumerate(calls):
        call()  # past the first capture of a V-cycle
        want = call()
        g.grid_barrier_give_up()
        with pytest.raises(RSOError, match="grid-barrier"):
            call()
        assert cuda.equal(call(), want), i


@pytest.mark.parametrize("precision,smoother", [(0, 0), (0, 1), (0, 2), (1, 0), (1, 1), (1, 2)])
def test_graphs_are_launched(cuda, precision, smoother):
    """V-cycles are replayed from graphs, all but the first few of a second solve, and a mixed solve under
    device control launches its own graph: none of them has fallen back to plain launches."""
    from robustoptspline3d_b200 import Config, HierarchyGrid
    prob = P.cantilever(48, 24, 24)
    g = HierarchyGrid(prob["emask"], prob["fixed"], prob["load"], None,
                      Config(precision=precision, smoother=smoother, poisson_ratio=0.4, n_levels=3, first_factor=2))
    g.set_density(prob["rho"].astype(np.float32).ravel())
    g.update_stencil()
    f = t(prob["f"], cuda)
    want, it, _, _ = g.solve(f, tol=1e-9)
    v0, _ = g.graph_launches()
    u, k, _, _ = g.solve(f, tol=1e-9)
    v1, s1 = g.graph_launches()
    assert k == it and cuda.equal(u, want)
    assert v1 - v0 >= it - 4 and s1 == 0
    g.set_vcycle_graphs(False)
    g.solve(f, tol=1e-9)
    assert g.graph_launches() == (v1, 0)
    if precision == 1:
        g.set_vcycle_graphs(True)
        g.set_solve_graphs(True)
        u, k, _, _ = g.solve(f, tol=1e-9)
        assert g.graph_launches()[1] > 0 and k == it and cuda.equal(u, want)


@pytest.mark.parametrize("smoother", [0, 1, 2])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("levels", [12, 13, 14, 15])
def test_more_levels_than_elements(cuda, levels, precision, smoother):
    """A level count past the last element is accepted, as any other: the solution of two levels to 1e-6
    relative (both solved to 1e-9), and a step size for every level."""
    from robustoptspline3d_b200 import Config, HierarchyGrid
    prob = P.cantilever(12, 8, 8)
    u = []
    for nl in (2, levels):
        g = HierarchyGrid(prob["emask"], prob["fixed"], prob["load"], None,
                          Config(precision=precision, smoother=smoother, n_levels=nl, first_factor=2))
        g.set_density(prob["rho"].astype(np.float32).ravel())
        g.update_stencil()
        assert g.n_levels() == nl
        u.append(g.solve(t(prob["f"], cuda), tol=1e-9, max_iter=400)[0].cpu().numpy())
        if smoother != 0:
            assert all(0 < g.level_lambda(i) < 10 for i in range(nl - 1))
    assert rel(u[1], u[0]) < 1e-6


@pytest.mark.parametrize("beta", [1e-310, 1e-14, 1e-9, 9.9e-4, 1e-3, 0.1, 8.0, 300.0, 1e5, -1e-12, -2.0])
def test_heaviside_slopes(cuda, beta):
    """The step and its slope against tanh in FP64, from nearly linear (where differences of exponentials
    cancel) to a jump; one FP32 rounding, 1e-7 relative to one."""
    from robustoptspline3d_b200 import Config, HierarchyGrid
    prob = P.voids_box(21, 13, 11, nvoids=1)
    g = HierarchyGrid(prob["emask"], prob["fixed"], prob["load"], prob["normals"],
                      Config(n_levels=2, first_factor=2, rho_min=1e-3))
    rng = np.random.default_rng(47)
    x, gin = rng.uniform(0, 1, g.ne).astype(np.float32), rng.standard_normal(g.ne).astype(np.float32)
    x[:9] = [0, 1, 0.5, 0.5 + 2.0 ** -24, 0.5 - 2.0 ** -25, 0.25, 0.75, 2, -1]
    on = prob["emask"].ravel() > 0
    s, th = beta * (x.astype(np.float64) - 0.5), np.tanh
    den = 2 * th(beta * 0.5)
    want = np.where(on, np.clip((th(beta * 0.5) + th(s)) / den, 1e-3, 1.0), 0.0)
    assert np.max(np.abs(g.projectDensities(x, beta).cpu().numpy() - want)) < 1e-7
    slope = np.where(on, gin * (beta / den) / np.cosh(np.minimum(np.abs(s), 300.0)) ** 2, 0.0)
    got = g.projectSensitivity(x, beta, gin).cpu().numpy()
    assert np.max(np.abs(got - slope)) < 1e-7 * max(1.0, np.max(np.abs(slope)))


# the kernel of few faces: one face, more faces than CTAs, boxes of a row and of the whole grid, several
# teams to a face; that of many: faces in the list (all of 48 rows), boxes clipped at the grid's edge
@pytest.mark.parametrize("subdiv,R,width,keep", [(0, 40, 30.0, 1.0), (3, 33, 1.1, 1.0), (3, 20, 4.0, 1.0),
                                                 (4, 17, 0.4, 1.0), (4, 30, 2.5, 0.5), (4, 49, 60.0, 0.002)])
@pytest.mark.parametrize("nfaces", [1, None])
def test_shell_faces(cuda, subdiv, R, width, keep, nfaces):
    """Shell elements of meshes of one to 5120 faces; the same bytes."""
    from oracle import boundary as OB
    from robustoptspline3d_b200 import boundary as B
    v, f = M.icosphere(subdiv, 4.0, rotation_seed=6)
    f = f[:nfaces]
    box = np.array([-4.2, -4.3, -4.4, 4.4, 4.3, 4.2], np.float32)
    solid = (np.random.default_rng(3).random((R, R, R)) < keep).astype(np.uint8) * 7
    got = B.shell_elements(v, f, box, R, width, solid)
    want = OB.shell_elements(v, f, box, R, width, (solid > 0).astype(np.uint8))
    assert np.array_equal(got, want), int(np.sum(got != want))


def test_shell_of_many_wide_faces(cuda):
    """Every face of 5120 in the list of large boxes: as the union of the shells of parts of few faces."""
    from robustoptspline3d_b200 import boundary as B
    v, f = M.icosphere(4, 4.0, rotation_seed=6)
    box = np.array([-4.2, -4.3, -4.4, 4.4, 4.3, 4.2], np.float32)
    solid = np.ones((64, 64, 64), np.uint8)
    got = B.shell_elements(v, f, box, 64, 19.0, solid)
    want = np.max([B.shell_elements(v, part, box, 64, 19.0, solid) for part in np.array_split(f, 2)], axis=0)
    assert np.array_equal(got, want) and 0 < got.sum() < got.size


@pytest.mark.parametrize("dims,n", [((18, 16, 16), 2430), ((18, 18, 16), 2700)])
def test_coarsest_inverse_line(cuda, dims, n):
    """The largest coarsest systems below and the next above the line between the two inversions: residual
    1e-9 relative, as the coarsest solve's parity test."""
    from robustoptspline3d_b200 import Config, HierarchyGrid
    prob = P.cantilever(*dims)
    g = HierarchyGrid(prob["emask"], prob["fixed"], prob["load"], None, Config(n_levels=2, first_factor=2))
    g.set_density(prob["rho"].astype(np.float32).ravel())
    g.update_stencil()
    mask = np.tile(g.level_masks(1)[1], 3)
    assert int(mask.sum()) == n
    f = np.random.default_rng(53).standard_normal(mask.size) * mask
    x = g.solve_coarsest(t(f, cuda))
    assert np.linalg.norm(g.coarse_residual(1, x, t(f, cuda)).cpu().numpy()) < 1e-9 * np.linalg.norm(f)


@pytest.mark.parametrize("dims", [(203, 203, 203), (203, 204, 203)])
def test_masks_at_the_ring_line(cuda, dims):
    """Results just under and over the 8 MB from which they go through the pinned ring; the same bytes."""
    from robustoptspline3d_b200 import boundary as B
    z, y, x = np.meshgrid(*(np.arange(n) for n in dims[::-1]), indexing="ij", sparse=True)
    want = ((x * 0.5 - y * 0.25 + z * 0.125 - 30.0) > 0).astype(np.uint8)
    assert np.array_equal(B.region_mask([B.halfspace(0.5, -0.25, 0.125, -30.0)], (0, 0, 0), 1.0, dims), want)


@pytest.mark.parametrize("nx", [1, 2, 3, 4, 5, 8, 9, 16, 17, 32])
def test_region_short_rows(cuda, nx):
    """Region masks with 1 to 32 lanes a row, whole and ragged; the same bytes."""
    from robustoptspline3d_b200 import boundary as B
    dims = (nx, 37, 53)
    got = B.region_mask([B.sphere((0.4, 0.3, 0.2), 0.9), B.halfspace(1, 0.5, -1, -1.0)], (-0.5, -0.4, -0.3), 0.1, dims)
    z, y, x = np.meshgrid(*(np.arange(n) for n in dims[::-1]), indexing="ij")
    x, y, z = -0.5 + x * 0.1, -0.4 + y * 0.1, -0.3 + z * 0.1
    want = ((x - 0.4) ** 2 + (y - 0.3) ** 2 + (z - 0.2) ** 2 < 0.9 ** 2) | (x + 0.5 * y - z - 1.0 > 0)
    assert np.array_equal(got, want.astype(np.uint8)) and 0 < got.sum() < got.size


def test_spline_set_up_allocates_for_the_constraint(cuda):
    """The first overhang call after a spline set-up allocates no device memory: what it needs is there."""
    from robustoptspline3d_b200 import Config, HierarchyGrid
    prob = P.cantilever(96, 96, 96)
    g = HierarchyGrid(prob["emask"], prob["fixed"], prob["load"], None, Config())
    n = g.set_spline_partition(28, 28, 28, 4)  # rows of 3 x 32 x 96 x 96 doubles: 7 MB
    c = t(np.random.default_rng(59).normal(0.5, 0.15, n).astype(np.float32), cuda)
    per, dc = cuda.empty(g.ne, device="cuda"), cuda.empty(n, device="cuda")
    cuda.cuda.synchronize()
    free, _ = cuda.cuda.mem_get_info()
    assert g.lib.rso_selfsupport(g.h, c.data_ptr(), 8.0, 4, 2.36, 2.36, per.data_ptr(), dc.data_ptr(), None, None,
                                 None) == 0
    assert cuda.cuda.mem_get_info()[0] == free


def test_reported_errors_are_not_left_over(cuda):
    """A call that failed for lack of memory leaves no error for the next launch, ours or the caller's."""
    from robustoptspline3d_b200 import Config, HierarchyGrid
    from robustoptspline3d_b200.rso import RSOError
    prob = P.cantilever(12, 10, 8)
    g = HierarchyGrid(prob["emask"], prob["fixed"], prob["load"], None, Config(n_levels=2, first_factor=2))
    with pytest.raises(RSOError):
        g.set_spline_partition(100000, 100000, 100000, 4)
    assert float((cuda.ones(4, device="cuda") + 1).sum()) == 8.0
    g.update_stencil()


def test_spline_set_up_that_failed(cuda):
    """A set-up whose coefficients do not fit the device fails, and the maps are refused until one succeeds,
    with the results of before."""
    from robustoptspline3d_b200 import Config, HierarchyGrid
    from robustoptspline3d_b200.rso import RSOError
    prob = P.cantilever(12, 10, 8)
    g = HierarchyGrid(prob["emask"], prob["fixed"], prob["load"], None, Config(n_levels=2, first_factor=2))
    n = g.set_spline_partition(3, 2, 4, 4)
    c = np.random.default_rng(61).normal(0.5, 0.15, n).astype(np.float32)
    want = g.coeff2density(c)
    with pytest.raises(RSOError):
        g.set_spline_partition(100000, 100000, 100000, 4)
    for call in (lambda: g.coeff2density(c), lambda: g.ddensity2dcoeff(want), lambda: g.deal_background_points(c, 8.0),
                 lambda: g.updateCoeff(c, -c, 0.3)):
        with pytest.raises(RSOError):
            call()
    assert g.set_spline_partition(3, 2, 4, 4) == n
    assert cuda.equal(g.coeff2density(c), want)


def test_design_iteration_after_a_finer_spline(cuda):
    """A design iteration on a spline set up anew with more coefficients: as on a handle that only ever had
    that spline."""
    from robustoptspline3d_b200 import MMA, Config, HierarchyGrid, IterParams
    prob = P.top_loaded_cube(12)
    out = []
    for first in (True, False):
        g = HierarchyGrid(prob["emask"], prob["fixed"], prob["load"], None, Config(n_levels=2, first_factor=2, smoother=1))
        for parts in ((1, 1, 1), (9, 8, 7)) if first else ((9, 8, 7),):
            n = g.set_spline_partition(*parts, 4)
            m = MMA(n, 2, 0.0, 1.0)
            m.set_x(np.random.default_rng(67).uniform(0.3, 0.7, n))
            g.design_iteration(m, IterParams(lanczos_steps=4, filter_radius=1.5))
        out.append(m.get())
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("parts", [(9, 8, 7), (40, 30, 30)])
def test_oc_with_more_coefficients_than_elements(oracle, cuda, parts):
    """The OC coefficient update on a box of 12 x 10 x 8 elements with fewer and with far more coefficients,
    against the oracle's at the bounds of its parity test."""
    from oracle import oc
    g, o = make(oracle, P.cantilever(12, 10, 8), n_levels=2, first_factor=2)
    n = o.spline_setup(4, parts)
    assert g.set_spline_partition(*parts, 4) == n
    rng = np.random.default_rng(71)
    c, s = rng.uniform(0.4, 0.6, n).astype(np.float32), -rng.uniform(0.5, 1.5, n).astype(np.float32)
    new, rho, info = g.updateCoeff(c, s, 0.5, step=0.1, damp=0.5, cmin=0.0, cmax=1.0)
    co, ro, go, vo, to = oc.update_coeff(o, c, s, 0.5, 0.1, 0.5, 0.0, 1.0)
    assert info["trials"] == to and abs(info["g"] - go) <= 1e-5 * go and abs(info["volume"] - vo) <= 1e-5
    assert np.max(np.abs(new.cpu().numpy() - co)) <= 1e-5
    assert np.max(np.abs(rho.cpu().numpy() - ro)) <= 1e-5


@pytest.mark.parametrize("precision", [0, 1])
def test_design_iteration_is_reproducible(cuda, precision):
    """The design iteration's update reads its gradients on another stream than they were written on: forty
    iterations from the same coefficients end in the same bits, those of the gradients passed by hand."""
    from robustoptspline3d_b200 import MMA, Config, HierarchyGrid, IterParams
    prob = P.top_loaded_cube(12)
    p = IterParams(lanczos_steps=4, filter_radius=1.5)
    g = HierarchyGrid(prob["emask"], prob["fixed"], prob["load"], None,
                      Config(n_levels=2, first_factor=2, smoother=2, precision=precision))
    n = g.set_spline_partition(9, 8, 7, 4)
    x = np.random.default_rng(67).uniform(0.3, 0.7, n)
    v, gl, gv, gs = g.design_gradient(t(x, cuda), p)
    ref = MMA(n, 2, 0.0, 1.0)
    ref.set_x(x)
    ref.update(p.sens_scale * gl, cuda.stack([p.vol_scale * gv, p.ss_scale * gs]),
               np.array([p.vol_scale * (v["volume"] - p.volume_ratio), p.ss_scale * v["ss"]]))
    for _ in range(40):
        m = MMA(n, 2, 0.0, 1.0)
        m.set_x(x)
        g.design_iteration(m, p)
        assert all(np.array_equal(a, b) for a, b in zip(m.get(), ref.get()))
        m.close()
    ref.close()
    g.close()


def test_host_iteration_of_another_size(cuda):
    """The host form of the design iteration refuses an MMA of another size before it copies anything."""
    from robustoptspline3d_b200 import MMA, Config, HierarchyGrid, IterParams
    from robustoptspline3d_b200.rso import RSOError
    prob = P.top_loaded_cube(12)
    g = HierarchyGrid(prob["emask"], prob["fixed"], prob["load"], None, Config(n_levels=2, first_factor=2))
    m = MMA(9, 2, 0.0, 1.0)
    x0 = m.get()[0]
    with pytest.raises(RSOError, match="not set up"):
        g.design_iteration_host(m, np.ones(9), IterParams())
    n = g.set_spline_partition(9, 8, 7, 4)
    with pytest.raises(RSOError, match="size differs"):
        g.design_iteration_host(m, np.ones(n), IterParams())
    assert np.array_equal(m.get()[0], x0)


# few rows, cut in chunks of 32 to 128 elements with a ragged last one: supports inside a chunk, over
# several, over all; and rows just too many for it
@pytest.mark.parametrize("dims,order,parts", [((1000, 4, 3), 4, (200, 2, 1)), ((333, 5, 4), 3, (2, 0, 1)),
                                              ((65, 8, 9), 5, (12, 3, 3)), ((129, 25, 24), 4, (9, 4, 5)),
                                              ((97, 40, 30), 2, (40, 3, 3)), ((33, 2, 2), 4, (0, 0, 0))])
@pytest.mark.parametrize("amplitude", [1.0, 3000.0])
def test_spline_rows_in_chunks(oracle, cuda, dims, order, parts, amplitude):
    """Adjoint 1e-6, constraint value 1e-5 and gradient 1e-4 relative, counts and probe sums equal: the
    bounds of these maps in the parity tests."""
    g, o = make(oracle, P.cantilever(*dims), n_levels=4, first_factor=2)
    n = o.spline_setup(order, parts)
    assert g.set_spline_partition(*parts, order) == n
    rng = np.random.default_rng(73)
    c = (amplitude * rng.normal(0.5, 0.15, n)).astype(np.float32)
    x = rng.standard_normal(o.ne).astype(np.float32)
    assert rel(g.ddensity2dcoeff(x).cpu().numpy(), o.density2coeff_adjoint(x.astype(np.float64))) < 1e-6
    for mode in (4, 5):
        v, per, dc, cnt, ds = g.deal_background_points(c, 8.0, mode)
        vo, pero, dco, cnto, dso = o.selfsupport(c.astype(np.float64), 8.0, mode)
        assert cnt == cnto and ds == dso and abs(v - vo) <= 1e-5 * max(abs(vo), 1e-12)
        assert rel(per.cpu().numpy(), pero) < 1e-5
        assert rel(dc.cpu().numpy(), dco) < 1e-4


@pytest.mark.parametrize("dims,order,parts,seed", [((40, 24, 20), 3, (3, 5, 2), 0), ((33, 9, 70), 4, (3, 5, 2), 1),
                                                   ((33, 9, 70), 5, (3, 5, 2), 0), ((12, 10, 8), 4, (30, 1, 12), 2)])
def test_overhang_with_a_positive_probe_sum(oracle, cuda, dims, order, parts, seed):
    """Coefficients so large that most probes land beyond the box or on the other side: the sum of the probes
    is not negative and the pass runs again; the bounds of the constraint's parity test."""
    g, o = make(oracle, P.cantilever(*dims), n_levels=2, first_factor=2)
    n = o.spline_setup(order, parts)
    assert g.set_spline_partition(*parts, order) == n
    positive = 0
    for k in range(4):
        c = (3e5 * np.random.default_rng(seed + 10 * k).normal(0.5, 0.15, n)).astype(np.float32)
        for mode in (0, 2, 4, 5):
            v, per, dc, cnt, ds = g.deal_background_points(c, 8.0, mode)
            vo, pero, dco, cnto, dso = o.selfsupport(c.astype(np.float64), 8.0, mode)
            assert cnt == cnto and ds == dso
            assert abs(v - vo) <= 1e-5 * max(abs(vo), 1e-12)
            assert rel(per.cpu().numpy(), pero) < 1e-5 and rel(dc.cpu().numpy(), dco) < 1e-4
        positive += ds >= 0
    assert positive > 0


@pytest.mark.parametrize("dims", [(1, 9, 40), (2, 33, 30), (5, 8, 50), (8, 8, 40), (9, 40, 9), (16, 5, 20), (17, 9, 9)])
@pytest.mark.parametrize("radius", [0.6, 6.2])
def test_general_filter_on_narrow_boxes(oracle, cuda, dims, radius):
    """FP64 sums rounded to FP32 once: 1e-6 relative, on tiles of every width."""
    g, o = make(oracle, P.cantilever(*dims), n_levels=2, first_factor=2)
    x = np.random.default_rng(83).standard_normal(o.ne).astype(np.float32)
    assert rel(g.filterSensitivity(radius, x).cpu().numpy(), o.filter(radius, x.astype(np.float64))) < 1e-6
    assert rel(g.densityFilter(radius, x, adjoint=True).cpu().numpy(),
               o.density_filter_adjoint(radius, x.astype(np.float64))) < 1e-6


def test_mesh_memory_is_given_back(cuda):
    """The mesh input's cached blocks and pinned ring go back on request, also while other threads call, and
    calls after it give the same bytes."""
    from concurrent.futures import ThreadPoolExecutor
    from robustoptspline3d_b200 import boundary as B
    from robustoptspline3d_b200.voxelize import voxelize
    v, f = M.icosphere(3, 4.0)

    def run(_=None):
        solid, R, box = voxelize(v, f, 140)
        return solid, B.shell_elements(v, f, box, R, 2.0, solid)

    B.release_memory()
    cuda.cuda.synchronize()
    free = cuda.cuda.mem_get_info()[0]
    want = run()
    assert cuda.cuda.mem_get_info()[0] < free
    B.release_memory()
    assert cuda.cuda.mem_get_info()[0] >= free
    with ThreadPoolExecutor(4) as pool:
        jobs = [pool.submit(run) if k % 3 else pool.submit(B.release_memory) for k in range(12)]
        got = [j.result() for j in jobs]
    for g in got:
        assert g is None or all(np.array_equal(a, b) for a, b in zip(g, want))


@pytest.mark.parametrize("shift", [-700, -1, 0, 1, 700])
def test_maps_on_overlapping_arrays(cuda, shift):
    """Outputs that overlap an input by all, most or a part of it, and the shell mask inside the output: the
    bits of the calls on separate arrays."""
    from robustoptspline3d_b200 import Config, HierarchyGrid
    prob = P.voids_box(21, 13, 11, nvoids=1)
    g = HierarchyGrid(prob["emask"], prob["fixed"], prob["load"], prob["normals"], Config(n_levels=2, first_factor=2))
    n = g.set_spline_partition(3, 2, 4, 4)
    rng = np.random.default_rng(89)
    x, y = rng.uniform(0, 1, g.ne).astype(np.float32), rng.standard_normal(g.ne).astype(np.float32)
    c = rng.normal(0.5, 0.15, n).astype(np.float32)
    sh = (rng.random(g.ne) < 0.2).astype(np.uint8)
    buf = cuda.empty(g.ne + 2000, device="cuda")
    at = lambda k, size=None: buf[1000 + k:1000 + k + (size or g.ne)]  # noqa: E731
    L, H = g.lib, g.h

    def overlapping(call):
        at(0).copy_(t(x, cuda))
        assert call(at(0).data_ptr(), at(shift).data_ptr()) == 0
        return at(shift).clone()

    other = t(y, cuda)
    assert cuda.equal(overlapping(lambda i, o: L.rso_heaviside(H, i, 8.0, None, o)), g.projectDensities(x, 8.0))
    assert cuda.equal(overlapping(lambda i, o: L.rso_heaviside_chain(H, i, 8.0, other.data_ptr(), o)),
                      g.projectSensitivity(x, 8.0, y))
    assert cuda.equal(overlapping(lambda i, o: L.rso_heaviside_chain(H, other.data_ptr(), 8.0, i, o)),
                      g.projectSensitivity(y, 8.0, x))
    for r in (0.7, 2.0, 5.5):
        assert cuda.equal(overlapping(lambda i, o: L.rso_filter(H, r, i, o)), g.filterSensitivity(r, x))
        assert cuda.equal(overlapping(lambda i, o: L.rso_density_filter_adjoint(H, r, i, o)),
                          g.densityFilter(r, x, adjoint=True))
    xin, cin, mask = t(x, cuda), t(c, cuda), t(sh, cuda)
    for call, want in ((lambda m, o: L.rso_heaviside(H, xin.data_ptr(), 8.0, m, o), g.projectDensities(x, 8.0, sh)),
                       (lambda m, o: L.rso_coeff2density(H, cin.data_ptr(), m, o), g.coeff2density(c, sh))):
        at(shift // 4, g.ne).view(cuda.uint8)[:g.ne].copy_(mask)
        assert call(at(shift // 4).data_ptr(), at(0).data_ptr()) == 0
        assert cuda.equal(at(0), want)
    at(0, n).copy_(cin)
    assert L.rso_coeff2density(H, at(0).data_ptr(), None, at(shift // 4).data_ptr()) == 0
    assert cuda.equal(at(shift // 4), g.coeff2density(c))


@pytest.mark.parametrize("radius", [0.7, 1.0, 2.0, 3.7, 4.4, 5.3])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, -3.4028234e38, 3.4028234e38])
def test_filter_and_sums_on_extreme_values(cuda, radius, value):
    """One extreme value, on an active or on an inactive element, against FP64 sums over the taps: it reaches
    the elements within the radius and no other, and none from where the mask is off; 1e-6 relative."""
    from robustoptspline3d_b200 import Config, HierarchyGrid
    ex, ey, ez = 37, 11, 13
    prob = P.voids_box(ex, ey, ez, nvoids=2)
    em = prob["emask"].astype(bool)
    em[6, 5, 30] = True
    em[6, 5, 7] = False
    prob["emask"] = em.astype(np.uint8)
    g = HierarchyGrid(prob["emask"], prob["fixed"], prob["load"], prob["normals"], Config(n_levels=2, first_factor=2))
    x = np.random.default_rng(97).standard_normal(em.shape).astype(np.float32)
    x[6, 5, 30] = value   # active
    x[6, 5, 7] = value    # inactive
    R = int(radius + 0.5)
    num, den = np.zeros(em.shape), np.zeros(em.shape)
    with np.errstate(invalid="ignore", over="ignore"):
        xv = np.where(em, x.astype(np.float64), 0.0)
        for dz in range(-R, R + 1):
            for dy in range(-R, R + 1):
                for dx in range(-R, R + 1):
                    d2 = dx * dx + dy * dy + dz * dz
                    if d2 > radius * radius:
                        continue
                    r = np.sqrt(d2) / radius
                    w = 1 - 6 * r ** 2 + 8 * r ** 3 - 3 * r ** 4
                    src = tuple(slice(max(d, 0), n + min(d, 0)) for d, n in zip((dz, dy, dx), em.shape))
                    dst = tuple(slice(max(-d, 0), n + min(-d, 0)) for d, n in zip((dz, dy, dx), em.shape))
                    num[dst] += np.where(em[src], w * xv[src], 0.0)
                    den[dst] += np.where(em[src], w, 0.0)
        want = np.where(em, num / np.where(em, den, 1.0), 0.0).astype(np.float32)
    got = g.filterSensitivity(radius, x.ravel()).cpu().numpy().reshape(em.shape)
    fin = np.isfinite(want)
    assert np.array_equal(np.isfinite(got), fin) and np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(got[np.isinf(got)], want[np.isinf(want)])
    assert np.all(np.abs(got[fin] - want[fin]) <= 1e-6 * np.maximum(np.abs(want[fin]), 1.0))
    vol = g.volumeRatio(x.ravel())
    ref = np.where(em, x.astype(np.float64), 0.0).sum()
    one = g.volumeRatio(np.ones(em.size, np.float32)) / em.sum()  # the divisor counts padded elements
    assert np.isnan(vol) if np.isnan(ref) else (vol == ref if np.isinf(ref) else abs(vol - ref * one) <= 1e-6 * abs(ref * one))
    with np.errstate(invalid="ignore", over="ignore"):
        s = 8.0 * (x.astype(np.float64) - 0.5)
        step = np.clip(np.nan_to_num((np.tanh(4.0) + np.tanh(s)) / (2 * np.tanh(4.0)), nan=1e-3), 1e-3, 1.0)
    heav = g.projectDensities(x.ravel(), 8.0).cpu().numpy().reshape(em.shape)
    assert np.max(np.abs(heav - np.where(em, step, 0.0))) < 1e-7


@pytest.mark.parametrize("dims", [(255, 5, 3), (256, 4, 4), (257, 3, 5), (1030, 3, 2), (16, 70, 70)])
def test_volume_of_long_rows(cuda, dims):
    """The volume on rows below, of and past a warp's 256 elements: FP64 sums, 1e-12 relative."""
    from robustoptspline3d_b200 import Config, HierarchyGrid
    prob = P.voids_box(*dims, nvoids=1)
    g = HierarchyGrid(prob["emask"], prob["fixed"], prob["load"], prob["normals"], Config(n_levels=4, first_factor=2))
    on = prob["emask"].ravel() > 0
    x = np.random.default_rng(101).uniform(0.1, 1, g.ne).astype(np.float32)
    per = g.volumeRatio(np.ones(g.ne, np.float32)) / on.sum()
    want = x[on].astype(np.float64).sum() * per
    assert abs(g.volumeRatio(x) - want) <= 1e-12 * want


@pytest.mark.parametrize("precision", [0, 1])
def test_worst_case_does_not_read_what_its_scratch_held(cuda, precision):
    """The Lanczos vectors share their memory with the load projection: what a
    projected vector left there (here NaN) has no part in the next search."""
    from robustoptspline3d_b200 import Config, HierarchyGrid
    prob = P.cantilever(16, 8, 8)
    g = HierarchyGrid(prob["emask"], prob["fixed"], prob["load"], prob["normals"],
                      Config(poisson_ratio=0.4, n_levels=2, first_factor=2, precision=precision))
    g.set_density(prob["rho"].astype(np.float32).ravel())
    g.update_stencil()
    want = g.worst_case(6, 0, 1e-10)
    assert np.isfinite(want[0]) and bool(cuda.isfinite(want[2]).all())
    g.forceProject(t(np.full(3 * g.nn, np.nan), cuda), 0)
    got = g.worst_case(6, 0, 1e-10)
    assert got[0] == want[0] and bool((got[1] == want[1]).all()) and bool((got[2] == want[2]).all())
    assert np.array_equal(got[3], want[3])
    g.close()


def test_set_density_has_read_its_argument(cuda):
    """The densities are the caller's again once the call returns, also where the handle's stream is behind."""
    import ctypes
    from robustoptspline3d_b200 import Config, HierarchyGrid
    prob = P.cantilever(24, 12, 12)
    g = HierarchyGrid(prob["emask"], prob["fixed"], prob["load"], prob["normals"], Config(n_levels=2, first_factor=2))
    stream = cuda.cuda.Stream()
    assert g.lib.rso_set_stream(g.h, ctypes.c_void_p(stream.cuda_stream)) == 0
    a = cuda.randn(4096, 4096, device="cuda")
    rho = cuda.full((g.ne,), 0.25, device="cuda")
    cuda.cuda.synchronize()
    with cuda.cuda.stream(stream):
        for _ in range(20):
            a = (a @ a) * 1e-4
    g.set_density(rho)
    rho.fill_(0.75)
    cuda.cuda.synchronize()
    got = g.get_density().cpu().numpy()
    assert (got[prob["emask"].ravel() > 0] == np.float32(0.25)).all()
    g.close()
