"""Kernels and dispatch rules at the sizes where they can go wrong (edges of tiles and chunks,
remainders, the smallest and largest of a range), against the FP64 oracle."""
import numpy as np
import pytest

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


# coarse levels of 2 to 17 nodes an edge: colours of one node, of fewer and of more than the 32 a CTA
# takes, with a ragged last CTA; the ellipsoid leaves inactive nodes inside the box
@pytest.mark.parametrize("gen", [lambda: P.cantilever(6, 4, 3), lambda: P.cantilever(30, 21, 13),
                                 lambda: P.ellipsoid(64, 36, 28)])
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
