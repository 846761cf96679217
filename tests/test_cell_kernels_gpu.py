"""The kernels that run one thread per cell with the upper nodes handed to the lane above (cell.cuh), against the oracle
at the levels where that can go wrong: partial warps and several columns per warp (1-3), one column per warp (5), a
column over two warps (6); and the two-kernel CG (lateral_cg.cuh) against the oracle's iterates, with part of a tile per
diamond (1-3), two tiles (4) and eight tiles and several runs of levels (5)."""
import functools

import numpy as np
import pytest
import torch

from helpers import random_vector, rel, viscosity_field
from oracle_lib import Mesh, pcg

pytestmark = pytest.mark.gpu
LEVELS = [1, 2, 3, 5, 6]
TOL = {torch.float64: 1e-12, torch.float32: 1e-5}  # the tolerances of the operators' other tests


def _run(shell, op, pm, u, dtype, out_mesh=None, ncomp=None):
    cls = {1: shell.VectorQ1Scalar, 3: shell.VectorQ1Vec}
    src = cls[3 if u.ndim == 5 else 1](pm if op is None or u.shape[-1] == pm.n1 else out_mesh, dtype)
    dst = cls[ncomp or src.ncomp](out_mesh or pm, dtype)
    src.set_numpy(u)
    shell.apply(op, src, dst)
    torch.cuda.synchronize()
    return dst.numpy().reshape((3,) + dst.mesh.shape if dst.ncomp == 3 else dst.mesh.shape).astype(np.float64)


@functools.lru_cache(maxsize=None)
def _case(L):
    from terraneo_b200 import shell
    om = Mesh(L)
    return om, shell.ShellMesh(L), viscosity_field(om, seed=L), random_vector(om, seed=L)


@pytest.fixture(scope="module", autouse=True)
def _release():
    yield
    _case.cache_clear()


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("treat", [True, False])
@pytest.mark.parametrize("L", LEVELS)
def test_divkgrad(L, treat, dtype):
    from terraneo_b200 import shell
    om, pm, k, u = _case(L)
    kv = shell.VectorQ1Scalar(pm, dtype)
    kv.set_numpy(k)
    for single in (False, True) if L < 6 else (False,):
        got = _run(shell, shell.DivKGrad(pm, kv, treat, single_quadpoint=single), pm, u[0], dtype)
        assert rel(got, om.divkgrad(k, u[0], treat, False, single)) <= TOL[dtype]


@pytest.mark.parametrize("treat", [True, False])
@pytest.mark.parametrize("L", LEVELS)
def test_epsdivdiv3x2(L, treat):
    from terraneo_b200 import shell
    om, pm, k, u = _case(L)
    kv = shell.VectorQ1Scalar(pm)
    kv.set_numpy(k)
    assert rel(_run(shell, shell.EpsilonDivDiv(pm, kv, treat), pm, u, torch.float64),
               om.epsdivdiv3x2(k, u, treat)) <= 1e-12


@pytest.mark.parametrize("L,kappa,treat,lumped",
                         [(L, *p) for L in LEVELS[:-1] for p in ((1e-3, True, False), (1e-6, False, False),
                                                                 (0.5, True, True), (0.0, True, False))]
                         + [(6, 1e-3, True, False)])
def test_supg(L, kappa, treat, lumped):
    """Peclet numbers from 1e-3 (the small-argument branch of tau) to 1e7; some nodes at rest"""
    from terraneo_b200 import shell
    om, pm, k, u = _case(L)
    vel = np.where(np.abs(u[:1]) > 1.5, 0.0, u)
    vv = shell.VectorQ1Vec(pm)
    vv.set_numpy(vel)
    op = shell.UnsteadyAdvectionDiffusionSUPG(pm, vv, kappa, 1e-2, treat, False, 1.5, lumped)
    assert rel(_run(shell, op, pm, u[0], torch.float64), om.supg(vel, u[0], kappa, 1e-2, 1.5, lumped, treat)) <= 1e-12


@pytest.mark.parametrize("bc", [(1, 2), (2, 0)])
@pytest.mark.parametrize("L", LEVELS[1:])  # the pressure mesh is one level coarser
def test_stokes_blocks(L, bc):
    from terraneo_b200 import shell
    om, pm, k, u = _case(L)
    oc, pc = Mesh(L - 1), shell.ShellMesh(L - 1)
    assert rel(_run(shell, shell.Divergence(pm, pc, *bc), pm, u, torch.float64, pc, 1),
               om.divergence(oc, u, *bc)) <= 1e-12
    p = random_vector(oc, seed=1, ncomp=1)
    vp, vu = shell.VectorQ1Scalar(pc), shell.VectorQ1Vec(pm)
    vp.set_numpy(p)
    shell.apply(shell.Gradient(pm, pc, *bc), vp, vu)
    assert rel(vu.numpy(), om.gradient(oc, p, *bc)) <= 1e-12


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("bc", [(0, 0), (1, 2), (2, 0)])
@pytest.mark.parametrize("L", LEVELS)
def test_viscosity_gradient(L, bc, dtype):
    """linear in k: d(lambda^T A(k) u)/dk times a perturbation of k, summed over the owned nodes, is lambda^T A(dk) u"""
    from terraneo_b200 import shell
    om, pm, _, _ = _case(L)
    u, lam = (random_vector(om, seed=L + i).astype(np.float32).astype(np.float64) for i in (0, 1))
    dk = random_vector(om, seed=L + 2, ncomp=1)
    vu, vl, g = shell.VectorQ1Vec(pm, dtype), shell.VectorQ1Vec(pm, dtype), shell.VectorQ1Scalar(pm, dtype)
    vu.set_numpy(u)
    vl.set_numpy(lam)
    shell.epsdivdiv_kgrad(pm, *bc, vu, vl, g)
    own = om.omask == 1
    terms = om.kerngen(dk, u, *bc) * lam
    want = float((terms * own).sum())
    # a sum of N terms of both signs: bounded by their absolute sum
    assert abs(float((g.numpy()[0] * dk * own).sum()) - want) <= TOL[dtype] * float(np.abs(terms * own).sum())


@pytest.mark.parametrize("L,its", [(L, i) for L in (1, 2, 3) for i in (1, 2, 9, 17)] + [(4, 2), (4, 9), (5, 2), (5, 9)])
def test_cg_iterates(L, its):
    """the iterate after 1, 2 (each direction field), 9 and 17 (the stopping flag is looked at by then) steps"""
    from terraneo_b200 import shell
    om, pm, k, u = _case(L)
    b = om.kmass(np.ones(om.shape), u[0], 0)
    b[..., 0] = b[..., -1] = 0.0
    vb, vx = shell.VectorQ1Scalar(pm), shell.VectorQ1Scalar(pm)
    vb.set_numpy(b)
    n, rr = shell.laplace_pcg(pm, vb, vx, its, 1e-11)
    want, m = om.laplace_pcg(b, its, 1e-11)
    assert abs(n - m) <= 1 and rel(vx.numpy()[0], want) <= 1e-11  # level 1 ends by exhausting its few directions
    fv = np.zeros(om.fv_shape)
    fv[:, 1:-1, 1:-1, 1:-1] = np.random.default_rng(its).normal(size=(10,) + (om.N,) * 3)
    n = shell.l2_project_fv_to_fe(pm, torch.as_tensor(fv, device="cuda"), vx, max_iterations=its)
    rhs, _ = om.fv_to_fe_rhs(fv)
    ones = np.ones(om.shape)
    # from x: the projection solves for the correction of its initial guess
    r0 = rhs - om.kmass(ones, want, 0)
    dx, m = pcg(lambda v: om.kmass(ones, v, 0), om.dot, r0, its, 1e-12, 1e-12)
    assert abs(n - m) <= 1 and rel(vx.numpy()[0], want + dx) <= 1e-11


@pytest.mark.parametrize("L,kappa", [(1, 1e-2), (3, 1e-2), (5, 0.0), (5, 1e-2), (6, 1e-2)])
def test_fct_runs(L, kappa):
    """the FCT kernels' runs along x: one cell per thread (1, 3), two (5) and eight (6), fewer than 32 cells in r (1, 3)"""
    from terraneo_b200 import shell
    om, pm = Mesh(L), shell.ShellMesh(L)
    N, rng = om.N, np.random.default_rng(L)
    vel, c = random_vector(om, seed=L), om.fv_cell_centers()
    inner = (slice(None),) + (slice(1, N + 1),) * 3
    T = np.zeros(om.fv_shape)
    T[inner] = rng.uniform(size=T[inner].shape)
    fct, v = shell.FCTAdvectionDiffusion(pm), shell.VectorQ1Vec(pm)
    v.set_numpy(vel)
    dt = om.fct_dt_stable(c, vel, kappa)
    assert fct.dt_stable(v, kappa) == pytest.approx(dt, rel=1e-12)
    ref, _ = om.fct_step(c, vel, om.fv_ghost_update(T), 0.5 * dt, kappa, None, True, None)
    Tg = torch.as_tensor(T, device="cuda")
    fct.step(Tg, v, 0.5 * dt, kappa, None, True, None)
    assert rel(Tg.cpu().numpy()[inner], ref[inner]) <= 1e-12  # the tolerance of the level-2 and 4 tests times ten: rough fields
