"""The separated form of the constant-coefficient operators (Laplace, VectorLaplace, mass matrix) against the oracle,
copy by copy: part of a tile of 8 x 16 columns per diamond (levels 1-3), two tiles (4) and eight (5), in one run of
levels (1, 2), with a shorter last run (3, 4) and in three equal ones (5), inputs whose duplicated nodes hold different
values, and each apply / communication mode; their CG (lateral_cg.cuh), tables and memory."""
import numpy as np
import pytest
import torch

from helpers import rel
from oracle_lib import Mesh, pcg

pytestmark = pytest.mark.gpu


def _apply(shell, C, pm, op_of, u, dtype, old, am, cm):
    cls = shell.VectorQ1Vec if u.ndim == 5 else shell.VectorQ1Scalar
    src, dst = cls(pm, dtype), cls(pm, dtype)
    src.set_numpy(u)
    dst.set_numpy(old)
    shell.apply(op_of(am, cm), src, dst)
    torch.cuda.synchronize()
    return dst.numpy().reshape(u.shape).astype(np.float64)


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-13), (torch.float32, 1e-5)])
@pytest.mark.parametrize("L", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("op,bc", [("laplace", 0), ("laplace", 1), ("vector", (0, 1)), ("vector", (1, 0)), ("mass", 0),
                                   ("mass_diag", 0)])
def test_every_copy_and_mode(op, bc, L, dtype, tol):
    """FP32: 1e-5 is the tolerance of the other single-precision operator tests"""
    from terraneo_b200 import shell, _capi as C
    om, pm = Mesh(L), shell.ShellMesh(L)
    rng = np.random.default_rng(L)
    u = rng.normal(size=((3,) if op == "vector" else ()) + om.shape).astype(np.float32).astype(np.float64)
    old = rng.normal(size=u.shape).astype(np.float32).astype(np.float64)
    if op == "laplace":
        ref, make = om.laplace(u, bc, 0), lambda am, cm: shell.Laplace(pm, bc, False, am, cm)
    elif op == "vector":
        ref, make = om.vector_laplace(u, *bc), lambda am, cm: shell.VectorLaplace(pm, *bc, False, am, cm)
    else:
        mode = int(op == "mass_diag")
        ref, make = om.kmass(np.ones(om.shape), u, mode), lambda am, cm: shell.KMass(pm, None, mode, am, cm)

    def halo(f):
        return om.halo_sum(f).reshape(u.shape)

    args = (shell, C, pm, make, u, dtype, old)
    assert rel(_apply(*args, C.APPLY_REPLACE, C.COMM_ADDITIVE), ref.reshape(u.shape)) <= tol
    own = _apply(*args, C.APPLY_REPLACE, C.COMM_SKIP)  # each copy its diamond's part: their sum is the result
    assert rel(halo(own), ref.reshape(u.shape)) <= tol
    assert rel(_apply(*args, C.APPLY_ADD, C.COMM_SKIP), own + old) <= tol
    assert rel(_apply(*args, C.APPLY_ADD, C.COMM_ADDITIVE), halo(own + old)) <= tol


@pytest.mark.parametrize("op", ["mass", "laplace", "vector_laplace"])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_first_apply_in_a_capture(op, dtype):
    """a mesh's first use of an operator's tables in a precision may be part of a graph, whatever was used before it"""
    from terraneo_b200 import shell
    cls = shell.VectorQ1Vec if op == "vector_laplace" else shell.VectorQ1Scalar
    make = {"mass": lambda m: shell.KMass(m), "laplace": lambda m: shell.Laplace(m, True),
            "vector_laplace": lambda m: shell.VectorLaplace(m, 1, 1)}[op]
    pm, warm = shell.ShellMesh(3), shell.ShellMesh(2)
    shell.apply(make(warm), *(cls(warm, dtype) for _ in range(2)))  # the module is loaded outside
    other = torch.float32 if dtype == torch.float64 else torch.float64
    shell.apply(make(pm), *(cls(pm, other) for _ in range(2)))
    src, dst, ref = (cls(pm, dtype) for _ in range(3))
    src.data.uniform_()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        shell.apply(make(pm), src, dst)
    graph.replay()
    shell.apply(make(pm), src, ref)
    torch.cuda.synchronize()
    assert torch.equal(dst.data, ref.data)


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-13), (torch.float32, 1e-5)])
def test_add_mode_from_two_streams(dtype, tol):
    """applies on several streams that add into one field without communication lose no term: each of the 32 is a
    thirty-second of the sum, far above the tolerance"""
    from terraneo_b200 import shell, _capi as C
    pm, n = shell.ShellMesh(5), 16
    src, dst, once = (shell.VectorQ1Scalar(pm, dtype) for _ in range(3))
    src.data.uniform_()
    shell.apply(shell.KMass(pm, None, 0, C.APPLY_REPLACE, C.COMM_SKIP), src, once)
    add = shell.KMass(pm, None, 0, C.APPLY_ADD, C.COMM_SKIP)
    dst.data.zero_()
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for s in streams:
        with torch.cuda.stream(s):
            torch.cuda._sleep(5_000_000)  # both queues fill before either runs
    for _ in range(n):
        for s in streams:
            with torch.cuda.stream(s):
                shell.apply(add, src, dst)
    torch.cuda.synchronize()
    want = 2 * n * once.data.double()
    assert float((dst.data.double() - want).norm() / want.norm()) <= tol


@pytest.mark.parametrize("solve", ["laplace", "projection"])
def test_cg_steps_after_convergence_are_nearly_free(solve):
    """a relative tolerance of 1e30 is met by the first step: the steps the host issued meanwhile cost little beside real
    ones (a quarter is the bound; half when they read their operands all the same)"""
    import time
    from terraneo_b200 import shell
    pm = shell.ShellMesh(6)
    b, x = shell.VectorQ1Scalar(pm), shell.VectorQ1Scalar(pm)
    b.data.normal_()
    b.data[..., 0] = b.data[..., -1] = 0.0
    fv = torch.randn((10,) + (pm.n1 + 1,) * 3, dtype=torch.float64, device="cuda")
    work = torch.empty(5 * pm.stored_nodes, dtype=torch.float64, device="cuda")

    def seconds(its, rtol):
        best = 1e9
        for _ in range(8):
            x.data.zero_()
            torch.cuda.synchronize()
            t = time.perf_counter()
            if solve == "laplace":
                n, _ = shell.laplace_pcg(pm, b, x, its, rtol)
            else:
                n = shell.l2_project_fv_to_fe(pm, fv, x, False, its, rtol, 1e-300, work)
            torch.cuda.synchronize()
            best = min(best, time.perf_counter() - t)
        assert n == (1 if rtol > 1 else its)
        return best

    one = seconds(1, 1e30)
    assert seconds(16, 1e30) - one <= 0.25 * (seconds(16, 1e-300) - one)


def _row_pattern(om):
    """A direction whose <p, A p> a plain sum along y gets wrong: in every row of interior columns one node of size one,
    then seven whose terms are each just below half a unit in the last place of the first one's"""
    import math
    ones, e = np.ones(om.shape), np.zeros(om.shape)
    s = np.full(om.shape, 2.0 ** -27)
    for _ in range(3):
        e[:, 1:-1, 1, 1:-1] = 1.0
        e[:, 1:-1, 3::2, 1:-1] = s[:, 1:-1, 3::2, 1:-1]
        e[:, :, -1] = 0.0
        terms = e * om.kmass(ones, e, 0)
        want = 0.95 * 2.0 ** -54 * terms[:, 1:-1, 1:2, 1:-1]
        s[:, 1:-1, 3:-1:2, 1:-1] *= np.sqrt(want / terms[:, 1:-1, 3:-1:2, 1:-1])
    return e, ones, lambda p, q: math.fsum((p * q)[om.omask == 1])


def test_projection_sums_every_product():
    """alpha = <r, r> / <p, A p> of the projection's first CG step, read off thousands of nodes, against exact sums of the
    rounded products: one unit in the last place; seven terms lost per row would move it by 3.5e-16"""
    from terraneo_b200 import shell
    om, pm = Mesh(4), shell.ShellMesh(4)
    e, ones, dot = _row_pattern(om)
    x0, _ = pcg(lambda v: om.kmass(ones, v, 0), om.dot, -e, 200, 1e-17)  # the residual of an empty right-hand side is e
    mass = shell.KMass(pm)
    x, p, ap = (shell.VectorQ1Scalar(pm) for _ in range(3))
    x.set_numpy(x0)
    shell.apply(mass, x, p)
    p.data.neg_()
    shell.apply(mass, p, ap)
    pn, apn = p.numpy()[0], ap.numpy()[0]
    assert rel(pn, e) <= 1e-12
    shell.l2_project_fv_to_fe(pm, torch.zeros((10,) + (om.N + 2,) * 3, dtype=torch.float64, device="cuda"), x,
                              max_iterations=1, relative_tolerance=0.0, absolute_tolerance=0.0)
    step = (x.numpy()[0].astype(np.longdouble) - x0)[pn > 0.5] / pn[pn > 0.5]
    alpha = dot(pn, pn) / dot(pn, apn)
    assert abs(float(step.mean() / alpha - 1)) <= 2.0 ** -52


def _mass_factors(om):
    """lateral stencil {offset: [10, N-1, N-1]} of the interior columns and radial factors [3][N] of the mass matrix in
    extended precision (the 3x2 rule: lateral points (2/3, 1/6), (1/6, 2/3), (1/6, 1/6), zeta = -+1/sqrt(3), weights 1/6)"""
    N, LD, lat = om.N, np.longdouble, {}
    P, r = om.coords.astype(LD), om.radii[0].astype(LD)
    for nodes in (((0, 0), (1, 0), (0, 1)), ((1, 1), (0, 1), (1, 0))):
        p = [P[:, x:x + N, y:y + N] for x, y in nodes]
        D = np.abs((np.cross(p[1] - p[0], p[2] - p[0]) * p[0]).sum(-1))
        for i, a in enumerate(nodes):
            for j, b in enumerate(nodes):
                e = lat.setdefault((b[0] - a[0], b[1] - a[1]), np.zeros(P.shape[:3], LD))
                e[:, a[0]:a[0] + N, a[1]:a[1] + N] += D / (12 if i == j else 24)
    h, g, f = (r[1:] - r[:-1]) / 2, 1 / np.sqrt(LD(3)), np.zeros((3, N), LD)
    for z in (-g, g):
        n, rr = ((1 - z) / 2, (1 + z) / 2), r[:-1] + h * (1 + z)
        for k in range(3):
            f[k] += h * rr * rr * n[k // 2] * n[(k + 1) // 2]
    return {e: v[:, 1:-1, 1:-1] for e, v in lat.items()}, f


@pytest.mark.parametrize("L,rmin", [(3, 0.55), (4, 0.35), (4, 0.55)])
def test_mass_tables_are_rounded_once(L, rmin):
    """entries of the mass matrix, read off by fields that are one at every third node: stencil and radial factor carry
    half a unit each, their product another (3 x 2^-53), and the node's own entry one for the sum of its two layers"""
    from terraneo_b200 import shell
    om, pm = Mesh(L, rmin), shell.ShellMesh(L, rmin, 1.0)
    lat, f = _mass_factors(om)
    N, op = om.N, shell.KMass(pm)
    src, dst = shell.VectorQ1Scalar(pm), shell.VectorQ1Scalar(pm)
    own = np.zeros(N + 1, np.longdouble)
    own[:-1] += f[0]
    own[1:] += f[2]
    worst = [0.0, 0.0]
    for a, b, c in np.ndindex(3, 3, 3):
        u = np.zeros(om.shape)
        u[:, a::3, b::3, c::3] = 1.0
        src.set_numpy(u)
        shell.apply(op, src, dst)
        got = dst.numpy()[0][:, 1:-1, 1:-1]
        for (dx, dy), s in lat.items():
            at = u[:, 1 + dx:N + dx, 1 + dy:N + dy] != 0.0  # columns whose neighbour (dx, dy) holds ones, at their levels
            for k, (here, want) in enumerate(((at, s[..., None] * own),
                                              (at[..., :-1], s[..., None] * f[1]), (at[..., 1:], s[..., None] * f[1]))):
                out = got if k == 0 else (got[..., 1:] if k == 1 else got[..., :-1])
                worst[k > 0] = max(worst[k > 0], float(np.abs(out[here] / want[here] - 1).max(initial=0)))
    assert worst[1] <= 3.01 * 2.0 ** -53 and worst[0] <= 4.01 * 2.0 ** -53, worst


def test_mesh_tables_take_one_launch_each():
    """what a mesh forms on the device, whatever it is used for: triangle vectors and mass stencils, both precisions at
    once"""
    from torch.profiler import ProfilerActivity, profile
    from terraneo_b200 import shell
    shell.ShellMesh(2)
    with profile(activities=[ProfilerActivity.CUDA], acc_events=True) as prof:
        mesh = shell.ShellMesh(3)
        torch.cuda.synchronize()
    del mesh
    kernels = [e.name for e in prof.events() if "_kernel" in e.name]
    assert len(kernels) == 2, kernels


@pytest.mark.parametrize("L,kept", [(5, 16 << 20), (7, 0)])
def test_solver_memory_is_given_back(L, kept):
    """a Laplace solve's four fields (11 MB at level 5, 700 MB at level 7) stay with the mesh up to 128 MiB and once,
    larger ones go back when the solve returns; allocations come in pages of 2 MiB"""
    from terraneo_b200 import shell
    pm = shell.ShellMesh(L)
    b, x = shell.VectorQ1Scalar(pm), shell.VectorQ1Scalar(pm)
    b.data.normal_()
    m2 = shell.ShellMesh(2)
    shell.laplace_pcg(m2, shell.VectorQ1Scalar(m2), shell.VectorQ1Scalar(m2), 1)  # the module is loaded
    shell.apply(shell.Laplace(pm, True), b, x)  # the operator's stencils stay with the mesh
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for _ in range(3):
        shell.laplace_pcg(pm, b, x, 2)
    assert before - torch.cuda.mem_get_info()[0] <= kept + (4 << 20)


@pytest.mark.parametrize("solve", ["laplace", "projection"])
def test_cg_with_any_iteration_limit(solve):
    """the limit sizes no memory (17 GB at the largest when every step had an entry): such a call takes no longer than one
    with a small limit; and steps are counted beyond the kept history of 4,096"""
    import time
    from terraneo_b200 import shell
    pm = shell.ShellMesh(2)
    b, x = shell.VectorQ1Scalar(pm), shell.VectorQ1Scalar(pm)
    x.data.normal_()
    shell.apply(shell.KMass(pm), x, b)  # equal copies of every node: the system has a solution
    b.data[..., 0] = b.data[..., -1] = 0.0
    fv = torch.randn((10,) + (pm.n1 + 1,) * 3, dtype=torch.float64, device="cuda")

    def run(its, rtol, atol):
        best, n = 1e9, 0
        for _ in range(4):
            x.data.zero_()
            torch.cuda.synchronize()
            t = time.perf_counter()
            if solve == "laplace":
                n, _ = shell.laplace_pcg(pm, b, x, its, rtol, atol)
            else:
                n = shell.l2_project_fv_to_fe(pm, fv, x, False, its, rtol, atol)
            best = min(best, time.perf_counter() - t)
        return n, best

    n, small = run(1000, 1e-10, 1e-30)
    assert 0 < n < 1000
    free = torch.cuda.mem_get_info()[0]
    m, large = run(2**31 - 1, 1e-10, 1e-30)
    assert m == n and large <= small + 1e-3 and free - torch.cuda.mem_get_info()[0] <= 4 << 20, (n, m, small, large)
    assert run(4096, -1.0, 0.0)[0] == 4096 and run(4100, -1.0, 0.0)[0] == 4100  # never met
