"""Performance cases: what a mantle-convection program has this framework do.

Every case is one pass through the public Python layer (terraneo_b200.shell):

  viscous          epsilon-div-div apply, one-point rule: the velocity block of every Stokes iteration and of
                   every multigrid smoothing step (FP64 in the Krylov loop, FP32 in the V-cycle)
  viscous3x2       the same operator with the six-point rule and interpolated viscosity
  poisson_cg       a scalar Laplace system solved with plain CG for a fixed number of iterations
  gradient_form    one apply of Laplace, VectorLaplace or DivKGrad (scalar and temperature problems, their smoothers)
  stokes_blocks    Divergence and Gradient, the two coupling blocks of one Stokes operator apply
  viscosity_grad   the backward pass: derivative of lambda^T A(k) u with respect to the nodal viscosity
  energy_fct       one explicit energy step: stable step size, FCT step, Dirichlet temperatures
  projection       FV temperature projected onto the FE space (a fixed number of mass-matrix CG iterations)
  energy_supg      one apply of the implicit SUPG energy operator (what its Krylov solver repeats)
  stokes_solve     buoyancy right-hand side and a Stokes solve with the application's solver settings, ten
                   FGMRES iterations with the FP32 multigrid preconditioner

The shell has 10 x N^3 cells with N = 2^level, so N + 1 nodes (an odd number) in every direction; levels run
from the coarsest multigrid level to the largest level a single time step is run at.
"""
import functools
import math

import numpy as np
import torch

from terraneo_b200 import _capi as C
from terraneo_b200 import shell

BC = {"neumann": C.BC_NEUMANN, "dirichlet": C.BC_DIRICHLET, "freeslip": C.BC_FREESLIP}
DTYPE = {"f64": torch.float64, "f32": torch.float32}
CG_ITERATIONS = 100
PROJECTION_ITERATIONS = 20  # a warm-started projection takes about as many
STOKES_ITERATIONS = 10
# the largest eigenvalue of D^-1 A per level, given: ten power iterations from a random start would give each solver
# object estimates, and so iterates, that differ in the third digit
CHEBYSHEV_ESTIMATE = 6.0
CFL = 0.5  # fraction of the stable step size taken by the energy step


# --- the cases -------------------------------------------------------------------------------------------------

def listed():
    return [
        # the published benchmark operator at the framework's benchmark level, no-slip boundaries
        dict(name="viscous_f64_l6", kind="viscous", level=6, dtype="f64", bc_cmb="dirichlet", bc_surface="dirichlet",
             r_min=0.55),
        # the finest smoother level of a level-7 time step: FP32, free-slip boundaries
        dict(name="viscous_f32_l7", kind="viscous", level=7, dtype="f32", bc_cmb="freeslip", bc_surface="freeslip",
             r_min=0.55),
        # a coarse multigrid level, where launches and latency count
        dict(name="viscous_f64_l3", kind="viscous", level=3, dtype="f64", bc_cmb="dirichlet", bc_surface="freeslip",
             r_min=0.5),
        # the fully integrated operator for strongly varying viscosity
        dict(name="viscous3x2_f64_l6", kind="viscous3x2", level=6, dtype="f64", treat=True, r_min=0.55),
        # the scalar model problem: 100 CG iterations at level 5
        dict(name="poisson_cg_l5", kind="poisson_cg", level=5, r_min=0.55),
        # variable-coefficient diffusion on a fine scalar multigrid level
        dict(name="divkgrad_f64_l6", kind="gradient_form", op="divkgrad", level=6, dtype="f64", treat=True,
             r_min=0.55),
        # both coupling blocks of a Stokes apply, free-slip
        dict(name="stokes_blocks_f64_l6", kind="stokes_blocks", level=6, dtype="f64", bc_cmb="freeslip",
             bc_surface="freeslip", r_min=0.55),
        # the backward pass of an adjoint viscosity inversion
        dict(name="viscosity_grad_f64_l6", kind="viscosity_grad", level=6, dtype="f64", bc_cmb="freeslip",
             bc_surface="freeslip", r_min=0.55),
        # the energy step of a level-7 run: the largest case
        dict(name="energy_fct_l7", kind="energy_fct", level=7, kappa=0.0, r_min=0.55),
        # the temperature hand-over of a level-6 run
        dict(name="projection_l6", kind="projection", level=6, r_min=0.55),
        # the implicit energy operator
        dict(name="energy_supg_f64_l6", kind="energy_supg", level=6, dtype="f64", kappa=1e-3, treat=True,
             lumped=False, r_min=0.55),
        # a whole call: right-hand side and ten preconditioned FGMRES iterations at level 5
        dict(name="stokes_solve_l5", kind="stokes_solve", level=5, bc_cmb="freeslip", bc_surface="freeslip",
             r_min=0.55),
    ]


# largest level drawn per kind; the smallest is 3 (2 where no multigrid hierarchy stands behind the call)
_MAX_LEVEL = {"viscous": 7, "viscous3x2": 6, "poisson_cg": 5, "gradient_form": 7, "stokes_blocks": 7,
              "viscosity_grad": 6, "energy_fct": 7, "projection": 6, "energy_supg": 6, "stokes_solve": 5}


def draw(rng):
    kind = rng.choice(sorted(_MAX_LEVEL))
    lo = {"stokes_solve": 4}.get(kind, 2)
    case = dict(kind=kind, level=rng.randint(lo, _MAX_LEVEL[kind]), r_min=round(rng.uniform(0.35, 0.75), 4))
    if kind in ("viscous", "stokes_blocks", "viscosity_grad"):
        bcs = ("dirichlet", "freeslip") if kind == "stokes_blocks" else ("dirichlet", "freeslip", "neumann")
        case["bc_cmb"], case["bc_surface"] = rng.choice(bcs), rng.choice(bcs)
    if kind == "stokes_solve":
        case["bc_cmb"] = case["bc_surface"] = rng.choice(("dirichlet", "freeslip"))
        case["r_min"] = round(rng.uniform(0.5, 0.7), 4)  # about the mantle's ratio of radii, 0.55
    if kind == "gradient_form":
        case["op"] = rng.choice(("laplace", "vector_laplace", "divkgrad"))
    if kind in ("gradient_form", "viscous3x2", "energy_supg"):
        case["treat"] = rng.random() < 0.75
    if kind in ("viscous", "viscous3x2", "gradient_form", "stokes_blocks", "viscosity_grad", "energy_supg"):
        case["dtype"] = rng.choice(("f64", "f64", "f32"))
    if kind == "energy_fct":
        case["kappa"] = rng.choice((0.0, 0.0, 1e-3))
    if kind == "energy_supg":
        case["kappa"], case["lumped"] = 10.0 ** rng.uniform(-6, -2), rng.random() < 0.25
    return case


# --- geometry and fields ---------------------------------------------------------------------------------------
# The lateral mesh in plain numpy: ten icosahedral diamonds refined by normalised chord bisection.

_DIAMONDS = ((0, 5, 6, 1), (0, 1, 7, 2), (0, 2, 8, 3), (0, 3, 9, 4), (0, 4, 10, 5),
             (11, 7, 1, 6), (11, 8, 2, 7), (11, 9, 3, 8), (11, 10, 4, 9), (11, 6, 5, 10))


@functools.lru_cache(maxsize=8)
def _lateral(level):
    """lateral points [10, N+1, N+1, 3], the number of distinct ones and the distinct point of each column"""
    N = 1 << level
    pi5 = 0.2 * math.pi
    w = 2.0 * math.acos(1.0 / (2.0 * math.sin(pi5)))
    ico = [(0.0, 0.0, 1.0)]
    ico += [(math.sin(w) * math.cos((2 * k - 1) * pi5), math.sin(w) * math.sin((2 * k - 1) * pi5), math.cos(w))
            for k in range(1, 6)]
    ico += [(math.sin(w) * math.cos(2 * (k - 1) * pi5), math.sin(w) * math.sin(2 * (k - 1) * pi5), -math.cos(w))
            for k in range(1, 6)]
    ico += [(0.0, 0.0, -1.0)]
    p = np.zeros((10, N + 1, N + 1, 3))
    for d, v in enumerate(_DIAMONDS):
        a, b = (1, 3) if d < 5 else (3, 1)
        p[d, 0, 0], p[d, N, 0], p[d, N, N], p[d, 0, N] = ico[v[0]], ico[v[a]], ico[v[2]], ico[v[b]]
    s = N
    while s > 1:
        h = s // 2
        p[:, 0::s, h::s] = p[:, 0::s, 0:-h:s] + p[:, 0::s, s::s]
        p[:, h::s, 0::s] = p[:, 0:-h:s, 0::s] + p[:, s::s, 0::s]
        p[:, h::s, h::s] = p[:, 0:-h:s, s::s] + p[:, s::s, 0:-h:s]
        for i, j in ((0, h), (h, 0), (h, h)):
            q = p[:, i::s, j::s]
            q /= np.linalg.norm(q, axis=-1, keepdims=True)
        s = h
    key = np.round(p.reshape(-1, 3) * 2.0 ** 30).astype(np.int64)
    order = np.lexsort(key.T)
    srt = key[order]
    new = np.concatenate(([True], np.abs(np.diff(srt, axis=0)).max(axis=1) > 0))
    gid = np.empty(len(order), np.int64)
    gid[order] = np.cumsum(new) - 1
    assert int(gid.max()) + 1 == 10 * N * N + 2
    return p, int(gid.max()) + 1, gid


class _Geo:
    """torch copies of the geometry of one mesh, and sums over duplicated nodes"""

    def __init__(self, level, r_min, device):
        p, self.groups, gid = _lateral(level)
        self.N = N = 1 << level
        self.n1, self.device = N + 1, device
        self.p = torch.as_tensor(p, device=device)
        self.gid = torch.as_tensor(gid, device=device)
        r = r_min + np.arange(N + 1) * ((1.0 - r_min) / N)
        r[N] = 1.0
        self.r = torch.as_tensor(r, device=device)
        first = np.full(self.groups, len(gid), np.int64)
        np.minimum.at(first, gid, np.arange(len(gid)))
        owned = np.zeros(len(gid), bool)
        owned[first] = True
        self.owned = torch.as_tensor(owned.reshape(10, N + 1, N + 1, 1), device=device)
        self.shape = (10, N + 1, N + 1, N + 1)

    def spread(self, columns):
        """values per distinct lateral point [G, N+1] as a consistent field"""
        return columns[self.gid].view(self.shape)

    def halo(self, f):
        c = f.reshape(-1, self.n1)
        return torch.zeros(self.groups, self.n1, dtype=f.dtype, device=f.device).index_add_(0, self.gid, c)[
            self.gid].view(self.shape)

    def position(self):
        return self.p[:, :, :, None, :] * self.r[:, None]

    def corner(self, f, w, n):
        """values of a node field at node n of wedge w of every cell [10, N, N, N]"""
        dx, dy, dr = _node(w, n)
        N = self.N
        return f[:, dx:dx + N, dy:dy + N, dr:dr + N]

    def lateral(self, w):
        """the three lateral vertices of wedge w of every cell, each [10, N, N, 1, 3]"""
        N = self.N
        out = []
        for n in range(3):
            dx, dy, _ = _node(w, n)
            out.append(self.p[:, dx:dx + N, dy:dy + N, None, :])
        return out


def _node(w, n):
    """(x, y, r) offset of node n of wedge w in its cell"""
    lat = ((0, 0), (1, 0), (0, 1)) if w == 0 else ((1, 1), (0, 1), (1, 0))
    return lat[n % 3] + (n // 3,)


def _rng(seed, device):
    return torch.Generator(device=device).manual_seed(1000003 * (seed + 1))


def _waves(geo, g, scale=3.0, count=4):
    """a smooth random field of unit size"""
    x = geo.position()
    out = torch.zeros(geo.shape, dtype=torch.float64, device=geo.device)
    for _ in range(count):
        k = torch.randn(3, generator=g, dtype=torch.float64, device=geo.device) * scale
        ph = torch.rand(1, generator=g, dtype=torch.float64, device=geo.device) * 6.28
        out += torch.sin((x * k).sum(-1) + ph)
    out /= math.sqrt(count / 2.0)
    # equal copies of a duplicated node, whatever the rounding of their positions
    first = torch.empty(geo.groups, geo.n1, dtype=torch.float64, device=geo.device)
    first[geo.gid[geo.owned.view(-1)]] = out.view(-1, geo.n1)[geo.owned.view(-1)]
    return geo.spread(first)


def _noise(geo, g):
    return geo.spread(torch.randn(geo.groups, geo.n1, generator=g, dtype=torch.float64, device=geo.device))


def _viscosity(geo, g):
    """contrast 1e4: a radial ramp and lateral anomalies"""
    ramp = (geo.r - geo.r[0]) / (1.0 - geo.r[0])
    return torch.exp(math.log(1e4) * (0.5 * ramp + 0.25 * (1.0 + _waves(geo, g).clamp(-1, 1)))).clamp(1.0, 1e4)


def _vector(geo, g):
    """what a Krylov vector holds: a smooth flow and rough components"""
    return torch.stack([_waves(geo, g) + 0.3 * _noise(geo, g) for _ in range(3)])


def _flow(geo, g):
    """a velocity: rotation and smooth cells"""
    w = torch.randn(3, generator=g, dtype=torch.float64, device=geo.device)
    x = geo.position()
    rot = torch.linalg.cross(w.expand_as(x), x)
    rot = rot.movedim(-1, 0)
    return torch.stack([geo.halo(torch.where(geo.owned, rot[c], 0.0)) + 0.3 * _waves(geo, g) for c in range(3)])


def _cell_positions(geo):
    p, r = geo.p, geo.r
    lat = 0.25 * (p[:, 1:, 1:] + p[:, :-1, 1:] + p[:, 1:, :-1] + p[:, :-1, :-1])
    return lat[:, :, :, None, :] * (0.5 * (r[1:] + r[:-1]))[:, None]


def _temperature_fv(geo, g):
    """a conductive profile, plumes and one sharp front, with (unset) ghost layers"""
    x = _cell_positions(geo)
    rr = x.norm(dim=-1)
    prof = ((1 / rr - 1) / (1 / geo.r[0] - 1)).clamp(0, 1)
    k = torch.randn(3, generator=g, dtype=torch.float64, device=geo.device) * 4.0
    T = prof + 0.2 * torch.sin((x * k).sum(-1)) + 0.3 * ((x * k.flip(0)).sum(-1) > 0.5)
    out = torch.zeros((10,) + (geo.N + 2,) * 3, dtype=torch.float64, device=geo.device)
    out[:, 1:-1, 1:-1, 1:-1] = T
    return out


def _inputs(case, seed, device):
    """the input fields of a case in FP64, rounded to the case's data type"""
    geo, g = _Geo(case["level"], case["r_min"], device), _rng(seed, device)
    dt = DTYPE[case.get("dtype", "f64")]
    kind, f = case["kind"], {}
    if kind in ("viscous", "viscous3x2"):
        f["k"], f["u"] = _viscosity(geo, g), _vector(geo, g)
    elif kind == "poisson_cg":
        # a load vector: a smooth source times the cell volume, zero on the boundary layers
        b = _waves(geo, g) * geo.r ** 2 / (geo.N ** 3)
        b[..., 0] = 0.0
        b[..., -1] = 0.0
        f["b"] = b
    elif kind == "gradient_form":
        n = 3 if case["op"] == "vector_laplace" else 1
        f["u"] = _vector(geo, g)[:n]
        if case["op"] == "divkgrad":
            f["k"] = _viscosity(geo, g)
    elif kind == "stokes_blocks":
        f["u"] = _vector(geo, g)
        gc = _Geo(case["level"] - 1, case["r_min"], device)
        f["p"] = _waves(gc, g) + 0.3 * _noise(gc, g)
    elif kind == "viscosity_grad":
        f["u"], f["lam"] = _vector(geo, g), _vector(geo, g)
    elif kind == "energy_fct":
        f["v"], f["T"] = _flow(geo, g), _temperature_fv(geo, g)
    elif kind == "projection":
        f["T"] = _temperature_fv(geo, g)
    elif kind == "energy_supg":
        f["v"], f["T"] = _flow(geo, g), _waves(geo, g) + 0.1 * _noise(geo, g)
    elif kind == "stokes_solve":
        f["k"] = _viscosity(geo, g)
        f["T"] = ((1 / geo.r - 1) / (1 / geo.r[0] - 1)).expand(geo.shape) + 0.1 * _waves(geo, g)
    return geo, {n: t.to(dt).contiguous() for n, t in f.items()}


# --- the measured passes ---------------------------------------------------------------------------------------

def _scalar(mesh, data):
    return shell.VectorQ1Scalar(mesh, data.dtype, data.view((1,) + mesh.shape))


def _vec(mesh, data):
    return shell.VectorQ1Vec(mesh, data.dtype, data)


def prepare(case, seed):
    _, f = _inputs(case, seed, "cuda")
    kind, level, r_min = case["kind"], case["level"], case["r_min"]
    dt = DTYPE[case.get("dtype", "f64")]
    m = shell.ShellMesh(level, r_min, 1.0)
    st = {"kind": kind, "mesh": m, "case": case}
    if "bc_cmb" in case:
        bc = BC[case["bc_cmb"]], BC[case["bc_surface"]]
    if kind == "viscous":
        st["op"] = shell.EpsilonDivDivKerngen(m, _scalar(m, f["k"]), *bc)
        st["src"], st["dst"] = _vec(m, f["u"]), shell.VectorQ1Vec(m, dt)
    elif kind == "viscous3x2":
        st["op"] = shell.EpsilonDivDiv(m, _scalar(m, f["k"]), case["treat"])
        st["src"], st["dst"] = _vec(m, f["u"]), shell.VectorQ1Vec(m, dt)
    elif kind == "poisson_cg":
        st["b"], st["x"] = _scalar(m, f["b"]), shell.VectorQ1Scalar(m)
    elif kind == "gradient_form":
        if case["op"] == "vector_laplace":
            b = BC["dirichlet" if case["treat"] else "neumann"]
            st["op"] = shell.VectorLaplace(m, b, b)
            st["src"], st["dst"] = _vec(m, f["u"]), shell.VectorQ1Vec(m, dt)
        else:
            st["op"] = (shell.Laplace(m, case["treat"]) if case["op"] == "laplace"
                        else shell.DivKGrad(m, _scalar(m, f["k"]), case["treat"]))
            st["src"], st["dst"] = _scalar(m, f["u"]), shell.VectorQ1Scalar(m, dt)
    elif kind == "stokes_blocks":
        mc = shell.ShellMesh(level - 1, r_min, 1.0)
        st["B"], st["BT"] = shell.Divergence(m, mc, *bc), shell.Gradient(m, mc, *bc)
        st["u"], st["p"] = _vec(m, f["u"]), _scalar(mc, f["p"])
        st["Bu"], st["BTp"] = shell.VectorQ1Scalar(mc, dt), shell.VectorQ1Vec(m, dt)
    elif kind == "viscosity_grad":
        st["bc"] = bc
        st["u"], st["lam"], st["out"] = _vec(m, f["u"]), _vec(m, f["lam"]), shell.VectorQ1Scalar(m, dt)
    elif kind == "energy_fct":
        st["fct"] = shell.FCTAdvectionDiffusion(m)
        st["bcs"] = st["fct"].dirichlet(1.0, 0.0)
        st["v"], st["T0"], st["T"] = _vec(m, f["v"]), f["T"], st["fct"].field()
        st["fct"].apply_dirichlet(st["T0"], st["bcs"])
    elif kind == "projection":
        st["fv"], st["T"] = f["T"], shell.VectorQ1Scalar(m)
        st["work"] = torch.empty(5 * m.stored_nodes, dtype=torch.float64, device="cuda")
    elif kind == "energy_supg":
        st["op"] = shell.UnsteadyAdvectionDiffusionSUPG(m, _vec(m, f["v"]), case["kappa"], _supg_dt(case),
                                                        case["treat"], lumped_mass=case["lumped"])
        st["src"], st["dst"] = _scalar(m, f["T"]), shell.VectorQ1Scalar(m, dt)
    elif kind == "stokes_solve":
        st["bc"], st["T"] = bc, _scalar(m, f["T"])
        st["eta"] = _scalar(m, f["k"])
        mp = shell.ShellMesh(level - 1, r_min, 1.0)
        st["fu"], st["fp"] = shell.VectorQ1Vec(m), shell.VectorQ1Scalar(mp)
        st["u"], st["p"] = shell.VectorQ1Vec(m), shell.VectorQ1Scalar(mp)
        st["work"] = torch.empty(3 * m.stored_nodes, dtype=torch.float64, device="cuda")
        st["solver"] = shell.StokesSolver(level, st["eta"], mg_levels=level - 2, bc_cmb=bc[0], bc_surface=bc[1],
                                          mg_fp32=True, chebyshev_order=2, smoothing_steps=2, restart=10,
                                          max_iterations=STOKES_ITERATIONS, relative_tolerance=1e-30, r_min=r_min,
                                          r_max=1.0, gca=1, chebyshev_estimates=[CHEBYSHEV_ESTIMATE] * (level - 2))
    return st


def run(st):
    kind = st["kind"]
    if kind in ("viscous", "viscous3x2", "gradient_form", "energy_supg"):
        shell.apply(st["op"], st["src"], st["dst"])
        return st["dst"].data
    if kind == "poisson_cg":
        st["x"].data.zero_()
        shell.laplace_pcg(st["mesh"], st["b"], st["x"], CG_ITERATIONS, 1e-30)
        return st["x"].data
    if kind == "stokes_blocks":
        shell.apply(st["B"], st["u"], st["Bu"])
        shell.apply(st["BT"], st["p"], st["BTp"])
        return {"divergence": st["Bu"].data, "gradient": st["BTp"].data}
    if kind == "viscosity_grad":
        shell.epsdivdiv_kgrad(st["mesh"], *st["bc"], st["u"], st["lam"], st["out"])
        return st["out"].data
    if kind == "energy_fct":
        fct, kappa = st["fct"], st["case"]["kappa"]
        st["T"].copy_(st["T0"])  # the step is in place: the next pass starts from the same temperature
        dt = CFL * fct.dt_stable(st["v"], kappa)
        fct.step(st["T"], st["v"], dt, kappa, None, True, st["bcs"])
        fct.apply_dirichlet(st["T"], st["bcs"])
        return {"T": st["T"], "dt": dt}
    if kind == "projection":
        st["T"].data.zero_()
        shell.l2_project_fv_to_fe(st["mesh"], st["fv"], st["T"], False, PROJECTION_ITERATIONS, 1e-30, 1e-30,
                                  work=st["work"])
        return st["T"].data
    shell.stokes_buoyancy_rhs(st["mesh"], st["T"], 1e5, *st["bc"], st["fu"], work=st["work"])
    st["u"].data.zero_()
    st["p"].data.zero_()
    st["solver"].solve(st["fu"], st["fp"], st["u"], st["p"])
    return {"u": st["u"].data, "p": st["p"].data}


def _supg_dt(case):
    return 0.5 / (1 << case["level"])


# --- necessary work and tolerances -----------------------------------------------------------------------------

def work(case):
    """inputs read once and outputs written once; operations of a factored evaluation of each wedge"""
    N = 1 << case["level"]
    ns, cells, s = 10 * (N + 1) ** 3, 10 * N ** 3, 4 if case.get("dtype") == "f32" else 8
    nc = 10 * (N // 2 + 1) ** 3
    kind = case["kind"]
    if kind == "viscous":
        return {"bytes": 7 * s * ns, "flops": 400 * cells}
    if kind == "viscous3x2":
        return {"bytes": 7 * s * ns, "flops": 1800 * cells}
    if kind == "poisson_cg":
        # an iteration reads and writes the direction, its image, the residual and the iterate
        return {"bytes": CG_ITERATIONS * 8 * s * ns, "flops": CG_ITERATIONS * 100 * ns}
    if kind == "gradient_form":
        n = {"laplace": 2, "vector_laplace": 6, "divkgrad": 3}[case["op"]]
        return {"bytes": n * s * ns, "flops": {"laplace": 80, "vector_laplace": 240, "divkgrad": 500}[case["op"]] * ns}
    if kind == "stokes_blocks":
        return {"bytes": 6 * s * ns + 2 * s * nc, "flops": 400 * cells}
    if kind == "viscosity_grad":
        return {"bytes": 7 * s * ns, "flops": 300 * cells}
    if kind == "energy_fct":
        # the velocity for the step size and again for the step, the temperature in and out
        return {"bytes": 48 * ns + 16 * cells, "flops": 300 * cells}
    if kind == "projection":
        return {"bytes": 8 * cells + 8 * ns + PROJECTION_ITERATIONS * 8 * s * ns,
                "flops": PROJECTION_ITERATIONS * 60 * ns}
    if kind == "energy_supg":
        return {"bytes": 5 * s * ns, "flops": 800 * cells}
    # per iteration: the FP64 operator and about twenty FP32 applies of the velocity block (smoothing on all levels)
    return {"bytes": STOKES_ITERATIONS * (20 * 28 + 56 + 100) * ns, "flops": STOKES_ITERATIONS * 20 * 400 * cells}


def tolerance(case):
    if case["kind"] == "stokes_solve":
        # rounding of the FP32 preconditioner travels through ten Krylov steps: two solver objects on the same
        # inputs, or a viscosity perturbed by 1e-7, move the iterate by up to 5e-6
        return {"rel": 3e-5}
    # seen against exact(): up to 1.4e-15 in FP64; in FP32 up to 7e-6 (differences of single-precision radii)
    return {"rel": 2e-14 if case.get("dtype", "f64") == "f64" else 3e-5}


# --- the same results in plain 64-bit torch --------------------------------------------------------------------

_GAUSS = 1.0 / math.sqrt(3.0)
_LATERAL3 = ((2.0 / 3.0, 1.0 / 6.0), (1.0 / 6.0, 2.0 / 3.0), (1.0 / 6.0, 1.0 / 6.0))


def _rule(six):
    """(xi, eta, zeta, weight) of the six-point rule or of the one-point rule"""
    if not six:
        return [(1.0 / 3.0, 1.0 / 3.0, 0.0, 1.0)]
    return [(xi, eta, z, 1.0 / 6.0) for z in (-_GAUSS, _GAUSS) for xi, eta in _LATERAL3]


def _wedge(geo, w, xi, eta, zeta):
    """shape functions, physical gradients [6] x [..., 3] and |det J| of the map
    x = r(zeta) (p0 + xi (p1 - p0) + eta (p2 - p0)) at one point of wedge w of every cell"""
    p0, p1, p2 = geo.lateral(w)
    a, b = p1 - p0, p2 - p0
    c = p0 + xi * a + eta * b
    r1, r2 = geo.r[:-1], geo.r[1:]
    h = 0.5 * (r2 - r1)
    r = r1 + h * (1.0 + zeta)
    v = torch.linalg.cross(a, b)
    D = (v * p0).sum(-1, keepdim=True)
    u1, u2 = torch.linalg.cross(b, c), torch.linalg.cross(c, a)
    u = (-(u1 + u2), u1, u2)
    lat = (1.0 - xi - eta, xi, eta)
    shp, grad = [], []
    for n in range(6):
        nr, s = 0.5 * (1.0 + (zeta if n > 2 else -zeta)), 0.5 if n > 2 else -0.5
        shp.append(lat[n % 3] * nr)
        grad.append((nr / r)[:, None] * (u[n % 3] / D) + (s * lat[n % 3] / h)[:, None] * (v / D))
    return shp, grad, (r * r * h) * D[..., 0].abs()


def _scatter(geo, out, w, n, val):
    dx, dy, dr = _node(w, n)
    N = geo.N
    out[:, dx:dx + N, dy:dy + N, dr:dr + N] += val


def _layers(geo, treat_bottom, treat_top):
    """per wedge node the cells (by radial index) whose node n is a boundary node"""
    N = geo.N
    none = torch.zeros(N, dtype=torch.bool, device=geo.device)
    bot, top = none.clone(), none.clone()
    bot[0], top[N - 1] = True, True
    return [(bot if treat_bottom else none) if n < 3 else (top if treat_top else none) for n in range(6)]


def _viscous_exact(geo, k, u, kind_cmb, kind_surface, six):
    """epsilon-div-div; kinds: natural, eliminated with kept diagonal (dirichlet) or tangential (freeslip)"""
    out = torch.zeros((3,) + geo.shape, dtype=torch.float64, device=geo.device)
    normal = geo.p / geo.p.norm(dim=-1, keepdim=True)
    for w in (0, 1):
        fixed = _layers(geo, kind_cmb == "dirichlet", kind_surface == "dirichlet")
        slip = _layers(geo, kind_cmb == "freeslip", kind_surface == "freeslip")
        kn = [geo.corner(k, w, n) for n in range(6)]
        un = [torch.stack([geo.corner(u[c], w, n) for c in range(3)], -1) for n in range(6)]
        nn = []
        for n in range(6):
            dx, dy, _ = _node(w, n)
            nn.append(normal[:, dx:dx + geo.N, dy:dy + geo.N, None, :])
        for xi, eta, zeta, wt in _rule(six):
            shp, g, det = _wedge(geo, w, xi, eta, zeta)
            kw = wt * det * (sum(s * v for s, v in zip(shp, kn)) if six else sum(kn) / 6.0)
            G = torch.zeros(kw.shape + (3, 3), dtype=torch.float64, device=geo.device)
            for n in range(6):
                t = un[n]
                t = torch.where(slip[n][:, None], t - (t * nn[n]).sum(-1, keepdim=True) * nn[n], t)
                t = torch.where(fixed[n][:, None], 0.0, t)
                G += g[n][..., :, None] * t[..., None, :]
            div = G.diagonal(dim1=-2, dim2=-1).sum(-1)
            S = G + G.transpose(-1, -2)
            for n in range(6):
                o = (S * g[n][..., :, None]).sum(-2) - (2.0 / 3.0) * div[..., None] * g[n]
                gg = (g[n] * g[n]).sum(-1, keepdim=True)
                ng = (nn[n] * g[n]).sum(-1, keepdim=True)
                o_slip = (o - (o * nn[n]).sum(-1, keepdim=True) * nn[n]
                          + (gg + ng * ng / 3.0) * (un[n] * nn[n]).sum(-1, keepdim=True) * nn[n])
                o = torch.where(slip[n][:, None], o_slip, o)
                o = torch.where(fixed[n][:, None], un[n] * (gg + g[n] * g[n] / 3.0), o)
                for c in range(3):
                    _scatter(geo, out[c], w, n, kw * o[..., c])
    if kind_cmb == kind_surface == "freeslip":
        # rigid rotations, orthonormal over the distinct nodes: they are added to every stored copy
        x = geo.position()
        own = geo.owned
        modes = [torch.linalg.cross(torch.eye(3, dtype=torch.float64, device=geo.device)[i].expand_as(x), x)
                 for i in range(3)]
        gram = torch.stack([torch.stack([(torch.where(own[..., None], a, 0.0) * b).sum() for b in modes])
                            for a in modes])
        uu = u.movedim(0, -1)
        rhs = torch.stack([(torch.where(own[..., None], a, 0.0) * uu).sum() for a in modes])
        for al, mode in zip(torch.linalg.solve(gram, rhs), modes):
            out += al * mode.movedim(-1, 0)
    return torch.stack([geo.halo(out[c]) for c in range(3)])


def _gradient_form_exact(geo, k, u, modes):
    """int k grad u . grad v; modes(): the decoupled nodes (kept diagonal) per wedge node and radial layer"""
    out = torch.zeros_like(u)
    for w in (0, 1):
        off = modes()
        kn = [geo.corner(k, w, n) for n in range(6)] if k is not None else None
        for xi, eta, zeta, wt in _rule(True):
            shp, g, det = _wedge(geo, w, xi, eta, zeta)
            kw = wt * det * (sum(s * v for s, v in zip(shp, kn)) if kn is not None else 1.0)
            for c in range(u.shape[0]):
                un = [geo.corner(u[c], w, n) for n in range(6)]
                G = sum(g[n] * torch.where(off[n], 0.0, un[n])[..., None] for n in range(6))
                for n in range(6):
                    gg = (g[n] * g[n]).sum(-1)
                    _scatter(geo, out[c], w, n, kw * torch.where(off[n], gg * un[n], (g[n] * G).sum(-1)))
    return torch.stack([geo.halo(o) for o in out])


def _cg(apply, geo, b, iterations):
    own = geo.owned.expand(geo.shape)
    dot = lambda p, q: float((torch.where(own, p, 0.0) * q).sum())  # noqa: E731
    x, r = torch.zeros_like(b), b.clone()
    p, rr = r.clone(), dot(r, r)
    for _ in range(iterations):
        q = apply(p)
        al = rr / dot(p, q)
        x += al * p
        r -= al * q
        new = dot(r, r)
        p = r + (new / rr) * p
        rr = new
    return x


# coarse lateral shape functions (constant, xi, eta) per vertex on the four fine triangles of a coarse one
_COARSE = (((1.0, -0.5, -0.5), (0.5, -0.5, -0.5), (0.5, -0.5, -0.5), (0.0, 0.5, 0.5)),
           ((0.0, 0.5, 0.0), (0.5, 0.5, 0.0), (0.0, 0.5, 0.0), (0.5, -0.5, 0.0)),
           ((0.0, 0.0, 0.5), (0.0, 0.0, 0.5), (0.5, 0.0, 0.5), (0.5, 0.0, -0.5)))


def _stokes_blocks_exact(geo, gc, u, p, kind_cmb, kind_surface):
    N, dev = geo.N, geo.device
    normal = geo.p / geo.p.norm(dim=-1, keepdim=True)
    ix = torch.arange(N, device=dev)
    Bu = torch.zeros(gc.shape, dtype=torch.float64, device=dev).view(-1)
    BTp = torch.zeros((3,) + geo.shape, dtype=torch.float64, device=dev)
    tab = torch.tensor(_COARSE, dtype=torch.float64, device=dev)
    d = torch.arange(10, device=dev).view(10, 1, 1, 1)
    for w in (0, 1):
        fixed = _layers(geo, kind_cmb == "dirichlet", kind_surface == "dirichlet")
        slip = _layers(geo, kind_cmb == "freeslip", kind_surface == "freeslip")
        quarter = (ix & 1)[None, :] * 2 + (ix & 1)[:, None]
        flat = quarter if w == 0 else 3 - quarter
        cidx = []
        for i in range(6):
            dx, dy, dr = _node(w, i)
            X, Y, R = (ix // 2 + dx).view(1, N, 1, 1), (ix // 2 + dy).view(1, 1, N, 1), (ix // 2 + dr).view(1, 1, 1, N)
            cidx.append((((d * gc.n1 + X) * gc.n1 + Y) * gc.n1 + R))
        pn = [p.reshape(-1)[c] for c in cidx]
        un, nn = [], []
        for n in range(6):
            dx, dy, _ = _node(w, n)
            nrm = normal[:, dx:dx + N, dy:dy + N, None, :]
            t = torch.stack([geo.corner(u[c], w, n) for c in range(3)], -1)
            t = torch.where(slip[n][:, None], t - (t * nrm).sum(-1, keepdim=True) * nrm, t)
            un.append(torch.where(fixed[n][:, None], 0.0, t))
            nn.append(nrm)
        for xi, eta, zeta, wt in _rule(True):
            _, g, det = _wedge(geo, w, xi, eta, zeta)
            div = sum((g[n] * un[n]).sum(-1) for n in range(6))
            lat = (tab[..., 0] + tab[..., 1] * xi + tab[..., 2] * eta)[:, flat]  # [3, N, N]
            top = 0.25 * (1.0 + zeta + 2.0 * (ix & 1).to(torch.float64))
            pq = 0.0
            for i in range(6):
                s = lat[i % 3][None, :, :, None] * (top if i > 2 else 1.0 - top)
                Bu.index_add_(0, cidx[i].reshape(-1), (-wt * det * s * div).expand(10, N, N, N).reshape(-1))
                pq = pq + s * pn[i]
            for n in range(6):
                o = (-wt * det * pq)[..., None] * g[n]
                o = torch.where(slip[n][:, None], o - (o * nn[n]).sum(-1, keepdim=True) * nn[n], o)
                o = torch.where(fixed[n][:, None], 0.0, o)
                for c in range(3):
                    _scatter(geo, BTp[c], w, n, o[..., c])
    return gc.halo(Bu.view(gc.shape)), torch.stack([geo.halo(BTp[c]) for c in range(3)])


def _viscosity_grad_exact(geo, u, lam, kind_cmb, kind_surface):
    out = torch.zeros(geo.shape, dtype=torch.float64, device=geo.device)
    normal = geo.p / geo.p.norm(dim=-1, keepdim=True)
    for w in (0, 1):
        fixed = _layers(geo, kind_cmb == "dirichlet", kind_surface == "dirichlet")
        slip = _layers(geo, kind_cmb == "freeslip", kind_surface == "freeslip")
        _, g, det = _wedge(geo, w, *_rule(False)[0][:3])
        G, bnd = [0.0, 0.0], 0.0
        for n in range(6):
            dx, dy, _ = _node(w, n)
            nrm = normal[:, dx:dx + geo.N, dy:dy + geo.N, None, :]
            a, b = (torch.stack([geo.corner(t[c], w, n) for c in range(3)], -1) for t in (u, lam))
            gg, ng = (g[n] * g[n]).sum(-1), (g[n] * nrm).sum(-1)
            an, bn = (a * nrm).sum(-1), (b * nrm).sum(-1)
            bnd = bnd + torch.where(fixed[n], (a * b * (gg[..., None] + g[n] * g[n] / 3.0)).sum(-1), 0.0)
            bnd = bnd + torch.where(slip[n], (gg + ng * ng / 3.0) * an * bn, 0.0)
            for i, (t, tn) in enumerate(((a, an), (b, bn))):
                t = torch.where(slip[n][:, None], t - tn[..., None] * nrm, t)
                t = torch.where(fixed[n][:, None], 0.0, t)
                G[i] = G[i] + g[n][..., :, None] * t[..., None, :]
        S = [x + x.transpose(-1, -2) for x in G]
        div = [x.diagonal(dim1=-2, dim2=-1).sum(-1) for x in G]
        cw = det * (0.5 * (S[0] * S[1]).sum((-1, -2)) - (2.0 / 3.0) * div[0] * div[1] + bnd) / 6.0
        for n in range(6):
            _scatter(geo, out, w, n, cw)
    return geo.halo(out)


def _fv_neighbours(geo):
    """flat index of the cell across each lateral face of the boundary cells of every diamond"""
    N, n2 = geo.N, geo.N + 2
    gid = geo.gid.view(10, geo.n1, geo.n1).cpu().numpy()
    t = np.arange(N)
    sides, faces = {}, []
    for d in range(10):
        for side in range(4):
            x, y = ((0, None), (N, None), (None, 0), (None, N))[side]
            a = gid[d][x if x is not None else t, y if y is not None else t]
            b = gid[d][x if x is not None else t + 1, y if y is not None else t + 1]
            gx = {0: 0, N: N + 1}[x] if x is not None else t + 1
            gy = {0: 0, N: N + 1}[y] if y is not None else t + 1
            cx = {0: 1, N: N}[x] if x is not None else t + 1
            cy = {0: 1, N: N}[y] if y is not None else t + 1
            ghost, cell = (d * n2 + gx) * n2 + gy, (d * n2 + cx) * n2 + cy
            faces.append((np.minimum(a, b), np.maximum(a, b), ghost + 0 * t, cell + 0 * t))
    lo, hi, ghost, cell = (np.concatenate(v) for v in zip(*faces))
    for i, e in enumerate(zip(lo, hi)):
        sides.setdefault(e, []).append(i)
    other = np.empty(len(lo), np.int64)
    for i, j in sides.values():
        other[i], other[j] = j, i
    return torch.as_tensor(ghost, device=geo.device), torch.as_tensor(cell[other], device=geo.device)


def _energy_fct_exact(geo, v, T, kappa):
    N, n2, dev = geo.N, geo.N + 2, geo.device
    ghost, across = _fv_neighbours(geo)
    inner = (slice(None),) + (slice(1, N + 1),) * 3

    def update(f):
        c = f.view(-1, n2)
        c[ghost, 1:-1] = c[across, 1:-1]

    def dirichlet(f):
        f[:, 1:-1, 1:-1, 0:2] = 1.0
        f[:, 1:-1, 1:-1, N:] = 0.0

    def shift(f, n):
        o = [1, 1, 1]
        o[n // 2] += -1 if n % 2 == 0 else 1
        return f[(slice(None),) + tuple(slice(i, i + N) for i in o)]

    r1, r2 = geo.r[:-1], geo.r[1:]
    h = 0.5 * (r2 - r1)
    gauss = [r1 + h * (1.0 + z) for z in (-_GAUSS, _GAUSS)]
    beta, S = [0.0] * 6, [0.0] * 6
    M, moment = 0.0, 0.0
    for w in (0, 1):
        p0, p1, p2 = geo.lateral(w)
        a, b = p1 - p0, p2 - p0
        un = [torch.stack([geo.corner(v[c], w, n) for c in range(3)], -1) for n in range(6)]
        face_x, face_y = (0, 2) if w == 0 else (1, 3)
        # the two lateral faces xi = 0 (nodes 0, 2) and eta = 0 (nodes 0, 1): 2 x 2 Gauss points
        for f, vec, m in ((face_x, torch.linalg.cross(b, p0), 2), (face_y, torch.linalg.cross(a, p0), 1)):
            for z, rq in zip((-_GAUSS, _GAUSS), gauss):
                nb, nt = 0.5 * (1 - z), 0.5 * (1 + z)
                nrm = (rq * h)[:, None] * vec
                uq = 0.5 * (nb * (un[0] + un[m]) + nt * (un[3] + un[3 + m]))
                beta[f] = beta[f] + (nrm * uq).sum(-1)
                S[f] = S[f] + nrm
        ab = torch.linalg.cross(a, b)
        for f, rq, ns in ((4, r1, (0, 1, 2)), (5, r2, (3, 4, 5))):
            nrm = 0.5 * (rq * rq)[:, None] * ab
            beta[f] = beta[f] + (nrm * sum(un[n] for n in ns) / 3.0).sum(-1)
            S[f] = S[f] + nrm
        D = (ab * p0).sum(-1).abs()
        for rq in gauss:
            M = M + 0.5 * h * D * rq * rq
            moment = moment + ((h * D * rq ** 3) / 6.0)[..., None] * (p0 + p1 + p2)
    centre = torch.zeros((3, 10, n2, n2, n2), dtype=torch.float64, device=dev)
    for c in range(3):
        centre[(c,) + inner] = moment[..., c] / M
        update(centre[c])
    c0 = torch.stack([centre[(c,) + inner] for c in range(3)], -1)
    for n in range(6):
        dc = torch.stack([shift(centre[c], n) for c in range(3)], -1) - c0
        flip = (S[n] * dc).sum(-1) < 0
        beta[n] = torch.where(flip, -beta[n], beta[n])
        S[n] = torch.where(flip[..., None], -S[n], S[n])
        S[n] = ((S[n] * S[n]).sum(-1), (dc * S[n]).sum(-1))  # |S|^2 and S . (c_j - c_i)
    lam = sum((-beta[n]).clamp(min=0.0) for n in range(6))
    if kappa > 0:
        lam = lam + sum(torch.where(S[n][1] > 0, kappa * S[n][0] / S[n][1], 0.0) for n in range(6))
    dt = CFL * float(torch.where(lam > 0, M / lam, 1e30).min())

    T = T.clone()
    dirichlet(T)
    update(T)
    Ti = T[inner]
    diag, upd, F = 0.0, 0.0, []
    for n in range(6):
        Tj = shift(T, n)
        diag = diag + beta[n].clamp(min=0.0) - beta[n]
        upd = upd + beta[n].clamp(max=0.0) * Tj
        if kappa != 0:
            dc = kappa * S[n][0] / S[n][1]
            diag, upd = diag + dc, upd - dc * Tj
        F.append((dt / M) * (beta[n].abs() / 2.0) * (Ti - Tj))
    TL, Rp, Rm = (torch.zeros_like(T) for _ in range(3))
    TL[inner] = Ti - (dt / M) * (diag * Ti + upd)
    dirichlet(TL)
    update(TL)
    ti = TL[inner]
    Pp, Pm = sum(f.clamp(min=0.0) for f in F), sum(f.clamp(max=0.0) for f in F)
    hi = functools.reduce(torch.maximum, [shift(TL, n) for n in range(6)], ti)
    lo = functools.reduce(torch.minimum, [shift(TL, n) for n in range(6)], ti)
    Rp[inner] = torch.where(Pp > 0, ((hi - ti) / Pp).clamp(max=1.0), 1.0)
    Rm[inner] = torch.where(Pm < 0, ((lo - ti) / Pm).clamp(max=1.0), 1.0)
    update(Rp)
    update(Rm)
    corr = sum(torch.where(F[n] > 0, torch.minimum(Rp[inner], shift(Rm, n)),
                           torch.minimum(Rm[inner], shift(Rp, n))) * F[n] for n in range(6))
    T[inner] = ti + corr
    dirichlet(T)
    return T, dt


def _projection_exact(geo, T):
    N = geo.N
    b = torch.zeros(geo.shape, dtype=torch.float64, device=geo.device)
    cell = T[:, 1:N + 1, 1:N + 1, 1:N + 1]
    points = [(w, _wedge(geo, w, *q[:3]), q[3]) for w in (0, 1) for q in _rule(True)]
    for w, (shp, _, det), wt in points:
        for n in range(6):
            _scatter(geo, b, w, n, wt * det * shp[n] * cell)

    def mass(x):
        out = torch.zeros_like(x)
        for w, (shp, _, det), wt in points:
            xq = sum(shp[n] * geo.corner(x, w, n) for n in range(6))
            for n in range(6):
                _scatter(geo, out, w, n, wt * det * shp[n] * xq)
        return geo.halo(out)

    return _cg(mass, geo, geo.halo(b), PROJECTION_ITERATIONS)


def _energy_supg_exact(geo, v, T, kappa, dt, treat, lumped):
    out = torch.zeros(geo.shape, dtype=torch.float64, device=geo.device)
    h = geo.r[1:] - geo.r[:-1]
    kv = max(kappa, 1e-8)
    for w in (0, 1):
        fixed = _layers(geo, treat, treat)
        vn = [torch.stack([geo.corner(v[c], w, n) for c in range(3)], -1) for n in range(6)]
        tn = [geo.corner(T, w, n) for n in range(6)]
        tm = [torch.where(fixed[n], 0.0, tn[n]) for n in range(6)]
        points = [(_wedge(geo, w, *q[:3]), q[3]) for q in _rule(True)]
        vel = [sum(s * x for s, x in zip(shp, vn)) for (shp, _, _), _ in points]
        tau = 0.0
        for x in vel:
            nv = x.norm(dim=-1)
            pe = nv * h / (2.0 * kv)
            t = torch.minimum(h / (2.0 * nv) * (1.0 / torch.tanh(pe) - 1.0 / pe), 10.0 * h / nv.clamp(min=1e-12))
            tau = tau + torch.where((nv > 1e-12) & (pe > 1e-8), t, 0.0) / 6.0
        for ((shp, g, det), wt), x in zip(points, vel):
            sq = sum(shp[n] * tm[n] for n in range(6))
            gs = sum(g[n] * tm[n][..., None] for n in range(6))
            ugs = (x * gs).sum(-1)
            for n in range(6):
                ugn, gg = (x * g[n]).sum(-1), (g[n] * g[n]).sum(-1)
                row = (shp[n] * (tm[n] if lumped else sq)
                       + dt * (kappa * (g[n] * gs).sum(-1) + shp[n] * ugs + tau * ugn * ugs))
                own = (shp[n] * (1.0 if lumped else shp[n])
                       + dt * (kappa * gg + shp[n] * ugn + tau * ugn * ugn)) * tn[n]
                _scatter(geo, out, w, n, wt * det * torch.where(fixed[n], own, row))
    return geo.halo(out)


def exact(case, seed, device="cuda"):
    kind = case["kind"]
    if kind == "stokes_solve":  # an unconverged Krylov iterate with an FP32 preconditioner
        return None
    geo, f = _inputs(case, seed, device)
    f = {n: t.double() for n, t in f.items()}
    if kind == "viscous":
        return _viscous_exact(geo, f["k"], f["u"], case["bc_cmb"], case["bc_surface"], False)
    if kind == "viscous3x2":
        bc = "dirichlet" if case["treat"] else "neumann"
        return _viscous_exact(geo, f["k"], f["u"], bc, bc, True)
    if kind == "poisson_cg":
        modes = lambda: _layers(geo, True, True)  # noqa: E731
        return _cg(lambda x: _gradient_form_exact(geo, None, x[None], modes)[0], geo, f["b"], CG_ITERATIONS)[None]
    if kind == "gradient_form":
        def modes():
            off = _layers(geo, case["treat"], case["treat"])
            if case["op"] == "vector_laplace" and case["treat"]:
                # a Dirichlet surface decouples the upper nodes of every cell above the lowest layer
                up = torch.ones_like(off[3])
                up[0] = False
                off = off[:3] + [up] * 3
            return off
        return _gradient_form_exact(geo, f.get("k"), f["u"], modes)
    if kind == "stokes_blocks":
        gc = _Geo(case["level"] - 1, case["r_min"], device)
        Bu, BTp = _stokes_blocks_exact(geo, gc, f["u"], f["p"], case["bc_cmb"], case["bc_surface"])
        return {"divergence": Bu[None], "gradient": BTp}
    if kind == "viscosity_grad":
        return _viscosity_grad_exact(geo, f["u"], f["lam"], case["bc_cmb"], case["bc_surface"])[None]
    if kind == "energy_fct":
        T, dt = _energy_fct_exact(geo, f["v"], f["T"], case["kappa"])
        return {"T": T, "dt": dt}
    if kind == "projection":
        return _projection_exact(geo, f["T"])[None]
    return _energy_supg_exact(geo, f["v"], f["T"], case["kappa"], _supg_dt(case), case["treat"], case["lumped"])[None]
