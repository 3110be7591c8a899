"""Timed cases of the edge assembly + Krylov library, through its Python entry points.

listed() names twelve pieces of the work an implicit low-Mach step does;
draw() gives more of the same ranges. A case is a box of nx x ny x nz hex
cells (or six tetrahedra per cell), with the fields of the benchmark
workloads: a log-law velocity with 5 % noise, eddy viscosity log-uniform in
[1e-5, 1e-2], nodes jittered by a few per cent of the cell size, z stretched
from the wall. Meshes and fields are made here with torch on the GPU from the
seed, in FP64, so that they do not depend on the library. exact() restates
each entry point's formulas in plain FP64 torch.
"""
from __future__ import annotations

import importlib.util
import itertools
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parent.parent
F8 = torch.float64


def _package():
    """The library's Python package (its directory name is not an identifier)."""
    if "nalu_wind_gb300" not in sys.modules:
        pkg = ROOT / "nalu-wind_gb300"
        spec = importlib.util.spec_from_file_location("nalu_wind_gb300", pkg / "__init__.py",
                                                      submodule_search_locations=[str(pkg)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["nalu_wind_gb300"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["nalu_wind_gb300"]


# ---------------------------------------------------------------------------
# cases

def listed():
    return [
        # the smallest whole step (test-size box): momentum and continuity
        # assembled with their time term, wall and open boundary; launches and
        # host calls count more than the kernels
        dict(name="step_24x20x12", kind="step", nx=24, ny=20, nz=12),
        # scalar transport on the 32^3 periodic block: assembly + Dirichlet rows
        dict(name="scalar_32cube", kind="scalar", nx=32, ny=32, nz=32, periodic=True, limiter=False, tanh=False),
        # scalar transport (enthalpy, turbulence quantities) on a mid-size
        # box, limiter and tanh Peclet function on
        dict(name="scalar_limited", kind="scalar", nx=97, ny=80, nz=59, periodic=False, limiter=True, tanh=True),
        # the assembly workload of the benchmark, its two systems
        dict(name="momentum_box", kind="momentum", nx=128, ny=128, nz=64, tets=False, order="rows", limiter=False,
             divu=False),
        dict(name="continuity_box", kind="continuity", nx=128, ny=128, nz=64, tets=False, order="rows",
             general=False),
        # unstructured, randomly numbered tets with every momentum option on
        dict(name="momentum_tets", kind="momentum", nx=53, ny=47, nz=41, tets=True, order="random", limiter=True,
             divu=True),
        # input producers (mass flow, velocity and pressure gradients, Peclet
        # factor) of every nonlinear iteration, on tets
        dict(name="producers_tets", kind="producers", nx=63, ny=55, nz=47, tets=True, order="rows"),
        # geometry update after mesh motion
        dict(name="geometry_hex", kind="geometry", nx=96, ny=90, nz=45, tets=False),
        # the plain solver at its smallest: GMRES(50) + Jacobi to 1e-8 on the
        # 32^3 scalar system
        dict(name="solve_scalar", kind="solve_scalar", nx=32, ny=32, nz=32, precond="jacobi", tol=1e-8, iters=500),
        # a momentum solve as an input file asks for it: GMRES(50), multicolour
        # symmetric Gauss-Seidel, 1e-5
        dict(name="solve_momentum", kind="solve_momentum", nx=47, ny=40, nz=33, precond="mt_sgs", tol=1e-5, iters=50),
        # a pressure solve with the default configuration (50 iterations of
        # GMRES(50) + Jacobi), 1.08 M rows
        dict(name="solve_poisson", kind="solve_poisson", nx=128, ny=128, nz=64, learned=False, tol=1e-4, iters=50),
        # a pressure solve to 1e-8 with the learned preconditioner in mixed
        # precision
        dict(name="solve_learned", kind="solve_poisson", nx=80, ny=80, nz=48, learned=True, tol=1e-8, iters=3000),
    ]


def _shape(rng, lo, hi):
    """A box of about lo..hi cells (log-uniform), ragged sides."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    a, b = rng.uniform(0.6, 1.6), rng.uniform(0.6, 1.6)
    side = (n / (a * b)) ** (1.0 / 3.0)
    nx, ny = max(4, int(side * a)), max(4, int(side * b))
    return dict(nx=nx, ny=ny, nz=max(4, int(n / (nx * ny))))


def draw(rng):
    kind = rng.choice(["step", "scalar", "momentum", "continuity", "producers", "geometry", "solve_scalar",
                       "solve_momentum", "solve_poisson"])
    flag = lambda: rng.random() < 0.5  # noqa: E731
    if kind == "step":
        return dict(kind=kind, **_shape(rng, 2e3, 4e5))
    if kind == "scalar":
        return dict(kind=kind, **_shape(rng, 4e3, 9e5), periodic=flag(), limiter=flag(), tanh=flag())
    tets = flag()
    if kind in ("momentum", "continuity", "producers"):
        c = dict(kind=kind, **_shape(rng, 2e3, 2e5 if tets else 1e6), tets=tets,
                 order=rng.choice(["rows", "rows", "random"]))
        if kind == "momentum":
            c.update(limiter=flag(), divu=flag())
        if kind == "continuity":
            c.update(general=rng.random() < 0.3)
        return c
    if kind == "geometry":
        return dict(kind=kind, **_shape(rng, 4e3, 1.5e5 if tets else 4e5), tets=tets)
    if kind == "solve_scalar":
        return dict(kind=kind, **_shape(rng, 4e3, 2e5), precond=rng.choice(["jacobi", "mt_sgs", "sgs"]),
                    tol=rng.choice([1e-5, 1e-6, 1e-8]), iters=200)
    if kind == "solve_momentum":
        return dict(kind=kind, **_shape(rng, 2e3, 1.2e5), precond=rng.choice(["mt_sgs", "jacobi", "sgs"]),
                    tol=rng.choice([1e-5, 1e-6]), iters=50)
    learned = flag()
    return dict(kind=kind, **_shape(rng, 2e4, 2.5e5 if learned else 9e5), learned=learned,
                tol=1e-8 if learned else 1e-4, iters=3000 if learned else 50)


# ---------------------------------------------------------------------------
# meshes: lattice nodes, edges, fields

def _mesh(c, gen):
    """Box of the case: coords (N, 3), edges (E, 2), edge areas, numbering."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    dev = "cuda"
    h = 1.0 / max(nx, ny)
    xs = torch.arange(nx + 1, dtype=F8, device=dev) * h
    ys = torch.arange(ny + 1, dtype=F8, device=dev) * h
    periodic = bool(c.get("periodic"))
    stretch = 1.0 if periodic else 1.03
    dz = h * 0.6 * torch.pow(torch.full((nz,), stretch, dtype=F8, device=dev),
                             torch.arange(nz, dtype=F8, device=dev))
    zs = torch.cat([torch.zeros(1, dtype=F8, device=dev), torch.cumsum(dz, 0)])
    K, J, I = torch.meshgrid(torch.arange(nz + 1, device=dev), torch.arange(ny + 1, device=dev),
                             torch.arange(nx + 1, device=dev), indexing="ij")
    I, J, K = I.reshape(-1), J.reshape(-1), K.reshape(-1)
    N = I.numel()
    x = torch.stack([xs[I], ys[J], zs[K]], 1)
    local = torch.stack([torch.full_like(x[:, 0], h), torch.full_like(x[:, 0], h),
                         torch.cat([dz, dz[-1:]])[K]], 1)
    if not periodic:
        inner = ((I > 0) & (I < nx) & (J > 0) & (J < ny) & (K > 0) & (K < nz)).to(F8)[:, None]
        x = x + 0.05 * local * inner * (torch.rand(N, 3, dtype=F8, device=dev, generator=gen) * 2 - 1)
    sx, sy, sz = 1, nx + 1, (nx + 1) * (ny + 1)
    node = torch.arange(N, device=dev)
    steps = [(1, 0, 0), (0, 1, 0), (0, 0, 1)]
    if c.get("tets"):
        steps += [(1, 1, 0), (1, 0, 1), (0, 1, 1), (1, 1, 1)]
    L, R, T = [], [], []
    for t, (a, b, d) in enumerate(steps):
        ok = (I + a <= nx) & (J + b <= ny) & (K + d <= nz)
        if periodic:  # the edges of the seam are listed once, from the master side
            ok = ok & (I < nx) & (J < ny)
        L.append(node[ok])
        R.append(node[ok] + a * sx + b * sy + d * sz)
        T.append(torch.full((int(ok.sum()),), t, device=dev))
    L, R, T = torch.cat(L), torch.cat(R), torch.cat(T)
    dual = local.prod(1)
    new = node
    if c.get("order") == "random":
        g7 = torch.Generator(device="cpu").manual_seed(7)
        new = torch.randperm(N, generator=g7).to(dev)  # old -> new
    order = torch.empty_like(new)
    order[new] = node  # new -> old
    x, I, J, K, dual = x[order], I[order], J[order], K[order], dual[order]
    L, R = new[L], new[R]
    L, R = torch.minimum(L, R), torch.maximum(L, R)
    s = torch.argsort(L * N + R)
    L, R, T = L[s], R[s], T[s]
    dx = x[R] - x[L]
    ln = dx.norm(dim=1, keepdim=True)
    # dual face of an edge: dual volume over edge length, a third of it per
    # edge family on tets, tilted by a few per cent
    a = 0.5 * (dual[L] + dual[R])[:, None] / ln * (0.4 if c.get("tets") else 1.0)
    area = a * (dx / ln + 0.04 * torch.randn(L.numel(), 3, dtype=F8, device=dev, generator=gen))
    nalu = node
    if periodic:
        nalu = (I % nx) * sx + (J % ny) * sy + K * sz
    return dict(N=N, E=L.numel(), x=x, L=L, R=R, area=area, dual=dual, I=I, J=J, K=K, master=nalu, new=new,
                shape=(nx, ny, nz), periodic=periodic, zs=zs)


def _lattice_gradient(m, f):
    """Central differences of f (N, k) on the unjittered lattice: (N, k, 3)."""
    nx, ny, nz = m["shape"]
    old = f[m["new"]].reshape(nz + 1, ny + 1, nx + 1, -1)
    h = 1.0 / max(nx, ny)
    z = m["zs"][:, None, None, None]
    out = []
    for dim, step in ((2, h), (1, h), (0, None)):
        up = torch.cat([old.narrow(dim, 1, old.shape[dim] - 1), old.narrow(dim, old.shape[dim] - 1, 1)], dim)
        dn = torch.cat([old.narrow(dim, 0, 1), old.narrow(dim, 0, old.shape[dim] - 1)], dim)
        if step is None:
            zu = torch.cat([z[1:], z[-1:]], 0)
            zd = torch.cat([z[:1], z[:-1]], 0)
            out.append((up - dn) / (zu - zd))
        else:
            out.append((up - dn) / (2 * step))
    g = torch.stack(out, -1).reshape(m["N"], -1, 3)
    res = torch.empty_like(g)
    res[m["new"]] = g
    return res


def _fields(c, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    m = _mesh(c, gen)
    N, L, R, x = m["N"], m["L"], m["R"], m["x"]
    rnd = lambda *s: torch.rand(*s, dtype=F8, device="cuda", generator=gen)  # noqa: E731
    nrm = lambda *s: torch.randn(*s, dtype=F8, device="cuda", generator=gen)  # noqa: E731
    vel = 0.05 * nrm(N, 3)
    zmax = float(x[:, 2].max())
    vel[:, 0] += torch.log1p(x[:, 2] / 1e-3) / math.log1p(zmax / 1e-3)
    f = dict(m, vel=vel, visc=torch.exp(math.log(1e-5) + rnd(N) * math.log(1e3)), rho=1.0 + 0.05 * (rnd(N) - 0.5),
             udiag=0.8 + 0.4 * rnd(N), p=0.01 * nrm(N), q=rnd(N), mask=torch.ones(N, dtype=F8, device="cuda"),
             bc=rnd(N, 3), pbc=0.01 * nrm(N))
    # wall velocity close to the nodes' own, as after the first iteration
    f["ubc"] = f["vel"] + 1e-3 * nrm(N, 3)
    if m["periodic"]:
        for k in ("vel", "visc", "rho", "udiag", "p", "q", "bc", "pbc"):
            f[k] = f[k][m["master"]].contiguous()
    f["dudx"] = _lattice_gradient(m, f["vel"]).reshape(N, 9).contiguous()
    f["dpdx"] = _lattice_gradient(m, f["p"][:, None]).reshape(N, 3).contiguous()
    f["dqdx"] = _lattice_gradient(m, f["q"][:, None]).reshape(N, 3).contiguous()
    if m["periodic"]:
        f["dqdx"] = f["dqdx"][m["master"]].contiguous()
    rho, A = f["rho"], f["area"]
    f["mdot"] = (0.5 * (rho[L, None] * f["vel"][L] + rho[R, None] * f["vel"][R]) * A).sum(1)
    diff = 0.5 * (f["visc"][L] / rho[L] + f["visc"][R] / rho[R])
    pe = (0.5 * (x[R] - x[L]) * (f["vel"][R] + f["vel"][L])).sum(1).abs() / (diff + 1e-16)
    f["pec"] = pe * pe / (5.0 + pe * pe)
    f["qold"] = (f["vel"] + 0.01 * nrm(N, 3)).contiguous()
    # the open side x+: four IPs per boundary quad (face node, node opposite)
    nx, ny, nz = m["shape"]
    dev = x.device
    j, k = torch.meshgrid(torch.arange(ny, device=dev), torch.arange(nz, device=dev), indexing="ij")
    j, k = j.reshape(-1), k.reshape(-1)
    corner = lambda i, a, b: m["new"][i + (nx + 1) * ((j + a) + (ny + 1) * (k + b))]  # noqa: E731
    ab = ((0, 0), (1, 0), (1, 1), (0, 1))
    f["ipR"] = torch.stack([corner(nx, a, b) for a, b in ab], 1).reshape(-1)
    f["ipL"] = torch.stack([corner(nx - 1, a, b) for a, b in ab], 1).reshape(-1)
    quad = (m["zs"][1:] - m["zs"][:-1])[k] / max(nx, ny) / 4.0
    n_ip = f["ipR"].numel()
    f["ipA"] = (quad.repeat_interleave(4)[:, None]
                * (torch.tensor([1.0, 0.0, 0.0], dtype=F8, device=dev) + 0.02 * nrm(n_ip, 3))).contiguous()
    f["wall"] = torch.nonzero(m["K"] == 0)[:, 0].contiguous()
    f["ends"] = torch.nonzero((m["K"] == 0) | (m["K"] == nz))[:, 0].contiguous()
    for key in ("x", "area", "mdot", "pec"):
        f[key] = f[key].contiguous()
    return f


def _elements(c):
    """Element connectivity over lattice nodes (Hex8 Exodus order or Tet4)."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    k, j, i = torch.meshgrid(torch.arange(nz), torch.arange(ny), torch.arange(nx), indexing="ij")
    at = lambda a, b, d: ((i + a) + (nx + 1) * ((j + b) + (ny + 1) * (k + d))).reshape(-1)  # noqa: E731
    if not c.get("tets"):
        return torch.stack([at(*v) for v in ((0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1),
                                             (1, 1, 1), (0, 1, 1))], 1)
    tets = []
    for p in itertools.permutations(range(3)):
        v = [[0, 0, 0]]
        for axis in p:
            w = list(v[-1])
            w[axis] = 1
            v.append(w)
        odd = sum(p[a] > p[b] for a in range(3) for b in range(a + 1, 3)) % 2
        if odd:
            v[1], v[2] = v[2], v[1]
        tets.append(torch.stack([at(*w) for w in v], 1))
    return torch.stack(tets, 1).reshape(-1, 4)


# ---------------------------------------------------------------------------
# options (the library's defaults where a case does not switch them)

def _scalar_opts(c):
    return dict(alpha=0.0, alpha_upw=0.5 if c.get("periodic") else 1.0, upw_factor=1.0, relax=1.0 if c.get("periodic") else 0.7,
                hybrid_factor=1.0, use_limiter=int(c.get("limiter", False)), tanh_form=int(c.get("tanh", False)),
                tanh_trans=2.0, tanh_width=4.0)


def _momentum_opts(c):
    return dict(alpha=0.0, alpha_upw=1.0, upw_factor=1.0, relax=0.7 if c.get("divu") else 1.0,
                include_div_u=float(c.get("divu", False)), use_limiter=int(c.get("limiter", False)))


def _continuity_opts(c):
    g = bool(c.get("general"))
    return dict(noc_fac=1.0, tau_scale=0.05, interp_together=0.0 if g else 1.0, solve_incompressible=1.0 if g else 0.0)


_OPEN = dict(tau_scale=0.05, noc_fac=1.0, pstab_fac=1.0, mdot_corr=0.0, solve_incompressible=0.0)
_DT, _GAMMA = 0.05, (1.5, -2.0, 0.5)


# ---------------------------------------------------------------------------
# state and passes

class _Device:
    """A device array owned by a library handle, as torch reads it; a tensor
    made from it keeps this object, and so the handle, alive."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=(n,), typestr="<f8", data=(ptr, False), version=3)


class _State:
    pass


def _system(nw, f, dof, cfg=None):
    ls = nw.LinearSystem(dof, cfg)
    edges = torch.stack([f["L"], f["R"]], 1).cpu().numpy()
    nid = (f["master"] + 1).cpu().numpy() if f["periodic"] else None
    ls.build_edge_graph(f["N"], edges, None if nid is None else np.arange(1, f["N"] + 1), nid)
    ls.finalize()
    nr, nz = ls.sizes()
    v, b, _, _ = ls.device_arrays()
    out = dict(values=torch.as_tensor(_Device(ls, v, nz), device="cuda"),
               rhs=torch.as_tensor(_Device(ls, b, nr), device="cuda"))
    return ls, out


def _ptrs(f, *names):
    return [f[k].data_ptr() for k in names]


def _assembly_args(nw, c, f):
    return dict(
        scalar=(nw.ScalarFields(*_ptrs(f, "x", "vel", "q", "dqdx", "rho", "visc", "area", "mdot")),
                nw.ScalarOpts(**_scalar_opts(c))),
        momentum=(nw.MomentumFields(*_ptrs(f, "x", "vel", "dudx", "visc", "rho", "mask", "area", "mdot", "pec")),
                  nw.MomentumOpts(**_momentum_opts(c))),
        continuity=(nw.ContinuityFields(*_ptrs(f, "x", "vel", "dpdx", "rho", "p", "udiag", "area")),
                    nw.ContinuityOpts(**_continuity_opts(c))),
        open=(nw.ContinuityOpenFields(*_ptrs(f, "x", "vel", "dpdx", "rho", "p", "pbc", "udiag", "ipA"), None),
              nw.ContinuityOpenOpts(**_OPEN)))


def _mass(ls, f):
    ls.assemble_mass_bdf("momentum", (f["rho"],) * 3, (f["dual"],) * 3, (f["qold"], f["qold"], f["vel"]), f["dpdx"],
                         dt=_DT, gamma=_GAMMA)


def _ip_nodes(f):
    return torch.stack([f["ipR"], f["ipL"]], 1).cpu().numpy()


def prepare(case, seed):
    nw = _package()
    c, kind = case, case["kind"]
    s = _State()
    s.nw, s.case = nw, c
    f = s.f = _fields(c, seed)
    s.args = _assembly_args(nw, c, f)
    if kind == "geometry":
        s.geo = nw.Geometry(f["N"], _elements(c).numpy(), torch.stack([f["L"], f["R"]], 1).cpu().numpy())
        s.area, s.vol = torch.zeros_like(f["area"]), torch.zeros_like(f["dual"])
    elif kind == "step":
        s.mom, s.mom_out = _system(nw, f, 3)
        s.con, s.con_out = _system(nw, f, 1)
        s.side = s.con.sideset(_ip_nodes(f))
        s.udiag = torch.zeros(f["N"], dtype=F8, device="cuda")
    elif kind == "producers":
        s.ls, _ = _system(nw, f, 1)
        s.out = dict(mdot=torch.zeros(f["E"], dtype=F8, device="cuda"),
                     dudx=torch.zeros(f["N"], 9, dtype=F8, device="cuda"),
                     dpdx=torch.zeros(f["N"], 3, dtype=F8, device="cuda"),
                     pecfac=torch.zeros(f["E"], dtype=F8, device="cuda"))
    elif kind in ("scalar", "momentum", "continuity"):
        s.ls, s.out = _system(nw, f, 3 if kind == "momentum" else 1)
    else:
        _prepare_solve(s)
    return s


def _prepare_solve(s):
    nw, c, f = s.nw, s.case, s.f
    if c["kind"] == "solve_poisson":
        if c["learned"]:
            cfg = nw.solver_cfg(method=nw.FGMRES, preconditioner=nw.PC_LEARNED, precision=nw.PREC_MIXED_BF16, kspace=30,
                                inner_kspace=30, max_iterations=c["iters"], tolerance=c["tol"])
        else:
            cfg = nw.solver_cfg(max_iterations=c["iters"], tolerance=c["tol"])
        s.ls, s.sys = _system(nw, f, 1, cfg)
        s.ls.zero_system()
        s.ls.assemble_continuity(*s.args["continuity"])
        s.side = s.ls.sideset(_ip_nodes(f))
        s.ls.assemble_continuity_open(s.side, *s.args["open"])
        if c["learned"]:
            s.net = nw.Learned()
            s.net.load(ROOT / "nalu-wind_gb300" / "weights" / "poisson_128cube.nwl")
            s.ls.attach_learned(s.net)
    else:
        momentum = c["kind"] == "solve_momentum"
        cfg = nw.solver_cfg_from_strings("gmres", c["precond"], kspace=50, max_iterations=c["iters"],
                                         tolerance=c["tol"])
        s.ls, s.sys = _system(nw, f, 3 if momentum else 1, cfg)
        s.ls.zero_system()
        if momentum:
            s.ls.assemble_momentum(*s.args["momentum"])
            _mass(s.ls, f)
            s.ls.apply_dirichlet(f["wall"].numel(), f["wall"], 0, 3, f["vel"], f["ubc"])
        else:
            s.ls.assemble_scalar(*s.args["scalar"])
            s.ls.apply_dirichlet(f["ends"].numel(), f["ends"], 0, 1, f["q"], f["bc"][:, 0].contiguous())
    s.x = torch.zeros(s.ls.sizes()[0], dtype=F8, device="cuda")
    s.ls.sync()


def run(s):
    c, f, kind = s.case, s.f, s.case["kind"]
    if kind == "scalar":
        s.ls.zero_system()
        s.ls.assemble_scalar(*s.args["scalar"])
        s.ls.apply_dirichlet(f["ends"].numel(), f["ends"], 0, 1, f["q"], f["pbc"])
        return s.out
    if kind == "momentum":
        s.ls.zero_system()
        s.ls.assemble_momentum(*s.args["momentum"])
        return s.out
    if kind == "continuity":
        s.ls.zero_system()
        s.ls.assemble_continuity(*s.args["continuity"])
        return s.out
    if kind == "producers":
        o = s.out
        s.ls.compute_mdot(s.args["continuity"][0], o["mdot"])
        s.ls.nodal_gradient(f["vel"], f["area"], f["dual"], o["dudx"], dim1=3)
        s.ls.nodal_gradient(f["p"], f["area"], f["dual"], o["dpdx"])
        s.ls.peclet_factor(f["x"], f["rho"], f["visc"], f["vel"], o["pecfac"])
        return o
    if kind == "geometry":
        s.geo.compute(f["x"], s.area, s.vol)
        return dict(area=s.area, volume=s.vol)
    if kind == "step":
        s.mom.zero_system()
        s.mom.assemble_momentum(*s.args["momentum"])
        _mass(s.mom, f)
        s.mom.extract_diagonal(s.udiag)
        s.mom.udiag_postprocess(f["rho"], f["dual"], s.udiag, _DT, _GAMMA[0], 0.7)
        s.mom.apply_dirichlet(f["wall"].numel(), f["wall"], 0, 3, f["vel"], f["ubc"])
        s.con.zero_system()
        s.con.assemble_continuity(*s.args["continuity"])
        s.con.assemble_continuity_open(s.side, *s.args["open"])
        return dict(momentum=s.mom_out, continuity=s.con_out, udiag=s.udiag)
    s.ls.solve(s.x)
    return s.x


# ---------------------------------------------------------------------------
# what a pass cannot do without

def _counts(c):
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    N = (nx + 1) * (ny + 1) * (nz + 1)
    E = nx * (ny + 1) * (nz + 1) + (nx + 1) * ny * (nz + 1) + (nx + 1) * (ny + 1) * nz
    if c.get("tets"):
        E += nx * ny * (nz + 1) + nx * (ny + 1) * nz + (nx + 1) * ny * nz + nx * ny * nz
    return N, E, N + 2 * E


def work(case):
    """Node inputs of each kind, edge inputs with 32-bit node pairs, the
    matrix and rhs written once (solves: read once); flops of the formulas."""
    c, kind = case, case["kind"]
    N, E, nnz = _counts(c)
    scalar = dict(bytes=40 * E + 96 * N + 8 * nnz + 8 * N, flops=150 * E)
    mom = dict(bytes=48 * E + 144 * N + 72 * nnz + 24 * N, flops=420 * E)
    con = dict(bytes=32 * E + 96 * N + 8 * nnz + 8 * N, flops=90 * E)
    if kind == "step":
        return dict(bytes=mom["bytes"] + con["bytes"] + 150 * N, flops=mom["flops"] + con["flops"])
    if kind in ("scalar", "momentum", "continuity"):
        return dict(scalar=scalar, momentum=mom, continuity=con)[kind]
    if kind == "producers":
        return dict(bytes=(8 + 24 + 16) * E + (24 + 24 + 24 + 8 * 5 + 96) * N, flops=250 * E)
    if kind == "geometry":
        M = c["nx"] * c["ny"] * c["nz"] * (6 if c["tets"] else 1)
        npe, ops = (4, 120) if c["tets"] else (8, 900)
        return dict(bytes=4 * npe * M + 24 * N + 24 * E + 8 * N, flops=ops * M)
    d = 3 if kind == "solve_momentum" else 1
    return dict(bytes=d * d * 12 * nnz + 16 * d * N, flops=2 * d * d * nnz)


# ---------------------------------------------------------------------------
# the same results in plain FP64 torch

def _rcp_limiter(m, p):
    return 2.0 * (m * p + (m * p).abs()) / ((m + p) ** 2 + 1e-16)


class _Pattern:
    """Node-level CSR pattern and sums into it, laid out as the library's."""

    def __init__(self, f, dof):
        self.d = dof
        master = f["master"]
        uniq = torch.unique(master)
        row = torch.empty_like(master)
        row[uniq] = torch.arange(uniq.numel(), device=row.device)
        self.row = row[master]
        n = self.n = uniq.numel()
        L, R = self.row[f["L"]], self.row[f["R"]]
        self.L, self.R = L, R
        i = torch.arange(n, device=L.device)
        self.keys = torch.unique(torch.cat([L * n + R, R * n + L, i * n + i]))
        self.v = torch.zeros(self.keys.numel(), dof, dof, dtype=F8, device=L.device)
        self.b = torch.zeros(n, dof, dtype=F8, device=L.device)

    def add(self, r, c, block):
        self.v.index_add_(0, torch.searchsorted(self.keys, r * self.n + c), block)

    def add_edges(self, LL, LR, RL, RR, bL, bR):
        L, R = self.L, self.R
        for r, c, blk in ((L, L, LL), (L, R, LR), (R, L, RL), (R, R, RR)):
            self.add(r, c, blk)
        self.b.index_add_(0, L, bL)
        self.b.index_add_(0, R, bR)

    def reset(self, nodes, rhs):
        r = self.row[nodes]
        hit = torch.zeros(self.n, dtype=torch.bool, device=r.device)
        hit[r] = True
        rows, cols = self.keys // self.n, self.keys % self.n
        self.v[hit[rows]] = 0.0
        self.v[hit[rows] & (rows == cols)] = torch.eye(self.d, dtype=F8, device=r.device)
        self.b[r] = rhs[nodes]

    def diagonal(self):
        rows, cols = self.keys // self.n, self.keys % self.n
        return self.v[rows == cols]

    def flat(self):
        """(values, rhs) in row order; also keeps row_ptr and columns."""
        d, n = self.d, self.n
        rows, cols = self.keys // n, self.keys % n
        cnt = torch.bincount(rows, minlength=n)
        start = torch.cumsum(cnt, 0) - cnt
        p = torch.arange(self.keys.numel(), device=rows.device)
        out = torch.empty(self.keys.numel() * d * d, dtype=F8, device=rows.device)
        col = torch.empty(out.numel(), dtype=torch.int64, device=rows.device)
        for q in range(d):
            for e in range(d):
                at = d * d * start[rows] + q * d * cnt[rows] + d * (p - start[rows]) + e
                out[at] = self.v[:, q, e]
                col[at] = d * cols + e
        lens = (d * cnt).repeat_interleave(d)
        self.row_ptr = torch.cat([torch.zeros(1, dtype=torch.int64, device=rows.device), torch.cumsum(lens, 0)])
        self.col = col
        return out, self.b.reshape(-1)


def _exact_scalar(c, f):
    o = _scalar_opts(c)
    P = _Pattern(f, 1)
    L, R, A, x = f["L"], f["R"], f["area"], f["x"]
    dx = x[R] - x[L]
    rho, mu, q, md = f["rho"], f["visc"], f["q"], f["mdot"]
    visc = 0.5 * (mu[L] + mu[R])
    diff = 0.5 * (mu[L] / rho[L] + mu[R] / rho[R])
    asq, axdx = (A * A).sum(1), (A * dx).sum(1)
    udx = (0.5 * dx * (f["vel"][R] + f["vel"][L])).sum(1)
    gL, gR = f["dqdx"][L], f["dqdx"][R]
    dqL, dqR = (0.5 * dx * gL).sum(1), (0.5 * dx * gR).sum(1)
    non = -(visc[:, None] * (A - (asq / axdx)[:, None] * dx) * 0.5 * (gL + gR)).sum(1)
    pe = udx.abs() / (diff + 1e-16)
    if o["tanh_form"]:
        pf = 0.5 * (1 + torch.tanh((pe - o["tanh_trans"]) / o["tanh_width"]))
    else:
        pf = pe * pe / (5 + pe * pe)
    dq = q[R] - q[L]
    limL = limR = 1.0
    if o["use_limiter"]:
        limL, limR = _rcp_limiter(4 * dqL - dq, dq), _rcp_limiter(4 * dqR - dq, dq)
    qL, qR = q[L] + dqL * limL, q[R] - dqR * limR
    lf = -visc * asq / axdx
    flux = lf * dq + non
    au = o["alpha_upw"]
    qip = 0.5 * (q[L] + q[R])
    adv = md * (pf * torch.where(md > 0, au * qL + (1 - au) * qip, au * qR + (1 - au) * qip) + (1 - pf) * qip)
    up = 0.5 * (md + md.abs()) * pf * au
    dn = 0.5 * (md - md.abs()) * pf * au
    ce = 0.5 * md * (pf * (1 - au) + (1 - pf))
    w = 1.0 / o["relax"]
    e = lambda t: t[:, None, None]  # noqa: E731
    P.add_edges(e((-lf + up + ce) * w), e(lf + dn + ce), e(lf - up - ce), e((-lf - dn - ce) * w),
                (-flux - adv)[:, None], (flux + adv)[:, None])
    return P


def _exact_momentum(c, f):
    o = _momentum_opts(c)
    P = _Pattern(f, 3)
    L, R, A, x, u = f["L"], f["R"], f["area"], f["x"], f["vel"]
    dx = x[R] - x[L]
    visc = 0.5 * (f["visc"][L] + f["visc"][R])
    asq, axdx = (A * A).sum(1), (A * dx).sum(1)
    G = f["dudx"].reshape(-1, 3, 3)
    gL, gR = G[L], G[R]
    duL, duR = (0.5 * dx[:, None] * gL).sum(2), (0.5 * dx[:, None] * gR).sum(2)
    du = u[R] - u[L]
    g = 0.5 * (gL + gR) + ((du - duL - duR) / axdx[:, None])[:, :, None] * A[:, None]
    limL = limR = 1.0
    if o["use_limiter"]:
        limL, limR = _rcp_limiter(4 * duL - du, du), _rcp_limiter(4 * duR - du, du)
    md, pf, mask = f["mdot"], f["pec"], torch.minimum(f["mask"][L], f["mask"][R])
    uip = 0.5 * (u[L] + u[R])
    upw = torch.where((md > 0)[:, None], u[L] + duL * limL, u[R] - duR * limR)
    adv = md[:, None] * (pf[:, None] * upw + (1 - pf)[:, None] * uip)
    sym = -visc[:, None] * ((g + g.transpose(1, 2)) * A[:, None]).sum(2)
    if o["include_div_u"]:
        sym = sym + 2.0 / 3.0 * o["include_div_u"] * (visc * (g[:, 0, 0] + g[:, 1, 1] + g[:, 2, 2]))[:, None] * A
    tf = sym * mask[:, None] + adv
    up, dn, ce = 0.5 * (md + md.abs()) * pf, 0.5 * (md - md.abs()) * pf, 0.5 * md * (1 - pf)
    d = -visc * asq / axdx
    Nb = (-visc / axdx)[:, None, None] * A[:, :, None] * A[:, None]
    eye = torch.eye(3, dtype=F8, device=A.device)
    LR = (dn + ce + d)[:, None, None] * eye + Nb
    RL = (-up - ce + d)[:, None, None] * eye + Nb
    P.add_edges(-RL / o["relax"], LR, RL, -LR / o["relax"], -tf, tf)
    return P


def _edge_flux(o, f, noc):
    """f and tmdot of the continuity edges (tmdot before the time scale)."""
    L, R, A, x, u, rho = f["L"], f["R"], f["area"], f["x"], f["vel"], f["rho"]
    dx = x[R] - x[L]
    asq, axdx = (A * A).sum(1), (A * dx).sum(1)
    iu = 1.0 / f["udiag"]
    pts = 0.5 * (iu[L] + iu[R])
    w = asq / axdx
    rip = 0.5 * (rho[L] + rho[R])
    it = o["interp_together"]
    ru = it * 0.5 * (rho[L, None] * u[L] + rho[R, None] * u[R]) + (1 - it) * rip[:, None] * 0.5 * (u[L] + u[R])
    g = 0.5 * (f["dpdx"][L] * iu[L, None] + f["dpdx"][R] * iu[R, None])
    tm = -pts * (f["p"][R] - f["p"][L]) * w + ((ru + g) * A - noc * (A - w[:, None] * dx) * g).sum(1)
    return w * pts, tm, rip


def _exact_continuity(c, f):
    o = _continuity_opts(c)
    P = _Pattern(f, 1)
    wp, tm, rip = _edge_flux(o, f, o["noc_fac"])
    si = o["solve_incompressible"]
    scale = (si / rip + (1 - si)) / o["tau_scale"]
    k, b = (-wp * scale)[:, None, None], (tm * scale)[:, None]
    P.add_edges(-k, k, k, -k, -b, b)
    return P


def _exact_open(P, f):
    o = _OPEN
    R, L, A, x = f["ipR"], f["ipL"], f["ipA"], f["x"]
    pts = 1.0 / f["udiag"][R]
    dx = x[R] - 0.5 * (x[R] + x[L])
    asq, axdx = (A * A).sum(1), (A * dx).sum(1)
    G = f["dpdx"][R]
    tm = -pts * (f["pbc"][R] - 0.5 * (f["p"][R] + f["p"][L])) * asq / axdx
    tm = tm + ((f["rho"][R, None] * f["vel"][R] + pts[:, None] * G) * A
               - o["noc_fac"] * pts[:, None] * (A - (asq / axdx)[:, None] * dx) * G).sum(1)
    k = (0.5 * asq / axdx * pts / o["tau_scale"])[:, None, None]
    r, l = P.row[R], P.row[L]
    P.add(r, r, k)
    P.add(r, l, k)
    P.b.index_add_(0, r, (-tm / o["tau_scale"])[:, None])


def _exact_mass(P, f):
    g1, g2, g3 = _GAMMA
    rv = f["rho"] * f["dual"]
    i = P.row
    P.add(i, i, (g1 * rv / _DT)[:, None, None] * torch.eye(3, dtype=F8, device=rv.device))
    P.b.index_add_(0, i, -(rv[:, None] * (g1 * f["vel"] + (g2 + g3) * f["qold"])) / _DT - f["dpdx"] * f["dual"][:, None])


def _exact_gradient(f, phi):
    g = torch.zeros(f["N"], phi.shape[1], 3, dtype=F8, device=phi.device)
    e = 0.5 * (phi[f["L"]] + phi[f["R"]])[:, :, None] * f["area"][:, None]
    g.index_add_(0, f["L"], e)
    g.index_add_(0, f["R"], -e)
    return (g / f["dual"][:, None, None]).reshape(f["N"], -1)


def _exact_geometry(c, f):
    conn = _elements(c).cuda()
    X = f["x"][conn]  # (M, npe, 3)
    hexes = not c["tets"]
    if hexes:
        pairs = ((0, 1), (1, 2), (2, 3), (0, 3), (4, 5), (5, 6), (6, 7), (4, 7), (0, 4), (1, 5), (2, 6), (3, 7))
        faces = ((0, 1, 2, 3), (4, 5, 6, 7), (0, 1, 5, 4), (1, 2, 6, 5), (2, 3, 7, 6), (3, 0, 4, 7))
    else:
        pairs = ((0, 1), (1, 2), (0, 2), (0, 3), (1, 3), (2, 3))
        faces = ((0, 1, 2), (0, 1, 3), (1, 2, 3), (0, 2, 3))
    mid = X.mean(1)
    keys = f["L"] * f["N"] + f["R"]
    area = torch.zeros_like(f["area"])
    for a, b in pairs:
        cen = [X[:, list(s)].mean(1) for s in faces if a in s and b in s]
        d1, d2 = mid - 0.5 * (X[:, a] + X[:, b]), cen[1] - cen[0]
        s = 0.5 * torch.linalg.cross(d1, d2)
        na, nb = conn[:, a], conn[:, b]
        lo, hi = torch.minimum(na, nb), torch.maximum(na, nb)
        along = f["x"][hi] - f["x"][lo]
        s = s * torch.sign((s * along).sum(1, keepdim=True))
        area.index_add_(0, torch.searchsorted(keys, lo * f["N"] + hi), s)
    vol = torch.zeros_like(f["dual"])
    if not hexes:
        v = torch.linalg.det(X[:, 1:] - X[:, :1]) / 24.0
        for q in range(4):
            vol.index_add_(0, conn[:, q], v)
        return area, vol
    # integral of the trilinear map's Jacobian over each octant, two Gauss
    # points a direction (exact for its degree)
    sgn = torch.tensor(((-1, -1, -1), (1, -1, -1), (1, 1, -1), (-1, 1, -1), (-1, -1, 1), (1, -1, 1), (1, 1, 1),
                        (-1, 1, 1)), dtype=F8, device="cuda")
    g = 0.5 / math.sqrt(3.0)
    for q in range(8):
        v = 0.0
        for o in itertools.product((-g, g), repeat=3):
            xi = 0.5 * sgn[q] + torch.tensor(o, dtype=F8, device="cuda")
            t = 1 + sgn * xi  # (8, 3)
            dn = torch.stack([sgn[:, 0] * t[:, 1] * t[:, 2], sgn[:, 1] * t[:, 0] * t[:, 2],
                              sgn[:, 2] * t[:, 0] * t[:, 1]], 1) / 8
            v = v + torch.linalg.det(torch.einsum("mnd,nk->mkd", X, dn)) / 8
        vol.index_add_(0, conn[:, q], v)
    return area, vol


def _gmres(A, b, d, m, iters, tol):
    """Restarted right-Jacobi GMRES(m), two Gram-Schmidt passes, from zero."""
    x = torch.zeros_like(b)
    bn = float(b.norm())
    r, its = b.clone(), 0
    V = torch.empty(m + 1, b.numel(), dtype=F8, device=b.device)
    while its < iters:
        beta = float(r.norm())
        V[0] = r / beta
        H = np.zeros((m + 1, m))
        done, j = False, 0
        while j < m and its < iters and not done:
            w = A @ (V[j] / d)
            h = V[: j + 1] @ w
            w = w - h @ V[: j + 1]
            h2 = V[: j + 1] @ w
            w = w - h2 @ V[: j + 1]
            hn = w.norm()
            H[: j + 1, j] = (h + h2).cpu().numpy()
            H[j + 1, j] = float(hn)
            V[j + 1] = w / hn
            j += 1
            its += 1
            if its % 5 == 0 or its == iters or j == m or tol >= 1e-9:
                g = np.zeros(j + 1)
                g[0] = beta
                y, *_ = np.linalg.lstsq(H[: j + 1, :j], g, rcond=None)
                done = np.linalg.norm(H[: j + 1, :j] @ y - g) <= tol * bn
        x = x + (torch.from_numpy(y).to(b) @ V[:j]) / d
        r = b - A @ x
        if done:
            break
    return x


def _bicgstab(A, b, d, iters, tol):
    x = torch.zeros_like(b)
    r = b.clone()
    rh, p = r.clone(), r.clone()
    rho, bn = rh @ r, b.norm()
    for k in range(iters):
        ph = p / d
        v = A @ ph
        a = rho / (rh @ v)
        s = r - a * v
        sh = s / d
        t = A @ sh
        w = (t @ s) / (t @ t)
        x = x + a * ph + w * sh
        r = s - w * t
        if k % 20 == 0 and float(r.norm() / bn) < tol:
            break
        rn = rh @ r
        p = r + (rn / rho) * (a / w) * (p - w * v)
        rho = rn
    return x


def exact(case, seed):
    c, kind = case, case["kind"]
    f = _fields(c, seed)
    if kind == "geometry":
        area, vol = _exact_geometry(c, f)
        return dict(area=area, volume=vol)
    if kind == "producers":
        o = _continuity_opts(c)
        _, md, _ = _edge_flux(o, f, 1.0)
        L, R = f["L"], f["R"]
        diff = 0.5 * (f["visc"][L] / f["rho"][L] + f["visc"][R] / f["rho"][R])
        pe = (0.5 * (f["x"][R] - f["x"][L]) * (f["vel"][R] + f["vel"][L])).sum(1).abs() / (diff + 1e-16)
        return dict(mdot=md, dudx=_exact_gradient(f, f["vel"]), dpdx=_exact_gradient(f, f["p"][:, None]),
                    pecfac=pe * pe / (5 + pe * pe))
    if kind in ("scalar", "solve_scalar"):
        P = _exact_scalar(c, f)
        P.reset(f["ends"], (f["pbc"] if kind == "scalar" else f["bc"][:, 0])[:, None] - f["q"][:, None])
    elif kind in ("momentum", "step", "solve_momentum"):
        P = _exact_momentum(c, f)
        if kind != "momentum":
            _exact_mass(P, f)
            u = P.diagonal()[:, 0, 0][P.row]
            P.reset(f["wall"], f["ubc"] - f["vel"])
    else:
        P = _exact_continuity(c, f)
        if kind == "solve_poisson":
            _exact_open(P, f)
    v, b = P.flat()
    if kind in ("scalar", "momentum", "continuity"):
        return dict(values=v, rhs=b)
    if kind == "step":
        pts = _GAMMA[0] / _DT
        u = (u / (f["rho"] * f["dual"]) - pts) * 0.7 + pts
        Q = _exact_continuity(c, f)
        _exact_open(Q, f)
        cv, cb = Q.flat()
        return dict(momentum=dict(values=v, rhs=b), continuity=dict(values=cv, rhs=cb), udiag=u)
    A = torch.sparse_csr_tensor(P.row_ptr, P.col, v, size=(b.numel(), b.numel()))
    diag = torch.diagonal(P.diagonal(), dim1=1, dim2=2).reshape(-1)
    if kind == "solve_poisson" and c["learned"]:
        return _bicgstab(A, b, diag, 6000, 1e-12)
    same = kind == "solve_poisson" or c["precond"] == "jacobi"
    return _gmres(A, b, diag, 50, c["iters"] if same else 1000, c["tol"] if same else 1e-13)
