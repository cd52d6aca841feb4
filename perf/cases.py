"""Cases of the solvers' work, for measuring.

One pass of a case is what a program does between two looks at its solution:
it advances a solver that it keeps by a number of iterations, with the
residual history, and takes the state.  The cases cover the explicit solvers
(Euler of first and second order, batched Euler, Navier-Stokes, RANS-SA,
scalar diffusion) and the discrete adjoint, each through the Python classes
of ``finitevolume_gb300.solvers``.

``exact`` restates each scheme in plain torch, in 64 bits, from the mesh's
nodes and cells: nothing of the package's arithmetic is used there.
"""
import functools
import math

import numpy as np
import torch

from finitevolume_gb300 import meshgen
from finitevolume_gb300 import solvers as S

GAMMA = 1.4
GAS_CONSTANT, PRANDTL, PRANDTL_T, REYNOLDS = 287.0, 0.72, 0.9, 6e6
FLUXES = {"rusanov": S.NumericalFluxScheme.Rusanov, "hllc": S.NumericalFluxScheme.HLLC}
LIMITERS = {"barth": S.Limiter.BarthJespersen, "venkat": S.Limiter.Venkatakrishnan}
GRADIENTS = {"lsq": S.GradientScheme.LeastSquares, "gauss": S.GradientScheme.GreenGauss}


# --------------------------------------------------------------------------
# The cases
# --------------------------------------------------------------------------
def _euler(name, mesh, ni, nj, steps, **kw):
    case = {"name": name, "kind": "euler", "mesh": mesh, "ni": ni, "nj": nj, "steps": steps, "order": 2, "rk": 3,
            "local_dt": True, "flux": "hllc", "limiter": "venkat", "fp32": False, "mach": 0.8, "aoa": 1.25, "cfl": 1.2}
    case.update(kw)
    return case


def listed():
    return [
        # the smallest solve in use (test and smoke size): launches and latency
        _euler("euler2_2k", "ogrid", 64, 32, 20, mach=0.5, aoa=2.0),
        # an ordinary airfoil mesh: quads near the wall, polygons of 3 to 9 sides outside
        _euler("euler2_mixed_61k", "mixed", 256, 128, 10),
        # the headline size, FP64 and with the FP32 flux
        _euler("euler2_1m", "ogrid", 1448, 724, 8),
        _euler("euler2_fp32_1m", "ogrid", 1448, 724, 20, fp32=True),
        # shock tube on perturbed triangles, time-accurate (global dt)
        _euler("tube2_tri_500k", "tube", 1000, 250, 8, local_dt=False, cfl=0.5),
        # the reference's own scheme: first order, forward Euler; a small steady solve ...
        _euler("euler1_32k", "ogrid", 256, 128, 256, order=1, rk=1, flux="rusanov", mach=0.5, aoa=2.0, cfl=0.5),
        # ... and a large one with the global time step
        _euler("euler1_500k", "ogrid", 1024, 488, 30, order=1, rk=1, local_dt=False, cfl=0.5),
        # a family of airfoils of uneven sizes advanced together
        {"name": "batch_16", "kind": "batch", "instances": 16, "lo": 4096, "hi": 65536, "steps": 10, "fp32": False},
        # laminar airfoil with a no-slip wall
        {"name": "ns_130k", "kind": "ns", "ni": 510, "nj": 255, "steps": 10, "flux": "hllc", "gradient": "gauss",
         "reynolds": 5000.0, "mach": 0.5, "aoa": 2.0},
        # turbulent airfoil on wall-clustered quads and triangles
        {"name": "rans_250k", "kind": "rans", "ni": 512, "nj": 220, "steps": 10, "flux": "hllc", "gradient": "gauss",
         "mach": 0.15, "aoa": 4.0},
        # lift or drag sensitivities: linearisation and pseudo-time adjoint iterations
        {"name": "adjoint_125k", "kind": "adjoint", "ni": 512, "nj": 244, "iterations": 20, "mach": 0.5, "aoa": 2.0,
         "objective": "drag"},
        # heat conduction on a plate
        {"name": "diffusion_260k", "kind": "diffusion", "nx": 512, "ny": 511, "steps": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["euler2", "euler2", "euler2", "tube", "euler1", "batch", "ns", "rans", "adjoint", "diffusion"])
    flow = {"mach": round(rng.uniform(0.3, 0.85), 3), "aoa": round(rng.uniform(-4.0, 8.0), 2)}
    if kind in ("euler2", "tube", "euler1"):
        cells = _log_int(rng, 1500, 900000 if kind != "tube" else 500000)
        steps = max(2, min(100, 1500000 // cells))
        if kind == "euler2":
            mesh = "mixed" if cells < 100000 and rng.random() < 0.4 else "ogrid"
            nj = max(16, int(math.sqrt(cells / 2.0)))
            return _drawn(_euler("", mesh, 2 * nj + (2 * rng.randrange(4) if mesh == "ogrid" else 0), nj, steps,
                                 fp32=rng.random() < 0.3, limiter=rng.choice(["venkat", "venkat", "barth"]),
                                 flux=rng.choice(["hllc", "hllc", "rusanov"]), **flow))
        if kind == "tube":
            ny = max(8, int(math.sqrt(cells / 8.0)))
            return _drawn(_euler("", "tube", 4 * ny + rng.randrange(4), ny, steps, local_dt=False, cfl=0.5,
                                 limiter=rng.choice(["venkat", "barth"]), flux=rng.choice(["hllc", "rusanov"])))
        nj = max(16, int(math.sqrt(cells / 2.0)))
        return _drawn(_euler("", "ogrid", 2 * nj + 2 * rng.randrange(4), nj, min(400, 8 * steps), order=1, rk=1, cfl=0.5,
                             flux=rng.choice(["hllc", "rusanov"]), local_dt=rng.random() < 0.5, **flow))
    if kind == "batch":
        return {"kind": kind, "instances": rng.randrange(4, 17), "lo": 4096, "hi": _log_int(rng, 8192, 65536),
                "steps": rng.randrange(5, 11), "fp32": rng.random() < 0.4}
    if kind == "ns":
        nj = _log_int(rng, 24, 300)
        return {"kind": kind, "ni": 2 * nj + 2 * rng.randrange(4), "nj": nj, "steps": rng.randrange(5, 20),
                "flux": rng.choice(["hllc", "rusanov"]), "gradient": rng.choice(["gauss", "lsq"]),
                "reynolds": float(_log_int(rng, 500, 20000)), "mach": flow["mach"], "aoa": flow["aoa"]}
    if kind == "rans":
        ni = 2 * _log_int(rng, 48, 256)
        return {"kind": kind, "ni": ni, "nj": max(40, int(0.43 * ni)), "steps": rng.randrange(5, 11),
                "flux": rng.choice(["hllc", "rusanov"]), "gradient": rng.choice(["gauss", "lsq"]),
                "mach": round(rng.uniform(0.1, 0.3), 3), "aoa": flow["aoa"]}
    if kind == "adjoint":
        nj = _log_int(rng, 24, 244)
        return {"kind": kind, "ni": 2 * nj + 2 * rng.randrange(4), "nj": nj, "iterations": rng.randrange(5, 21),
                "mach": flow["mach"], "aoa": flow["aoa"], "objective": rng.choice(["drag", "lift"])}
    nx = _log_int(rng, 48, 700)
    return {"kind": "diffusion", "nx": nx, "ny": max(40, int(nx * rng.uniform(0.5, 1.0))), "steps": rng.randrange(8, 65)}


def _drawn(case):
    del case["name"]
    return case


@functools.lru_cache(maxsize=2)
def _poly(kind, ni, nj):
    if kind == "ogrid":
        return meshgen.naca_ogrid(ni, nj)
    if kind == "mixed":
        return meshgen.naca_mixed(ni=ni, nj=nj)
    if kind == "tube":
        return meshgen.sod_strip(ni, nj, seed=0)
    if kind == "hybrid":
        return meshgen.naca_hybrid(ni=ni, n_layers=40, tri_rows=nj)
    return meshgen.cartesian(ni, nj, 1.0, nj / ni)


@functools.lru_cache(maxsize=2)
def _mesh(kind, ni, nj):
    return S.Mesh(_poly(kind, ni, nj))


@functools.lru_cache(maxsize=2)
def _family(instances, lo, hi):
    cases = meshgen.batch_cases(instances, seed=3, cells=(lo, hi))
    polys = [meshgen.naca_ogrid(c["ni"], c["nj"], shape=c["shape"]) for c in cases]
    return cases, polys, [S.Mesh(p) for p in polys]


def _case_poly(case):
    kind = case["kind"]
    if kind == "diffusion":
        return _poly("plate", case["nx"], case["ny"])
    return _poly({"ns": "ogrid", "adjoint": "ogrid", "rans": "hybrid"}.get(kind) or case["mesh"], case["ni"], case["nj"])


def _case_mesh(case):
    kind = case["kind"]
    if kind == "diffusion":
        return _mesh("plate", case["nx"], case["ny"])
    return _mesh({"ns": "ogrid", "adjoint": "ogrid", "rans": "hybrid"}.get(kind) or case["mesh"], case["ni"], case["nj"])


# --------------------------------------------------------------------------
# Inputs
# --------------------------------------------------------------------------
def _freestream(mach, aoa):
    a = math.radians(aoa)
    return 1.0, mach * math.cos(a), mach * math.sin(a), 1.0 / GAMMA


def _conserved(w):
    r, u, v, p = w[..., 0], w[..., 1], w[..., 2], w[..., 3]
    return np.stack([r, r * u, r * v, p / (GAMMA - 1.0) + 0.5 * r * (u * u + v * v)], -1)


def _waves(xy, rng, n):
    """n seeded smooth fields of size about one over the points xy."""
    out = []
    for _ in range(n):
        k, ph = rng.uniform(0.5, 3.0, size=(3, 2)), rng.uniform(0, 2 * np.pi, size=3)
        out.append(sum(np.sin(xy @ k[i] + ph[i]) for i in range(3)) / 3.0)
    return out


def _points(poly):
    """A point inside each cell (the mean of its vertices)."""
    n = np.diff(poly.cell_off)
    xy = poly.nodes[poly.cell_nodes]
    return np.add.reduceat(xy, poly.cell_off[:-1], axis=0) / n[:, None]


def _perturbed(poly, rng, fs):
    """The freestream with a smooth perturbation of 1%: a uniform start would leave the gradients zero."""
    f = _waves(_points(poly), rng, 4)
    r, u, v, p = fs
    m = math.hypot(u, v)
    return _conserved(np.stack([r * (1.0 + 0.01 * f[0]), u + 0.01 * m * f[1], v + 0.01 * m * f[2],
                                p * (1.0 + 0.01 * f[3])], -1))


def _start(case, seed):
    """The seeded initial state of a case, in the mesh's cell order."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "batch":
        cases, polys, _ = _family(case["instances"], case["lo"], case["hi"])
        return np.concatenate([_perturbed(p, rng, _freestream(c["mach"], c["aoa_deg"])) for c, p in zip(cases, polys)])
    poly = _case_poly(case)
    if kind == "diffusion":
        return 1.0 + 0.5 * _waves(4.0 * _points(poly), rng, 1)[0]
    if kind == "euler" and case["mesh"] == "tube":
        f = _waves(4.0 * _points(poly), rng, 4)
        left = _points(poly)[:, 0] < 0.5
        return _conserved(np.stack([np.where(left, 1.0, 0.125) * (1.0 + 0.01 * f[0]), 0.01 * f[1], 0.01 * f[2],
                                    np.where(left, 1.0, 0.1) * (1.0 + 0.01 * f[3])], -1))
    return _perturbed(poly, rng, _freestream(case["mach"], case["aoa"]))


def _start_nut(case, seed):
    nu = case["mach"] / REYNOLDS
    return 3.0 * nu * (1.0 + 0.1 * _waves(_points(_case_poly(case)), np.random.default_rng(seed + 7919), 1)[0])


def _force_ref(case):
    r, u, v, p = _freestream(case["mach"], case["aoa"])
    return (r, u, v, p, 1.0, 0.25, 0.0)


# --------------------------------------------------------------------------
# One pass
# --------------------------------------------------------------------------
class _DeviceState:
    """The solver's state on the GPU, for torch."""

    def __init__(self, solver):
        ptr, _ = solver.device_state()
        self.__cuda_array_interface__ = {"shape": (solver.n_cells, 4), "typestr": "<f8", "data": (ptr, False),
                                         "version": 3}


def _with_state(solver, case, **kw):
    """A solver, its state as a tensor (device cell order) and each cell's place there."""
    perm = solver.mesh.permutation()
    place = np.empty_like(perm)
    place[perm] = np.arange(perm.size, dtype=perm.dtype)
    holder = _DeviceState(solver)
    return {"case": case, "solver": solver, "holder": holder, "U": torch.as_tensor(holder, device="cuda"),
            "place": torch.from_numpy(place.astype(np.int64)).cuda()[:, None].expand(-1, 4), **kw}


def _euler_solver(case, order=2, rk=3, local_dt=True, flux="hllc", limiter="venkat", fp32=False, cfl=1.2):
    fs = _freestream(case["mach"], case["aoa"])
    mesh = _case_mesh(case)
    T = S.EulerBoundaryType
    if case.get("mesh") == "tube":
        bcs = [S.EulerBoundaryCondition(t) for t in (T.Wall, T.Outflow, T.Wall, T.Outflow)]
    else:
        bcs = [S.EulerBoundaryCondition(T.Wall),
               S.EulerBoundaryCondition(T.CharacteristicFarfield, S.from_primitive(*fs, GAMMA))]
    ic = S.EulerInitialCondition(S.EulerICMode.Freestream, rho=fs[0], u=fs[1], v=fs[2], p=fs[3])
    return S.EulerFVMSolver(mesh, bcs, GAMMA, cfl, ic, FLUXES[flux], order=order, rk_stages=rk, local_dt=local_dt,
                            limiter=LIMITERS[limiter], fp32_flux=fp32)


def prepare(case, seed):
    kind = case["kind"]
    U0 = _start(case, seed)
    if kind == "euler":
        s = _euler_solver(case, case["order"], case["rk"], case["local_dt"], case["flux"], case["limiter"],
                          case["fp32"], case["cfl"])
        s.set_field(U0)
        return _with_state(s, case)
    if kind == "batch":
        cases, _, meshes = _family(case["instances"], case["lo"], case["hi"])
        T = S.EulerBoundaryType
        b = S.BatchSolver(meshes, [T.Wall, T.CharacteristicFarfield],
                          [_freestream(c["mach"], c["aoa_deg"]) for c in cases], GAMMA, 1.2, fp32_flux=case["fp32"])
        b.set_field(U0)
        return {"case": case, "solver": b}
    if kind in ("ns", "rans"):
        fs = _freestream(case["mach"], case["aoa"])
        far = S.NSBoundaryCondition(S.NSBoundaryType.Farfield, farfield_state=list(S.from_primitive(*fs, GAMMA)))
        wall = S.NSBoundaryCondition(S.NSBoundaryType.NoSlipWall)
        ic = S.EulerInitialCondition(S.EulerICMode.Freestream, rho=fs[0], u=fs[1], v=fs[2], p=fs[3])
        how = FLUXES[case["flux"]], GRADIENTS[case["gradient"]]
        if kind == "ns":
            s = S.NavierStokesFVMSolver(_case_mesh(case), [wall, far], GAMMA, GAS_CONSTANT,
                                        case["mach"] / case["reynolds"], PRANDTL, 0.5, ic, *how)
            s.set_field(U0)
        else:
            mu = case["mach"] / REYNOLDS
            s = S.RANSTurbulenceSASolver(_case_mesh(case), [S.RANSBoundaryConditionSA(wall),
                                                            S.RANSBoundaryConditionSA(far, 3.0 * mu)],
                                         GAMMA, GAS_CONSTANT, mu, PRANDTL, PRANDTL_T, 0.5, ic, 3.0 * mu, *how)
            s.set_field(U0, _start_nut(case, seed))
        return _with_state(s, case)
    if kind == "adjoint":
        s = _euler_solver(case)
        s.set_field(U0)
        return {"case": case, "solver": s, "adjoint": S.DiscreteAdjoint(s), "ref": _force_ref(case),
                "objective": S.Objective.Drag if case["objective"] == "drag" else S.Objective.Lift}
    h = 1.0 / case["nx"]
    s = S.UnstructuredFVMSolver(_case_mesh(case), 1.0, 0.2 * h * h, 1.0, 0.0,
                                {"bottom": (S.BoundaryType.Dirichlet, 1.0), "top": (S.BoundaryType.Neumann, 0.1),
                                 "left": (S.BoundaryType.Dirichlet, 0.5), "right": (S.BoundaryType.Neumann, -0.1)})
    s.set_field(U0)
    return {"case": case, "solver": s}


def run(state):
    case, s = state["case"], state["solver"]
    kind = case["kind"]
    if kind == "batch":
        s.run(case["steps"])
        return {"state": s.field_all(), "norms": s.status()[2]}
    if kind == "diffusion":
        history = s.run(case["steps"], history=True)
        return {"state": s.field(), "history": history}
    if kind == "adjoint":
        residual = state["adjoint"].forward()
        J, g = S.force_gradient(s, state["objective"], state["ref"])
        lam, fsbar, history, _ = state["adjoint"].solve(g, max_iter=case["iterations"], tol=1e-300)
        return {"residual": residual, "J": J, "dJdU": g, "lambda": lam, "fsbar": fsbar, "history": history}
    history = s.run(case["steps"], history=True)
    out = {"state": state["U"].gather(0, state["place"]), "history": history}
    if kind == "rans":
        out["nut"] = s.nut_field()
    return out


# --------------------------------------------------------------------------
# What a pass cannot do without
# --------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "batch":
        cells = sum(c["ni"] * c["nj"] for c in meshgen.batch_cases(case["instances"], seed=3,
                                                                   cells=(case["lo"], case["hi"])))
        faces, stages, order, size = 2 * cells, 3 * case["steps"], 2, 4 if case["fp32"] else 8
    else:
        poly = _case_poly(case)
        cells = poly.n_cells
        faces = (poly.cell_nodes.size + poly.bedges.shape[0]) // 2
        stages = case["steps"] * case.get("rk", 1) if kind != "adjoint" else 3 * case["iterations"] + 1
        order, size = case.get("order", 2 if kind == "adjoint" else 1), 4 if case.get("fp32") else 8
    if kind == "diffusion":
        return {"bytes": stages * (24 * cells + 24 * faces), "flops": stages * (8 * cells + 5 * faces)}
    if kind == "adjoint":
        # per stage the cotangent, its two face Jacobians and the reconstruction geometry
        return {"bytes": stages * (96 * cells + (256 + 48) * faces), "flops": stages * (140 * cells + 130 * faces)}
    # per stage: the state read and written, each face's geometry and cells, at order 2 the cells' reconstruction
    byte = 64 * cells + (4 * size + 8) * faces + (order - 1) * (4 * size * faces + size * cells)
    flops = 30 * cells + 110 * faces + (order - 1) * (130 * cells + 70 * faces)
    if kind in ("ns", "rans"):
        byte += 7 * 8 * faces
        flops += (60 * cells + 110 * faces) * (2 if kind == "rans" else 1)
    return {"bytes": stages * byte, "flops": stages * flops}


# --------------------------------------------------------------------------
# The schemes in plain torch
# --------------------------------------------------------------------------
class _Geometry:
    """Faces, cells and weights of a polygon mesh, from its nodes and cells."""

    def __init__(self, poly):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        off, cn, xy = poly.cell_off.astype(np.int64), poly.cell_nodes.astype(np.int64), poly.nodes
        n, nn = off.size - 1, xy.shape[0]
        size = np.diff(off)
        cell = np.repeat(np.arange(n), size)
        nxt = np.arange(cn.size) + 1
        nxt[off[1:] - 1] = off[:-1]
        a, b = cn, cn[nxt]
        # a face belongs to the cell that comes first; its direction is that cell's
        key = np.minimum(a, b) * nn + np.maximum(a, b)
        uniq, first, face = np.unique(key, return_index=True, return_inverse=True)
        face = face.reshape(-1)
        owner = first[face] == np.arange(cn.size)
        fl, fr = cell[first], np.full(uniq.size, -1)
        fr[face[~owner]] = cell[~owner]
        patch = np.full(uniq.size, -1)
        be = poly.bedges.astype(np.int64)
        patch[np.searchsorted(uniq, be.min(1) * nn + be.max(1))] = poly.bpatch
        # polygons: area, centroid
        cross = xy[a, 0] * xy[b, 1] - xy[b, 0] * xy[a, 1]
        area = 0.5 * np.add.reduceat(cross, off[:-1])
        cen = np.stack([np.add.reduceat((xy[a, d] + xy[b, d]) * cross, off[:-1]) / (6.0 * area) for d in (0, 1)], 1)
        d = xy[b[first]] - xy[a[first]]
        length = np.sqrt((d * d).sum(1))
        mid = 0.5 * (xy[a[first]] + xy[b[first]])
        # per cell its entries (edges), padded
        pad = np.full((n, size.max()), cn.size)
        pad[cell, np.arange(cn.size) - off[cell]] = np.arange(cn.size)
        other = np.where(owner, fr[face], fl[face])
        t = lambda x: torch.as_tensor(np.ascontiguousarray(x), device=dev)  # noqa: E731
        bnd = np.flatnonzero(fr < 0)
        slot = np.full(uniq.size, -1)
        slot[bnd] = np.arange(bnd.size)
        self.n, self.dev = n, dev
        self.bnd, self.bpatch = t(bnd), t(patch[bnd])
        self.fl, self.fr, self.inner = t(fl), t(np.where(fr < 0, fl, fr)), t(fr >= 0)
        # the place of the right state among (cells, boundary values)
        self.right = t(np.where(fr < 0, n + slot, fr))
        self.nx, self.ny, self.len = t(d[:, 1] / length), t(-d[:, 0] / length), t(length)
        self.vol, self.cen, self.mid = t(area), t(cen), t(mid)
        self.pad, self.cell, self.face = t(pad), t(cell), t(face)
        self.sign = t(np.where(owner, -1.0, 1.0))
        self.nb = t(np.where(other < 0, n + slot[face], other))

    def per_cell(self, x, fill=0.0):
        """The entries' values [E, ...] gathered per cell [N, K, ...]."""
        return torch.cat([x, torch.full_like(x[:1], fill)])[self.pad]

    def residual(self, flux):
        """Each cell's sum of the face fluxes (times length): its own faces out, the others in."""
        s = self.sign.view(-1, *([1] * (flux.dim() - 1)))
        return self.per_cell(s * flux[self.face]).sum(1)

    def centre(self, nb_point):
        """The points that a cell's differences reach to: neighbour centroids and boundary midpoints."""
        return torch.cat([self.cen, self.mid[self.bnd]])[nb_point]

    def lsq(self):
        """Least-squares weights per entry, inverse-distance-squared."""
        d = self.centre(self.nb) - self.cen[self.cell]
        w = 1.0 / (d * d).sum(1)
        m = self.per_cell(torch.stack([w * d[:, 0] ** 2, w * d[:, 0] * d[:, 1], w * d[:, 1] ** 2], 1)).sum(1)[self.cell]
        det = m[:, 0] * m[:, 2] - m[:, 1] ** 2
        return torch.stack([(m[:, 2] * d[:, 0] - m[:, 1] * d[:, 1]) * w / det,
                            (m[:, 0] * d[:, 1] - m[:, 1] * d[:, 0]) * w / det], 1)

    def gradient(self, phi, ext, scheme):
        """Gradients [N, k, 2] of cell fields phi [N, k]; ext: phi with the boundary values behind it."""
        if scheme == "lsq":
            if not hasattr(self, "_lsq"):
                self._lsq = self.lsq()
            return self.per_cell(self._lsq[:, None, :] * (ext[self.nb] - phi[self.cell])[:, :, None]).sum(1)
        far = self.nb >= self.n
        dc = (self.cen[self.cell] - self.mid[self.face]).norm(dim=1)
        do = (self.centre(self.nb) - self.mid[self.face]).norm(dim=1)
        w = torch.where(far, torch.zeros_like(dc), do / (dc + do))[:, None]
        value = w * phi[self.cell] + (1.0 - w) * ext[self.nb]
        normal = torch.stack([self.nx, self.ny], 1)[self.face] * (-self.sign * self.len[self.face])[:, None]
        return self.per_cell(value[:, :, None] * normal[:, None, :]).sum(1) / self.vol[:, None, None]


def _prim(U):
    r, u, v = U[:, 0], U[:, 1] / U[:, 0], U[:, 2] / U[:, 0]
    return torch.stack([r, u, v, (GAMMA - 1.0) * (U[:, 3] - 0.5 * r * (u * u + v * v))], 1)


def _flux(scheme, L, R, nx, ny):
    """Numerical flux per unit length of primitive states [F, 4]."""
    def side(w):
        r, u, v, p = w.unbind(1)
        vn, c, E = u * nx + v * ny, torch.sqrt(GAMMA * p / r), p / (GAMMA - 1.0) + 0.5 * r * (u * u + v * v)
        U = torch.stack([r, r * u, r * v, E], 1)
        return r, vn, v * nx - u * ny, p, c, E, U, torch.stack([r * vn, r * u * vn + p * nx, r * v * vn + p * ny,
                                                               (E + p) * vn], 1)
    rl, nl, tl, pl, cl, El, Ul, Fl = side(L)
    rr, nr, tr, pr, cr, Er, Ur, Fr = side(R)
    if scheme == "rusanov":
        s = torch.maximum(nl.abs() + cl, nr.abs() + cr)[:, None]
        return 0.5 * (Fl + Fr) - 0.5 * s * (Ur - Ul)
    sl, sr = torch.minimum(nl - cl, nr - cr), torch.maximum(nl + cl, nr + cr)
    sm = (pr - pl + rl * nl * (sl - nl) - rr * nr * (sr - nr)) / (rl * (sl - nl) - rr * (sr - nr))

    def star(r, vn, vt, p, E, U, F, s):
        fac = r * (s - vn) / (s - sm)
        Us = torch.stack([fac, fac * (sm * nx - vt * ny), fac * (sm * ny + vt * nx),
                          fac * (E / r + (sm - vn) * (sm + p / (r * (s - vn))))], 1)
        return F + s[:, None] * (Us - U)
    mid = torch.where((sm >= 0)[:, None], star(rl, nl, tl, pl, El, Ul, Fl, sl), star(rr, nr, tr, pr, Er, Ur, Fr, sr))
    return torch.where((sl >= 0)[:, None], Fl, torch.where((sr <= 0)[:, None], Fr, mid))


def _ghost(kinds, fs, w, nx, ny, patch):
    """Boundary states: kinds[patch] of wall, outflow, farfield, noslip, characteristic; fs the freestream."""
    r, u, v, p = w.unbind(1)
    vn = u * nx + v * ny
    rf, uf, vf, pf = fs
    ones = torch.ones_like(r)
    out = {"outflow": w, "farfield": torch.stack([rf * ones, uf * ones, vf * ones, pf * ones], 1),
           "noslip": torch.stack([r, -u, -v, p], 1),
           "wall": torch.stack([r, u - 2.0 * vn * nx, v - 2.0 * vn * ny, p], 1)}
    if "characteristic" in kinds:
        c, cf, vnf = torch.sqrt(GAMMA * p / r), (GAMMA * pf / rf) ** 0.5, uf * nx + vf * ny
        k = 2.0 / (GAMMA - 1.0)
        vb, cb = 0.5 * (vn + k * c + vnf - k * cf), 0.25 * (GAMMA - 1.0) * (vn + k * c - vnf + k * cf)
        leaves = vb > 0
        rb = torch.where(leaves, r * (cb.abs() / c) ** k, rf * (cb.abs() / cf) ** k)
        ut, vt = torch.where(leaves, u - vn * nx, uf - vnf * nx), torch.where(leaves, v - vn * ny, vf - vnf * ny)
        b = torch.stack([rb, ut + vb * nx, vt + vb * ny, rb * cb * cb / GAMMA], 1)
        b = torch.where((vn >= c)[:, None], w, b)
        out["characteristic"] = torch.where((vnf <= -cf)[:, None], out["farfield"], b)
    g = torch.zeros_like(w)
    for i, kind in enumerate(kinds):
        g = torch.where((patch == i)[:, None], out[kind], g)
    return g


def _boundary(m, kinds, fs, w):
    return _ghost(kinds, fs, w, m.nx[m.bnd], m.ny[m.bnd], m.bpatch)


def _limited(m, W, grad, ext, limiter):
    """The limiter values [N, 4] of the unlimited gradients."""
    d = m.per_cell((ext[m.nb] - W[m.cell]))
    dmax, dmin = d.amax(1)[m.cell], d.amin(1)[m.cell]  # the padding's zero is the cell's own value
    step = (grad[m.cell] * (m.mid[m.face] - m.cen[m.cell])[:, None, :]).sum(2)
    up = step > 0
    d1, y = torch.where(up, dmax.clamp(min=0), -dmin.clamp(max=0)), step.abs()
    if limiter == "barth":
        psi = d1 / y
    else:
        e = ((5.0 * torch.sqrt(m.vol)) ** 3)[m.cell][:, None]
        psi = (d1 * d1 + e + 2.0 * d1 * y) / (d1 * d1 + 2.0 * y * y + d1 * y + e)
    psi = torch.where(y > 0, psi.clamp(max=1.0), torch.ones_like(psi))
    return m.per_cell(psi, 1.0).amin(1)


def _face_states(m, case, kinds, fs, W, psi=None):
    """Left and right states at the faces."""
    if case.get("order", 2) == 1:
        left, right = W[m.fl], W[m.fr]
    else:
        ext = torch.cat([W, 0.5 * (W[m.fl[m.bnd]] + _boundary(m, kinds, fs, W[m.fl[m.bnd]]))])
        grad = m.gradient(W, ext, "lsq")
        if psi is None:
            psi = _limited(m, W, grad, ext, case.get("limiter", "venkat"))
        grad = grad * psi[:, :, None]

        def to_face(c):
            w = W[c] + (grad[c] * (m.mid - m.cen[c])[:, None, :]).sum(2)
            return torch.where(((w[:, 0] > 0) & (w[:, 3] > 0))[:, None], w, W[c])
        left, right = to_face(m.fl), to_face(m.fr)
    ghost = _boundary(m, kinds, fs, left[m.bnd])
    return left, torch.cat([right, ghost])[torch.where(m.inner, torch.arange(m.fl.numel(), device=m.dev), m.right - m.n
                                                       + m.fl.numel())]


def _euler_residual(m, case, kinds, fs, U, psi=None):
    left, right = _face_states(m, case, kinds, fs, _prim(U), psi)
    return m.residual(_flux(case.get("flux", "hllc"), left, right, m.nx, m.ny) * m.len[:, None])


def _speeds(m, W):
    """Each face's largest wave speed, of the cells on its sides."""
    c = torch.sqrt(GAMMA * W[:, 3] / W[:, 0])
    s = lambda i: (W[i, 1] * m.nx + W[i, 2] * m.ny).abs() + c[i]  # noqa: E731
    return torch.where(m.inner, torch.maximum(s(m.fl), s(m.fr)), s(m.fl))


def _step_over_volume(m, W, cfl, local):
    lam = _speeds(m, W)
    if local:
        return cfl / m.per_cell((lam * m.len)[m.face]).sum(1)
    size = torch.where(m.inner, torch.minimum(m.vol[m.fl], m.vol[m.fr]), m.vol[m.fl]) / m.len
    return (cfl * size / lam).min() / m.vol


def _euler_steps(m, case, kinds, fs, U):
    history = []
    for _ in range(case["steps"]):
        k = _step_over_volume(m, _prim(U), case["cfl"], case["local_dt"])[:, None]
        R = _euler_residual(m, case, kinds, fs, U)
        history.append((R * R).sum(0).sqrt())
        V = U + k * R
        if case["rk"] == 3:
            V = 0.75 * U + 0.25 * (V + k * _euler_residual(m, case, kinds, fs, V))
            V = U / 3.0 + (2.0 / 3.0) * (V + k * _euler_residual(m, case, kinds, fs, V))
        U = V
    return U, torch.stack(history)


def _sa_fv1(nut, nu):
    chi3 = (nut / nu) ** 3
    return torch.where(nut > 0, chi3 / (chi3 + 7.1 ** 3), torch.zeros_like(nut))


def _sa_source(nut, nu, omega, d, g):
    cb1, cb2, sigma, kappa, cw2, cw3, cv2, cv3 = 0.1355, 0.622, 2.0 / 3.0, 0.41, 0.3, 2.0, 0.7, 0.9
    chi = torch.where(nut > 0, nut / nu, torch.zeros_like(nut))
    sbar = nut / (kappa * d) ** 2 * (1.0 - chi / (1.0 + chi * _sa_fv1(nut, nu)))
    s = torch.where(sbar >= -cv2 * omega, omega + sbar,
                    omega + omega * (cv2 * cv2 * omega + cv3 * sbar) / ((cv3 - 2.0 * cv2) * omega - sbar))
    r = (nut / (s.clamp(min=1e-10) * (kappa * d) ** 2)).clamp(max=10.0)
    q = r + cw2 * (r ** 6 - r)
    fw = q * ((1.0 + cw3 ** 6) / (q ** 6 + cw3 ** 6)) ** (1.0 / 6.0)
    cw1 = cb1 / kappa ** 2 + (1.0 + cb2) / sigma
    destroyed = torch.where(nut > 0, cw1 * fw * (nut / d) ** 2, torch.zeros_like(nut))
    return cb1 * s * nut - destroyed + cb2 / sigma * (g * g).sum(1)


def _wall_distance(m, poly, patch):
    e = torch.as_tensor(poly.nodes[poly.bedges[poly.bpatch == patch].astype(np.int64)], device=m.dev)
    a, d = e[:, 0], e[:, 1] - e[:, 0]
    out = []
    for c in m.cen.split(1 << 14):
        t = (((c[:, None] - a) * d).sum(2) / (d * d).sum(1)).clamp(0.0, 1.0)
        out.append((c[:, None] - a - t[:, :, None] * d).norm(dim=2).amin(1))
    return torch.cat(out)


def _viscous_steps(m, poly, case, fs, U, nut):
    """Navier-Stokes, and with nut the Spalart-Allmaras model on top of it: wall patch 0, farfield patch 1."""
    kinds, sa = ["noslip", "farfield"], nut is not None
    mu = case["mach"] / (REYNOLDS if sa else case["reynolds"])
    cp = GAMMA * GAS_CONSTANT / (GAMMA - 1.0)
    ob, wall = m.fl[m.bnd], (m.bpatch == 0)
    reach = torch.where(m.inner[:, None], m.cen[m.fr], m.mid) - m.cen[m.fl]
    dist = reach.norm(dim=1)
    normal = torch.stack([m.nx, m.ny], 1)
    cos = (reach * normal).sum(1) / dist
    skew = normal - reach / (dist * cos)[:, None]
    gap = (reach * normal).sum(1)
    dl, dr = (m.cen[m.fl] - m.mid).norm(dim=1), (m.cen[m.fr] - m.mid).norm(dim=1)
    wl = torch.where(m.inner, dr / (dl + dr), torch.ones_like(dl))[:, None, None]
    carries = m.inner.clone()
    carries[m.bnd] = wall
    walld = _wall_distance(m, poly, 0) if sa else None
    history, nut_history = [], []
    for _ in range(case["steps"]):
        W = _prim(U)
        T = W[:, 3] / (W[:, 0] * GAS_CONSTANT)
        phi = torch.stack([W[:, 1], W[:, 2], T], 1)
        at_wall = torch.stack([torch.zeros_like(T[ob]), torch.zeros_like(T[ob]), T[ob]], 1)
        value = torch.where(wall[:, None], at_wall, phi[ob])
        if sa:
            phi = torch.cat([phi, nut[:, None]], 1)
            value = torch.cat([value, torch.where(wall, torch.zeros_like(nut[ob]), 3.0 * mu + 0.0 * nut[ob])[:, None]], 1)
        ext = torch.cat([phi, value])
        grad = m.gradient(phi, ext, case["gradient"])
        left, right = phi[m.fl], ext[m.right]
        # face gradients: the mean, its normal part from the difference across the face
        g = wl * grad[m.fl] + (1.0 - wl) * grad[m.fr]
        dn = (right - left) / (dist * cos)[:, None] + (g * skew[:, None, :]).sum(2)
        g = g + (dn - (g * normal[:, None, :]).sum(2))[:, :, None] * normal[:, None, :]
        ghost = _boundary(m, kinds, fs, W[ob])
        WR = torch.cat([W, ghost])[m.right]
        inv = _flux(case["flux"], W[m.fl], WR, m.nx, m.ny)
        nu = mu / W[:, 0]
        nu_r = torch.where(m.inner, nu[m.fr], nu[m.fl])
        rho_r = torch.where(m.inner, W[m.fr, 0], W[m.fl, 0])
        if sa:
            nut_of = lambda x, n: x * _sa_fv1(x, n)  # noqa: E731
            nt = nut_of(nut, nu)
            nt_r = torch.where(m.inner, nt[m.fr], nut_of(right[:, 3], nu_r))
            turb = 0.5 * (W[m.fl, 0] * nt[m.fl] + rho_r * nt_r)
            most = torch.maximum(nu[m.fl], nu_r) + torch.where(m.inner, torch.maximum(nt[m.fl], nt[m.fr]), nt[m.fl])
        else:
            turb, most = torch.zeros_like(nu_r), torch.maximum(nu[m.fl], nu_r)
        visc, cond = mu + turb, cp * (mu / PRANDTL + turb / PRANDTL_T)
        div = (2.0 / 3.0) * (g[:, 0, 0] + g[:, 1, 1])
        txx, tyy = visc * (2.0 * g[:, 0, 0] - div), visc * (2.0 * g[:, 1, 1] - div)
        txy = visc * (g[:, 0, 1] + g[:, 1, 0])
        q = torch.where(m.inner[:, None], -cond[:, None] * g[:, 2], torch.zeros_like(g[:, 2]))
        uf = torch.where(m.inner[:, None], 0.5 * (left + right)[:, :2], right[:, :2])
        F = torch.stack([torch.zeros_like(txx), txx * m.nx + txy * m.ny, txy * m.nx + tyy * m.ny,
                         (uf[:, 0] * txx + uf[:, 1] * txy - q[:, 0]) * m.nx
                         + (uf[:, 0] * txy + uf[:, 1] * tyy - q[:, 1]) * m.ny], 1)
        R = m.residual((inv - torch.where(carries[:, None], F, torch.zeros_like(F))) * m.len[:, None])
        k = (0.5 * gap / (_speeds(m, W) + 2.0 * most / gap)).min() / m.vol
        history.append((R * R).sum(0).sqrt())
        if sa:
            vn = 0.5 * ((W[m.fl, 1] + WR[:, 1]) * m.nx + (W[m.fl, 2] + WR[:, 2]) * m.ny)
            adv = vn * torch.where(vn >= 0, left[:, 3], right[:, 3])
            dif = (0.5 * (nu[m.fl] + nu_r) + 0.5 * (nt[m.fl] + nt_r)) / (2.0 / 3.0) * dn[:, 3]
            Rn = m.residual((adv - torch.where(carries, dif, torch.zeros_like(dif))) * m.len)
            omega = (grad[:, 1, 0] - grad[:, 0, 1]).abs()
            Rn = Rn + m.vol * _sa_source(nut, nu, omega, walld, grad[:, 3])
            nut = nut + k * Rn
        U = U + k[:, None] * R
    return U, torch.stack(history), nut


def _adjoint(m, case, kinds, fs, U):
    """Residual, drag or lift with its gradient, and the pseudo-time adjoint iterations, limiter values held."""
    r, u, v, p = fs
    W = _prim(U)
    ext = torch.cat([W, 0.5 * (W[m.fl[m.bnd]] + _boundary(m, kinds, fs, W[m.fl[m.bnd]]))])
    psi = _limited(m, W, m.gradient(W, ext, "lsq"), ext, "venkat")
    free = [torch.tensor(x, dtype=torch.float64, device=m.dev, requires_grad=True) for x in fs]
    X = U.clone().requires_grad_()

    R = _euler_residual(m, case, kinds, free, X, psi)
    q = 0.5 * r * (u * u + v * v)
    wall = m.bnd[m.bpatch == 0]
    Y = U.clone().requires_grad_()
    pw = (_prim(Y)[m.fl[wall], 3] - p) * m.len[wall]
    fx, fy = (pw * m.nx[wall]).sum(), (pw * m.ny[wall]).sum()
    s = math.hypot(u, v)
    J = ((fx * u + fy * v) if case["objective"] == "drag" else (fy * u - fx * v)) / (s * q)
    g, = torch.autograd.grad(J, Y)
    k = _step_over_volume(m, W, 1.2, True)[:, None]
    back = lambda lam: torch.autograd.grad(R, X, lam, retain_graph=True)[0] - g  # noqa: E731
    lam, history = torch.zeros_like(U), []
    for _ in range(case["iterations"]):
        d = back(lam)
        history.append((d * d).sum(0).sqrt())
        nxt = lam + k * d
        nxt = 0.75 * lam + 0.25 * (nxt + k * back(nxt))
        lam = lam / 3.0 + (2.0 / 3.0) * (nxt + k * back(nxt))
    fsbar = torch.stack(torch.autograd.grad(R, free, lam))
    return R.detach(), J.detach(), g, lam, torch.stack([torch.zeros_like(fsbar), fsbar]), torch.stack(history)


def _diffusion(m, case, phi):
    h = 1.0 / case["nx"]
    dt, ob = 0.2 * h * h, m.fl[m.bnd]
    dist = (torch.where(m.inner[:, None], m.cen[m.fr], m.mid) - m.cen[m.fl]).norm(dim=1)
    held = (m.bpatch == 0) | (m.bpatch == 3)  # bottom, left: given values; right, top: given fluxes
    value = torch.where(m.bpatch == 0, 1.0, 0.5).to(phi)
    given = torch.where(m.bpatch == 1, -0.1, 0.1).to(phi) * m.len[m.bnd]
    history = []
    for _ in range(case["steps"]):
        flux = -(phi[m.fr] - phi[m.fl]) / dist * m.len
        flux[m.bnd] = torch.where(held, -(value - phi[ob]) / dist[m.bnd] * m.len[m.bnd], given)
        R = m.residual(flux)
        history.append((R * R).sum().sqrt())
        phi = phi + dt / m.vol * R
    return {"state": phi, "history": torch.stack(history)}


def exact(case, seed):
    kind = case["kind"]
    U0 = _start(case, seed)
    if kind == "batch":
        cases, polys, _ = _family(case["instances"], case["lo"], case["hi"])
        setup = {"steps": case["steps"], "order": 2, "rk": 3, "cfl": 1.2, "local_dt": True}
        states, norms, at = [], [], 0
        for c, poly in zip(cases, polys):
            m = _Geometry(poly)
            U = torch.as_tensor(U0[at:at + m.n], device=m.dev)
            at += m.n
            U, h = _euler_steps(m, setup, ["wall", "characteristic"], _freestream(c["mach"], c["aoa_deg"]), U)
            states.append(U.cpu())
            norms.append(h[-1].cpu())
        return {"state": torch.cat(states), "norms": torch.stack(norms)}
    poly = _case_poly(case)
    m = _Geometry(poly)
    U = torch.as_tensor(U0, device=m.dev)
    if kind == "diffusion":
        return _diffusion(m, case, U)
    fs = _freestream(case["mach"], case["aoa"])
    if kind == "euler":
        kinds = ["wall", "outflow", "wall", "outflow"] if case["mesh"] == "tube" else ["wall", "characteristic"]
        U, h = _euler_steps(m, case, kinds, fs, U)
        return {"state": U, "history": h}
    if kind == "adjoint":
        R, J, g, lam, fsbar, h = _adjoint(m, case, ["wall", "characteristic"], fs, U)
        return {"residual": R, "J": float(J), "dJdU": g, "lambda": lam, "fsbar": fsbar, "history": h}
    nut = torch.as_tensor(_start_nut(case, seed), device=m.dev) if kind == "rans" else None
    U, h, nut = _viscous_steps(m, poly, case, fs, U, nut)
    out = {"state": U, "history": h}
    if nut is not None:
        out["nut"] = nut
    return out
