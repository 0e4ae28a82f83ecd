"""The timed cases: what programs on this library do, through its public entry points.

A case is one pass of one of the example solvers or of the operator set:

* ``advection``   explicit upwind transport, many forward-Euler steps in one call;
* ``explicit``    every explicit operator once, as a program that forms its own
                  right-hand sides calls them;
* ``heat``        one implicit heat-conduction step (assembly, solve, boundary);
* ``cavity``      one PISO step of the lid-driven cavity (two pressure solves);
* ``convection``  one implicit upwind convection-diffusion step (BiCGStab);
* ``batch``       one implicit step of many uneven boxes packed into one system;
* ``serve``       a burst of requests through the serving loop, host to host.

``exact`` restates each pass with plain torch in 64 bits, every linear solve
carried to round-off, from the mesh arrays the program holds.
"""
from __future__ import annotations

import ctypes as C
import functools
import math
import time

import numpy as np
import torch

from foamadapter_gb300 import abi, apps, mesh, neon
from foamadapter_gb300.mesh import DeviceMesh

_PRECISION = {"fp64": abi.PREC_FP64, "mixed": abi.PREC_MIXED_IR}
_PRECOND = {"jacobi": abi.PRECOND_JACOBI, "multigrid": abi.PRECOND_MULTIGRID, "ilu": abi.PRECOND_ILU}
_P = abi.ptr


def listed():
    return [
        # the smallest calls: the 64 x 64 blob transport, 100 steps in one call
        {"name": "advection_64", "kind": "advection", "n": 64, "steps": 100},
        # a coarse 3-D mesh with odd edges: launch latency, ragged last slices and blocks
        {"name": "explicit_ragged", "kind": "explicit", "nx": 37, "ny": 29, "nz": 23, "jitter": 0.1},
        # the operator benchmark's mesh, larger than the L2 cache
        {"name": "explicit_128", "kind": "explicit", "nx": 128, "ny": 128, "nz": 128, "jitter": 0.1},
        # implicit heat conduction at scale, as OpenFOAM's PCG with a diagonal preconditioner runs it
        {"name": "heat_128_fp64", "kind": "heat", "nx": 128, "ny": 128, "nz": 128, "jitter": 0.1,
         "precision": "fp64", "precond": "jacobi"},
        # the same with the FP32 inner solve
        {"name": "heat_128_mixed", "kind": "heat", "nx": 128, "ny": 128, "nz": 128, "jitter": 0.1,
         "precision": "mixed", "precond": "jacobi"},
        # a tutorial-size cavity: many small calls per step
        {"name": "cavity_40_fp64", "kind": "cavity", "n": 40, "precision": "fp64", "precond": "jacobi"},
        # the cavity of the precision study, pressure in FP64, in mixed precision, and with GAMG's counterpart
        {"name": "cavity_512_fp64", "kind": "cavity", "n": 512, "precision": "fp64", "precond": "jacobi"},
        {"name": "cavity_512_mixed", "kind": "cavity", "n": 512, "precision": "mixed", "precond": "jacobi"},
        {"name": "cavity_512_multigrid", "kind": "cavity", "n": 512, "precision": "fp64", "precond": "multigrid"},
        # PBiCGStab + DILU, the pair OpenFOAM's transport equations name
        {"name": "convection_ilu", "kind": "convection", "nx": 77, "ny": 64, "nz": 58, "jitter": 0.1,
         "precision": "fp64", "precond": "ilu"},
        # a parameter study: uneven boxes (edges 16 to 64) advanced together
        {"name": "batch_48_mixed", "kind": "batch", "cases": 48, "precision": "mixed", "dims_seed": 4},
        # a burst of requests of different sizes through the serving loop
        {"name": "serve_16_mixed", "kind": "serve", "requests": 16, "max_edge": 96, "max_steps": 40,
         "precision": "mixed", "dims_seed": 5},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["advection", "explicit", "explicit", "heat", "heat", "cavity", "cavity", "convection",
                       "batch", "serve"])
    if kind == "advection":
        return {"kind": kind, "n": _log_int(rng, 24, 400), "steps": rng.choice([20, 50, 100])}
    if kind in ("explicit", "heat", "convection"):
        hi = 128 if kind != "convection" else 80
        c = {"kind": kind, "nx": _log_int(rng, 9, hi), "ny": _log_int(rng, 9, hi), "nz": _log_int(rng, 9, hi),
             "jitter": rng.choice([0.0, 0.1, 0.2])}
        if kind == "heat":
            c["precision"] = rng.choice(["fp64", "mixed"])
            c["precond"] = rng.choice(["jacobi", "jacobi", "multigrid"])
        if kind == "convection":
            c["precond"] = rng.choice(["jacobi", "ilu"])
            c["precision"] = "fp64" if c["precond"] == "ilu" else rng.choice(["fp64", "mixed"])
        return c
    if kind == "cavity":
        return {"kind": kind, "n": _log_int(rng, 20, 512), "precision": rng.choice(["fp64", "mixed"]),
                "precond": rng.choice(["jacobi", "jacobi", "multigrid"])}
    if kind == "batch":
        return {"kind": kind, "cases": _log_int(rng, 3, 48), "precision": rng.choice(["fp64", "mixed"]),
                "dims_seed": rng.randrange(1, 1000)}
    return {"kind": kind, "requests": _log_int(rng, 2, 16), "max_edge": _log_int(rng, 24, 96),
            "max_steps": rng.randrange(10, 40), "precision": rng.choice(["fp64", "mixed"]),
            "dims_seed": rng.randrange(1, 1000)}


# ------------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=3)
def _box(nx, ny, nz, jitter, two_d=False):
    """A hex box; its geometry is a function of the case, the fields on it of the seed."""
    if two_d:
        return mesh.box(nx, ny, 1, 1.0, 1.0, 1.0 / nx, jitter=jitter, seed=12345, two_d=True)
    return mesh.box(nx, ny, nz, jitter=jitter, seed=12345)


def _batch_dims(case):
    rng = np.random.default_rng(case["dims_seed"])
    return np.rint(np.exp(rng.uniform(np.log(16), np.log(64), size=(case["cases"], 3)))).astype(int)


@functools.lru_cache(maxsize=1)
def _packed(dims):
    return mesh.concat([mesh.box(*d, jitter=0.1, seed=400000 + k) for k, d in enumerate(dims)])


def _batch_mesh(case):
    return _packed(tuple(tuple(int(e) for e in d) for d in _batch_dims(case)))


def _requests(case, seed):
    """(nx, ny, nz, steps, U, D, dt, T_init): sizes from the case, physics and fields from the seed."""
    rd = np.random.default_rng(case["dims_seed"])
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(case["requests"]):
        e = np.rint(np.exp(rd.uniform(np.log(16), np.log(case["max_edge"]), size=3))).astype(int)
        steps = int(rd.integers(10, case["max_steps"] + 1))
        d = rng.standard_normal(3)
        U = d / np.linalg.norm(d) * rng.uniform(0.1, 2.0)
        D = float(np.exp(rng.uniform(np.log(1e-4), np.log(1e-2))))
        dt = 0.5 / float(e.max()) / float(np.linalg.norm(U))
        x, y, z = ((np.arange(k) + 0.5) / k for k in (e[0], e[1], e[2]))
        c = rng.uniform(0.3, 0.7, size=3)
        blob = (np.exp(-(x - c[0]) ** 2 / 0.02)[None, None, :] * np.exp(-(y - c[1]) ** 2 / 0.02)[None, :, None] *
                np.exp(-(z - c[2]) ** 2 / 0.02)[:, None, None])
        out.append((int(e[0]), int(e[1]), int(e[2]), steps, U, D, dt, np.ascontiguousarray(blob.reshape(-1))))
    return out


def _advection_inputs(case, seed):
    rng = np.random.default_rng(seed)
    a = rng.uniform(0.0, 2.0 * np.pi)
    speed = rng.uniform(0.5, 1.5)
    return ((speed * math.cos(a), speed * math.sin(a), 0.0), tuple(rng.uniform(0.25, 0.75, size=2)),
            0.05, 0.1 / case["n"] / speed)


def _explicit_inputs(case, seed):
    hm = _box(case["nx"], case["ny"], case["nz"], case["jitter"])
    rng = np.random.default_rng(seed)
    nf = hm.nif + hm.nbf
    return hm, dict(T=300.0 + rng.standard_normal(hm.n), U=rng.standard_normal((hm.n, 3)),
                    flux=rng.standard_normal(nf), gamma=np.exp(0.5 * rng.standard_normal(nf)),
                    wall=rng.uniform(350.0, 450.0))


def _heat_inputs(case, seed):
    hm = _box(case["nx"], case["ny"], case["nz"], case["jitter"])
    rng = np.random.default_rng(seed)
    return hm, np.exp(0.5 * rng.standard_normal(hm.n)), 300.0 + rng.standard_normal(hm.n), rng.uniform(350.0, 450.0)


def _cavity_inputs(case, seed):
    """A swirling flow under a moving lid."""
    hm = _box(case["n"], case["n"], 1, 0.05, True)
    rng = np.random.default_rng(seed)
    x, y = hm.C[:, 0], hm.C[:, 1]
    U = np.zeros((hm.n, 3))
    for k in range(1, 4):
        a = 0.2 * rng.standard_normal() / k
        U[:, 0] += a * np.sin(np.pi * x) ** 2 * np.sin(2 * k * np.pi * y)
        U[:, 1] -= a * np.sin(2 * np.pi * x) * np.sin(k * np.pi * y) ** 2
    return hm, U, (float(rng.uniform(0.5, 1.5)), 0.0, 0.0)


def _convection_inputs(case, seed):
    hm = _box(case["nx"], case["ny"], case["nz"], case["jitter"])
    rng = np.random.default_rng(seed)
    d = rng.standard_normal(3)
    U = d / np.linalg.norm(d) * rng.uniform(0.5, 1.5)
    dt = 2.0 / max(case["nx"], case["ny"], case["nz"]) / float(np.linalg.norm(U))
    return hm, U, dt, rng.random(hm.n)


def _batch_inputs(case, seed):
    big, ranges, slices = _batch_mesh(case)
    rng = np.random.default_rng(seed)
    ref, kappa = np.zeros(big.nbf), np.ones(big.n)
    for k in range(case["cases"]):
        ref[slices[k][0]] = rng.uniform(350.0, 450.0)
        lo, hi = int(ranges[2 * k]), int(ranges[2 * k + 1])
        kappa[lo:hi] = np.exp(0.5 * rng.standard_normal(hi - lo))
    xmin = slice(slices[0][0].start, slices[-1][0].stop)
    return big, ranges, kappa, ref[xmin]


# ------------------------------------------------------------------ programs
class _Advection:
    def __init__(self, case, seed):
        U, centre, sigma, dt = _advection_inputs(case, seed)
        self.app = apps.Advection(n=case["n"], U=U, centre=centre, sigma=sigma, dt=dt)
        self.steps = case["steps"]
        self.T0, self.Tb0 = self.app.T.internal.clone(), self.app.T.boundary.clone()

    def run(self):
        T = self.app.T
        T.internal.copy_(self.T0)
        T.boundary.copy_(self.Tb0)
        self.app.run(self.steps)
        return [T.internal, T.boundary]


class _Explicit:
    def __init__(self, case, seed):
        hm, a = _explicit_inputs(case, seed)
        self.dm = dm = DeviceMesh(hm)
        walls = [("zeroGradient", 0.0)] * (hm.npatch - 1)
        self.T = neon.VolumeField(dm, a["T"], [("fixedValue", a["wall"])] + walls)
        self.U = neon.VolumeField(dm, a["U"], [("fixedValue", [1.0, 0.0, 0.0])] + walls, ncomp=3)
        self.flux, self.gamma = neon.SurfaceField(dm, a["flux"]), neon.SurfaceField(dm, a["gamma"])
        self.faces = [neon.SurfaceField(dm) for _ in range(4)]
        zeros = lambda k: torch.zeros(k * hm.n, dtype=torch.float64, device="cuda")
        self.cells = [zeros(1), zeros(1), zeros(3), zeros(3), zeros(1), zeros(1)]

    def run(self):
        dm, T, U, flux, gamma = self.dm, self.T, self.U, self.flux, self.gamma
        lin, up, sn, snc = self.faces
        for c in self.cells:  # the operators accumulate
            c.zero_()
        dl, du, dv, g, lap, lapc = self.cells
        neon.SurfaceInterpolation(dm, "linear").interpolate(T, lin)
        neon.SurfaceInterpolation(dm, "upwind").interpolate(T, up, flux=flux)
        neon.GaussGreenDiv(dm, "linear").div(dl, flux, T)
        neon.GaussGreenDiv(dm, "upwind").div(du, flux, T)
        neon.GaussGreenDiv(dm, "linear").div(dv, flux, U)
        neon.GaussGreenGrad(dm).grad(T, 1.0, g)
        neon.GaussGreenLaplacian(dm).laplacian(lap, gamma, T)
        neon.GaussGreenLaplacian(dm, "Gauss linear corrected").laplacian(lapc, gamma, T)
        neon.FaceNormalGradient(dm).faceNormalGrad(T, sn)
        neon.FaceNormalGradient(dm, "corrected").faceNormalGrad(T, snc)
        return [f.values for f in self.faces] + list(self.cells)


class _Heat:
    def __init__(self, case, seed):
        hm, kappa, T0, wall = _heat_inputs(case, seed)
        self.app = apps.HeatTransfer(hm, kappa, T0=0.0, Twall=wall, precision=_PRECISION[case["precision"]])
        self.app.cfg.preconditioner = _PRECOND[case["precond"]]
        self.T0 = neon.dev(T0)

    def run(self):
        T = self.app.T
        T.internal.copy_(self.T0)
        T.correctBoundaryConditions()
        self.app.step()
        return [T.internal, T.boundary]


class _Cavity:
    def __init__(self, case, seed):
        hm, U, lid = _cavity_inputs(case, seed)
        self.app = a = apps.CavityPiso(n=case["n"], lid=lid, dt=_cavity_dt(case), precision=_PRECISION[case["precision"]],
                                       preconditioner=_PRECOND[case["precond"]])
        self.U0 = neon.dev(U.reshape(-1))
        a.U.internal.copy_(self.U0)
        abi.check(abi.lib().fvgb_flux_vec(a.dm.handle, _P(a.U.internal), _P(a.U.boundary), _P(a.phi.values),
                                          torch.cuda.current_stream().cuda_stream))
        self.phi0 = a.phi.values.clone()

    def run(self):
        a = self.app
        a.U.internal.copy_(self.U0)
        a.U.correctBoundaryConditions()
        a.p.internal.zero_()
        a.p.correctBoundaryConditions()
        a.phi.values.copy_(self.phi0)
        a.step()
        return [a.U.internal, a.p.internal, a.phi.values]


def _cavity_dt(case):
    return 0.25 / case["n"]


class _Convection:
    def __init__(self, case, seed):
        hm, U, self.dt, T0 = _convection_inputs(case, seed)
        self.dm = dm = DeviceMesh(hm)
        self.F = neon.SurfaceField(dm)
        Uc, Ub = neon.dev(np.tile(U, hm.n)), neon.dev(np.tile(U, hm.nbf))
        abi.check(abi.lib().fvgb_flux_vec(dm.handle, _P(Uc), _P(Ub), _P(self.F.values),
                                          torch.cuda.current_stream().cuda_stream))
        self.T = neon.VolumeField(dm, T0, [("fixedValue", 1.0)] + [("zeroGradient", 0.0)] * (hm.npatch - 1), name="T")
        self.old = self.T.internal.clone()
        D = neon.SurfaceField(dm, np.full(hm.nif + hm.nbf, 1e-3))
        self.ls = neon.LinearSystem(dm)
        self.terms = [neon.ddt(self.old), neon.div(self.F, "upwind"), neon.laplacian(D, -1.0)]
        self.kw = dict(method=abi.SOLVER_BICGSTAB, precision=_PRECISION[case["precision"]],
                       preconditioner=_PRECOND[case["precond"]], max_iter=5000)

    def run(self):
        T = self.T
        T.internal.copy_(self.old)
        T.correctBoundaryConditions()
        self.ls.assemble(self.terms, self.dt, T)
        self.ls.solve(T.internal, **self.kw)
        T.correctBoundaryConditions()
        return [T.internal, T.boundary]


class _Batch:
    def __init__(self, case, seed):
        big, ranges, kappa, ref = _batch_inputs(case, seed)
        self.dm = dm = DeviceMesh(big)
        walls = [("zeroGradient", 0.0)] * 5
        self.T = neon.VolumeField(dm, np.full(big.n, 300.0), [("fixedValue", ref)] + walls, name="T")
        k = neon.VolumeField(dm, kappa, [("zeroGradient", 0.0)] * 6)
        self.gamma = neon.SurfaceInterpolation(dm, "linear").interpolate(k)
        self.old = torch.empty_like(self.T.internal)
        self.ls = neon.LinearSystem(dm)
        self.batch = neon.Batch(self.ls, ranges)
        self.terms = [neon.ddt(self.old), neon.laplacian(self.gamma, -1.0)]
        self.kw = dict(precision=_PRECISION[case["precision"]], inner_rel_tol=0.1, inner_max_iter=2000, max_iter=4000)

    def run(self):
        T = self.T
        T.internal.fill_(300.0)
        T.correctBoundaryConditions()
        self.old.copy_(T.internal)
        self.ls.assemble(self.terms, 0.01, T)
        self.batch.solve(T.internal, **self.kw)
        T.correctBoundaryConditions()
        return [T.internal, T.boundary]


class _Serve:
    def __init__(self, case, seed):
        self.reqs = _requests(case, seed)
        self.precision = _PRECISION[case["precision"]]
        cfg = abi.ServerCfg(int(20e9), 64, 16)
        self.server = C.c_void_p()
        abi.check(abi.lib().fvgb_server_create(C.byref(cfg), C.byref(self.server)))

    def run(self):
        L, sv = abi.lib(), self.server
        outs, waiting = [], set()
        for nx, ny, nz, steps, U, D, dt, T_init in self.reqs:
            T = np.empty_like(T_init)
            req = abi.ServeRequest(nx=nx, ny=ny, nz=nz, steps=steps, U=(C.c_double * 3)(*U), D=D, dt=dt,
                                   precision=self.precision, kernel_mode=0, flags=0, T_out=_P(T), T_init=_P(T_init))
            rid = C.c_int64()
            abi.check(L.fvgb_server_submit(sv, C.byref(req), C.byref(rid)))
            outs.append(T)
            waiting.add(rid.value)
        buf, cnt = (abi.ServeResult * 64)(), C.c_int32()
        while waiting:
            abi.check(L.fvgb_server_poll(sv, buf, 64, C.byref(cnt)))
            for i in range(cnt.value):
                abi.check(buf[i].status)
                waiting.discard(buf[i].id)
            time.sleep(0.0002)
        return outs

    def __del__(self):
        try:
            abi.lib().fvgb_server_destroy(self.server)
        except Exception:
            pass


_PROGRAM = {"advection": _Advection, "explicit": _Explicit, "heat": _Heat, "cavity": _Cavity,
            "convection": _Convection, "batch": _Batch, "serve": _Serve}


def prepare(case, seed):
    return _PROGRAM[case["kind"]](case, seed)


def run(state):
    return state.run()


# ---------------------------------------------------------------------- work
def _box_counts(nx, ny, nz):
    n = nx * ny * nz
    return n, (nx - 1) * ny * nz + nx * (ny - 1) * nz + nx * ny * (nz - 1), 2 * (nx * ny + ny * nz + nx * nz)


def _solve_work(n, nif, iters, spmvs=1):
    """One implicit step: geometry, coefficients and old field in, the new field out;
    an iteration is `spmvs` products with the matrix and 12 operations a row beside each."""
    nnz = n + 2 * nif
    return {"bytes": 8 * (2 * nif + 4 * n) + 8 * nif, "flops": iters * spmvs * (2 * nnz + 12 * n)}


def work(case):
    k = case["kind"]
    if k == "advection":
        n = case["n"] ** 2
        nif = 2 * case["n"] * (case["n"] - 1)
        return {"bytes": 16 * nif + 24 * n, "flops": case["steps"] * (3 * nif + 4 * n)}
    if k == "explicit":
        n, nif, nbf = _box_counts(case["nx"], case["ny"], case["nz"])
        # every array once: owner, neighbour, Sf, |Sf|, w, delta, correction vectors, flux and gamma; T, U, V,
        # the centres' boundary data; four face fields and ten cell components written
        return {"bytes": nif * (8 + 24 + 3 * 8 + 24 + 16 + 32) + nbf * 120 + n * 8 * (5 + 10),
                "flops": nif * (3 + 6 + 3 + 18 + 12 + 5 + 28 + 2 + 26) + 40 * n}
    if k in ("heat", "convection"):
        n, nif, _ = _box_counts(case["nx"], case["ny"], case["nz"])
        edge = max(case["nx"], case["ny"], case["nz"])
        if k == "convection":
            return _solve_work(n, nif, 6 if case["precond"] == "ilu" else 28, 2)
        return _solve_work(n, nif, 33 if case["precond"] == "multigrid" else 2.4 * edge)
    if k == "cavity":
        n = case["n"] ** 2
        nif = 2 * case["n"] * (case["n"] - 1)
        w = _solve_work(n, nif, 2 * (70 if case["precond"] == "multigrid" else 6 * case["n"]))
        return {"bytes": w["bytes"] + 8 * (9 * nif + 12 * n), "flops": w["flops"] + 60 * (nif + n)}
    if k == "batch":
        counts = [_box_counts(*d) for d in _batch_dims(case).tolist()]
        edges = [max(d) for d in _batch_dims(case).tolist()]
        ws = [_solve_work(n, nif, 2.4 * e) for (n, nif, _), e in zip(counts, edges)]
        return {q: sum(w[q] for w in ws) for q in ("bytes", "flops")}
    ws = []
    for nx, ny, nz, steps, *_ in _requests(case, 0):
        n, nif, _ = _box_counts(nx, ny, nz)
        w = _solve_work(n, nif, 7 * steps)
        ws.append({"bytes": w["bytes"], "flops": w["flops"] + steps * 6 * nif})
    return {q: sum(w[q] for w in ws) for q in ("bytes", "flops")}


# --------------------------------------------------------------------- exact
class _Ref:
    """A mesh's arrays and the face-loop operators in plain torch, 64 bits."""

    def __init__(self, hm):
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a)).cuda()
        self.n, self.nif, self.nbf = hm.n, hm.nif, hm.nbf
        self.P, self.N, self.B = t(hm.own).long(), t(hm.nei).long(), t(hm.bcells).long()
        self.V, self.C, self.w = t(hm.V), t(hm.C), t(hm.w)
        self.Sf, self.mag, self.delta = t(hm.Sf), t(hm.magSf), t(hm.delta)
        self.bSf, self.bmag, self.bdelta = t(hm.bSf), t(hm.bmagSf), t(hm.bdelta)
        self.corr = self.Sf / self.mag[:, None] - (self.C[self.N] - self.C[self.P]) * self.delta[:, None]

    def lin(self, x):
        w = self.w if x.dim() == 1 else self.w[:, None]
        return w * (x[self.P] - x[self.N]) + x[self.N]

    def faces(self, x, xb):
        return torch.cat([self.lin(x), xb])

    def gather(self, f):
        """Sum of a face quantity over each cell's faces, outward."""
        out = torch.zeros((self.n,) + f.shape[1:], dtype=torch.float64, device=f.device)
        out.index_add_(0, self.P, f[:self.nif])
        out.index_add_(0, self.N, -f[:self.nif])
        out.index_add_(0, self.B, f[self.nif:])
        return out

    def flux(self, U, Ub):
        return torch.cat([(self.Sf * self.lin(U)).sum(1), (self.bSf * Ub).sum(1)])

    def upwind(self, F, x, xb):
        return torch.cat([torch.where(F[:self.nif] >= 0, x[self.P], x[self.N]), xb])

    def grad(self, x, xb):
        S = torch.cat([self.Sf, self.bSf])
        return self.gather(S * self.faces(x, xb)[:, None]) / self.V[:, None]

    def sngrad(self, x, xb):
        return torch.cat([self.delta * (x[self.N] - x[self.P]), self.bdelta * (xb - x[self.B])])

    def correction(self, x, xb):
        """Non-orthogonal part of the face-normal gradient (none on the boundary)."""
        g = self.lin(self.grad(x, xb))
        return torch.cat([(self.corr * g).sum(1), torch.zeros_like(xb)])

    def mags(self):
        return torch.cat([self.mag, self.bmag])

    def fixed(self, hm, values):
        """1 on the faces of the fixed-value patches, and the values there."""
        m, v = torch.zeros(self.nbf, dtype=torch.float64), torch.zeros(self.nbf, dtype=torch.float64)
        for name, val in values.items():
            m[hm.patch_slice(name)] = 1.0
            v[hm.patch_slice(name)] = torch.as_tensor(val, dtype=torch.float64)
        return m.cuda(), v.cuda()


class _Matrix:
    """diagonal, a_PN (row owner) and a_NP (row neighbour) of a system, and its solves."""

    def __init__(self, ref):
        z = lambda k: torch.zeros(k, dtype=torch.float64, device="cuda")
        self.r, self.d, self.up, self.lo = ref, z(ref.n), z(ref.nif), z(ref.nif)

    def laplacian(self, gamma, fixed, sign):
        """sign * laplacian(gamma, .); returns what the fixed values put on the right-hand side."""
        r = self.r
        g = sign * gamma[:r.nif] * r.mag * r.delta
        gb = sign * gamma[r.nif:] * r.bmag * r.bdelta * fixed
        self.up += g
        self.lo += g
        self.d.index_add_(0, r.P, -g)
        self.d.index_add_(0, r.N, -g)
        self.d.index_add_(0, r.B, -gb)
        return gb

    def div(self, F, wP, fixed):
        """div(F, .) with owner weight wP; zero-gradient faces take the cell value."""
        r = self.r
        Fi, Fb = F[:r.nif], F[r.nif:]
        self.d.index_add_(0, r.P, Fi * wP)
        self.up += Fi * (1 - wP)
        self.d.index_add_(0, r.N, -Fi * (1 - wP))
        self.lo += -Fi * wP
        self.d.index_add_(0, r.B, Fb * (1 - fixed))

    def off(self, x):
        """The off-diagonal part times x (scalar or vector)."""
        r = self.r
        ex = (lambda a: a) if x.dim() == 1 else (lambda a: a[:, None])
        y = torch.zeros_like(x)
        y.index_add_(0, r.P, ex(self.up) * x[r.N])
        y.index_add_(0, r.N, ex(self.lo) * x[r.P])
        return y

    def csr(self):
        r = self.r
        i = torch.arange(r.n, device="cuda")
        idx = torch.stack([torch.cat([i, r.P, r.N]), torch.cat([i, r.N, r.P])])
        return torch.sparse_coo_tensor(idx, torch.cat([self.d, self.up, self.lo]), (r.n, r.n)).coalesce().to_sparse_csr()

    def solve(self, b, x, symmetric=True, tol=1e-13, max_iter=30000):
        """Jacobi CG or BiCGStab to round-off, the residual formed again from x at the end of each run."""
        A, di = self.csr(), 1.0 / self.d
        mv = lambda v: torch.mv(A, v)
        x, scale = x.clone(), None
        for _ in range(4):
            r = b - mv(x)
            res = float(r.norm())
            scale = res if scale is None else scale
            if res <= tol * scale or scale == 0.0:
                break
            x = x + (self._cg if symmetric else self._bicgstab)(mv, di, r, tol * scale, max_iter)
        return x

    @staticmethod
    def _cg(mv, di, r, stop, max_iter):
        x, z = torch.zeros_like(r), di * r
        p, rz = z.clone(), torch.dot(r, z)
        for it in range(max_iter):
            q = mv(p)
            a = rz / torch.dot(p, q)
            x += a * p
            r = r - a * q
            z = di * r
            rz, old = torch.dot(r, z), rz
            p = z + (rz / old) * p
            if it % 25 == 24 and not float(r.norm()) > stop:
                break
        return x

    @staticmethod
    def _bicgstab(mv, di, r, stop, max_iter):
        x, rr, p = torch.zeros_like(r), r.clone(), r.clone()
        rho = torch.dot(rr, r)
        for it in range(max_iter):
            y = di * p
            v = mv(y)
            a = rho / torch.dot(rr, v)
            s = r - a * v
            if not float(s.norm()) > stop:
                return x + a * y
            z = di * s
            t = mv(z)
            om = torch.dot(t, s) / torch.dot(t, t)
            x += a * y + om * z
            r = s - om * t
            if not float(r.norm()) > stop:
                break
            rho, old = torch.dot(rr, r), rho
            p = r + (rho / old) * (a / om) * (p - om * v)
        return x


def _exact_advection(case, seed):
    U, centre, sigma, dt = _advection_inputs(case, seed)
    hm = _box(case["n"], case["n"], 1, 0.0, True)
    r = _Ref(hm)
    x, y = r.C[:, 0], r.C[:, 1]
    T = torch.exp(-((x - centre[0]) ** 2 + (y - centre[1]) ** 2) / (2 * sigma ** 2))
    Uc = torch.tensor(U, dtype=torch.float64, device="cuda")
    F = torch.cat([(r.Sf * Uc).sum(1), (r.bSf * Uc).sum(1)])
    for _ in range(case["steps"]):
        T = T - dt * r.gather(F * r.upwind(F, T, T[r.B])) / r.V
    return [T, T[r.B]]


def _exact_explicit(case, seed):
    hm, a = _explicit_inputs(case, seed)
    r = _Ref(hm)
    t = lambda v: torch.as_tensor(v).cuda()
    T, U, F, g = t(a["T"]), t(a["U"]), t(a["flux"]), t(a["gamma"])
    m, v = r.fixed(hm, {"xmin": a["wall"]})
    Tb = m * v + (1 - m) * T[r.B]
    Ub = (1 - m)[:, None] * U[r.B]
    Ub[:, 0] += m
    Tf, up = r.faces(T, Tb), r.upwind(F, T, Tb)
    sn = r.sngrad(T, Tb)
    snc = sn + r.correction(T, Tb)
    gm = g * r.mags()
    return [Tf, up, sn, snc, r.gather(F * Tf) / r.V, r.gather(F * up) / r.V,
            (r.gather(F[:, None] * r.faces(U, Ub)) / r.V[:, None]).reshape(-1), r.grad(T, Tb).reshape(-1),
            r.gather(gm * sn) / r.V, r.gather(gm * snc) / r.V]


def _heat_step(hm, r, kappa, T0, fixed, wall, dt):
    gamma = r.faces(kappa, kappa[r.B])
    A = _Matrix(r)
    gb = A.laplacian(gamma, fixed, -1.0)
    A.d += r.V / dt
    b = r.V / dt * T0
    b.index_add_(0, r.B, -gb * wall)
    T = A.solve(b, T0)
    return [T, fixed * wall + (1 - fixed) * T[r.B]]


def _exact_heat(case, seed):
    hm, kappa, T0, wall = _heat_inputs(case, seed)
    r = _Ref(hm)
    m, v = r.fixed(hm, {"xmin": wall})
    return _heat_step(hm, r, torch.as_tensor(kappa).cuda(), torch.as_tensor(T0).cuda(), m, v, 0.01)


def _exact_batch(case, seed):
    big, _, kappa, ref = _batch_inputs(case, seed)
    r = _Ref(big)
    m, v = r.fixed(big, {"xmin": ref})
    T0 = torch.full((big.n,), 300.0, dtype=torch.float64, device="cuda")
    return _heat_step(big, r, torch.as_tensor(kappa).cuda(), T0, m, v, 0.01)


def _exact_convection(case, seed):
    hm, U, dt, T0 = _convection_inputs(case, seed)
    r = _Ref(hm)
    m, v = r.fixed(hm, {"xmin": 1.0})
    Uc, T0 = torch.as_tensor(U).cuda(), torch.as_tensor(T0).cuda()
    F = torch.cat([(r.Sf * Uc).sum(1), (r.bSf * Uc).sum(1)])
    A = _Matrix(r)
    A.d += r.V / dt
    A.div(F, (F[:r.nif] >= 0).double(), m)
    gb = A.laplacian(torch.full_like(F, 1e-3), m, -1.0)
    b = r.V / dt * T0
    b.index_add_(0, r.B, -(F[r.nif:] * m + gb) * v)
    T = A.solve(b, T0, symmetric=False)
    return [T, m * v + (1 - m) * T[r.B]]


def _exact_cavity(case, seed):
    hm, U, lid = _cavity_inputs(case, seed)
    r, dt = _Ref(hm), _cavity_dt(case)
    U = torch.as_tensor(U).cuda()
    Ub = torch.zeros((r.nbf, 3), dtype=torch.float64, device="cuda")
    Ub[hm.patch_slice("ymax")] = torch.tensor(lid, dtype=torch.float64, device="cuda")
    ones, none = torch.ones_like(r.bmag), torch.zeros_like(r.bmag)
    phi = r.flux(U, Ub)
    A = _Matrix(r)
    A.d += r.V / dt
    A.div(phi, r.w, ones)
    gb = A.laplacian(torch.full_like(phi, 0.01), ones, -1.0)
    b = (r.V / dt)[:, None] * U
    b.index_add_(0, r.B, -(phi[r.nif:] + gb)[:, None] * Ub)
    p = torch.zeros_like(r.V)
    for _ in range(2):
        rAU = r.V / A.d
        H = (b - A.off(U)) / A.d[:, None]
        rAUf = r.faces(rAU, rAU[r.B])
        phiH = r.flux(H, Ub)
        M = _Matrix(r)
        M.laplacian(rAUf, none, 1.0)
        M.d[0] *= 2.0
        p = M.solve(r.gather(phiH), p)
        phi = phiH.clone()
        phi[:r.nif] -= M.up * (p[r.N] - p[r.P])
        U = H - rAU[:, None] * r.grad(p, p[r.B])
    return [U.reshape(-1), p, phi]


def _exact_serve(case, seed):
    out = []
    for nx, ny, nz, steps, U, D, dt, T_init in _requests(case, seed):
        r = _Ref(mesh.box(nx, ny, nz))
        Uc, T = torch.as_tensor(U).cuda(), torch.as_tensor(T_init).cuda()
        F = torch.cat([(r.Sf * Uc).sum(1), (r.bSf * Uc).sum(1)])
        A = _Matrix(r)
        A.d += r.V / dt
        A.laplacian(torch.full_like(F, D), torch.zeros_like(r.bmag), -1.0)
        M, di = A.csr(), 1.0 / A.d
        for _ in range(steps):
            b = r.V / dt * T - r.gather(F * r.upwind(F, T, T[r.B]))
            res = b - torch.mv(M, T)
            stop = 1e-13 * float(res.norm())
            T = T + _Matrix._cg(lambda v: torch.mv(M, v), di, res, stop, 2000)
        out.append(T)
    return out


_EXACT = {"advection": _exact_advection, "explicit": _exact_explicit, "heat": _exact_heat, "cavity": _exact_cavity,
          "convection": _exact_convection, "batch": _exact_batch, "serve": _exact_serve}


def exact(case, seed):
    return _EXACT[case["kind"]](case, seed)
