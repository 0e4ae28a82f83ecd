"""fvgb_advect_euler_steps against as many single steps, bit for bit.

Calls of four or more steps on meshes of at most one 1024-thread block per SM run
one kernel whose blocks exchange their neighbouring cells step by step; the sizes
sit at its block sizes' edges (128, 256, 512, 1024 threads), below its fewest steps
and beyond its largest mesh.  Flows in one direction only, random fluxes, every
boundary condition and a random cell numbering (neighbours in every block).
"""
import ctypes as C
import threading

import numpy as np
import pytest
import torch

from foamadapter_gb300 import abi, mesh, neon
from foamadapter_gb300.mesh import DeviceMesh
from test_gpu_resident import renumber

pytestmark = pytest.mark.gpu


def run(hm, flux, T0, bcs, nsteps, dt):
    dm = DeviceMesh(hm)
    F = neon.SurfaceField(dm, flux)
    L, s = abi.lib(), torch.cuda.current_stream().cuda_stream
    one, many = (neon.VolumeField(dm, T0, bcs) for _ in range(2))
    bc = one.bc_struct()
    w, wb = torch.empty_like(one.internal), torch.empty_like(one.boundary)
    abi.check(L.fvgb_advect_euler_steps(dm.handle, abi.ptr(F.values), abi.ptr(many.internal), abi.ptr(many.boundary), dt,
                                        C.byref(many.bc_struct()), nsteps, abi.ptr(w), abi.ptr(wb), s))
    a, ab, b, bb = one.internal, one.boundary, torch.empty_like(one.internal), torch.empty_like(one.boundary)
    for _ in range(nsteps):
        abi.check(L.fvgb_advect_euler_step(dm.handle, abi.ptr(F.values), abi.ptr(a), abi.ptr(ab), dt, C.byref(bc),
                                           abi.ptr(b), abi.ptr(bb), s))
        a, b, ab, bb = b, a, bb, ab
    np.testing.assert_array_equal(many.internal.cpu().numpy(), a.cpu().numpy())
    np.testing.assert_array_equal(many.boundary.cpu().numpy()[:hm.nbf], ab.cpu().numpy()[:hm.nbf])


@pytest.mark.parametrize("n,nsteps", [(1, 5), (11, 7), (12, 100), (64, 3), (64, 4), (64, 101), (139, 12), (140, 9),
                                      (198, 8), (279, 6), (394, 5), (395, 5)])
def test_uniform_flow(cuda, n, nsteps):
    hm = mesh.box(n, n, 1, 1.0, 1.0, 1.0 / n, two_d=True)
    U = np.array([1.0, 0.5, 0.0])
    flux = np.concatenate([hm.Sf @ U, hm.bSf @ U])
    T0 = np.random.default_rng(1).random(hm.n)
    run(hm, flux, T0, [("zeroGradient", 0.0)] * hm.npatch, nsteps, 0.3 / n)


@pytest.mark.parametrize("dims,shuffled", [((7, 5, 3), False), ((31, 23, 17), False), ((31, 23, 17), True),
                                           ((61, 47, 40), True)])
def test_random_flux_and_boundaries(cuda, dims, shuffled):
    hm = mesh.box(*dims, jitter=0.1, seed=5)
    if shuffled:
        hm = renumber(hm, 9)
    rng = np.random.default_rng(2)
    flux = rng.standard_normal(hm.nif + hm.nbf) * 1e-3
    flux[::17] = 0.0
    flux[5::31] = -0.0
    nz = hm.bdelta.size // hm.npatch
    bcs = [("fixedValue", 3.0), ("fixedGradient", 0.7), ("zeroGradient", 0.0), ("calculated", 0.0),
           ("fixedValue", -1.0), ("zeroGradient", 0.0)]
    assert nz
    T0 = rng.standard_normal(hm.n)
    T0[::13] = 0.0
    run(hm, flux, T0, bcs, 25, 1e-2)


def test_calls_on_two_threads(cuda):
    """Two meshes whose blocks (384 and 512 threads) are launched from the same kernel,
    each advanced on a thread and stream of its own."""
    L = abi.lib()

    def case(dims):
        hm = mesh.box(*dims)
        dm = DeviceMesh(hm)
        rng = np.random.default_rng(4)
        F = neon.SurfaceField(dm, rng.standard_normal(hm.nif + hm.nbf) * 1e-3)
        T = neon.VolumeField(dm, rng.standard_normal(hm.n), [("zeroGradient", 0.0)] * hm.npatch)
        return dm, F, T, T.internal.clone(), T.boundary.clone(), torch.empty_like(T.internal), torch.empty_like(T.boundary)

    def call(c, stream):
        dm, F, T, _, _, w, wb = c
        bc = T.bc_struct()
        return lambda: L.fvgb_advect_euler_steps(dm.handle, abi.ptr(F.values), abi.ptr(T.internal), abi.ptr(T.boundary),
                                                 1e-2, C.byref(bc), 4, abi.ptr(w), abi.ptr(wb), stream.cuda_stream)

    def restore(c):
        c[2].internal.copy_(c[3])
        c[2].boundary.copy_(c[4])
        torch.cuda.synchronize()

    cases = [case(d) for d in ((40, 36, 33), (60, 40, 30), (40, 36, 33), (60, 40, 30))]
    streams = [torch.cuda.Stream() for _ in cases]
    calls = [call(c, s) for c, s in zip(cases, streams)]
    want = []
    for c, f in zip(cases, calls):
        assert f() == abi.OK
        torch.cuda.synchronize()
        want.append(c[2].internal.clone())
        restore(c)
    bad = []

    def loop(f):
        for _ in range(5000):
            if f() != abi.OK:
                bad.append(abi.lib().fvgb_last_error())
                return

    threads = [threading.Thread(target=loop, args=(f,)) for f in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not bad
    for c, f, w in zip(cases, calls, want):
        restore(c)
        assert f() == abi.OK
        torch.cuda.synchronize()
        assert torch.equal(c[2].internal, w)
