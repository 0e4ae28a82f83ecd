"""The resident single-case solves (one block per SM, kernel_mode 2) against the
graph of kernels, bit for bit: iterates, counts and residual norms.

Sizes at the edges of the kernel's layout: one row, a partial slice, one block
more and less, the switch of rows per thread (2^15), the largest system with
one block per SM and the first one beyond it (which takes the grid-barrier
kernel).  Numberings: the box's own, and a random one in which almost every
matrix slot reaches into another block (it fits the shared memory with 4 rows
per thread and does not with 8).
"""
import ctypes as C
import time

import numpy as np
import pytest
import torch

from foamadapter_gb300 import abi, mesh, neon
from foamadapter_gb300.mesh import DeviceMesh

pytestmark = pytest.mark.gpu


def renumber(hm, seed):
    """The same mesh under a random cell numbering, faces back in upper-triangular order."""
    perm = np.random.default_rng(seed).permutation(hm.n).astype(np.int32)
    inv = np.argsort(perm)
    o, n = perm[hm.own], perm[hm.nei]
    flip = o > n
    own, nei = np.where(flip, n, o).astype(np.int32), np.where(flip, o, n).astype(np.int32)
    order = np.lexsort((nei, own))
    hm.own, hm.nei = np.ascontiguousarray(own[order]), np.ascontiguousarray(nei[order])
    hm.Sf = np.ascontiguousarray(np.where(flip[:, None], -hm.Sf, hm.Sf)[order])
    hm.w = np.ascontiguousarray(np.where(flip, 1.0 - hm.w, hm.w)[order])
    for k in ("Cf", "magSf", "delta"):
        setattr(hm, k, np.ascontiguousarray(getattr(hm, k)[order]))
    hm.V, hm.C = np.ascontiguousarray(hm.V[inv]), np.ascontiguousarray(hm.C[inv])
    hm.bcells = np.ascontiguousarray(perm[hm.bcells])
    return hm


def system(dims, shuffled=False, two_d=False, dt=0.05):
    hm = mesh.box(*dims, 1.0, 1.0, 1.0 / max(dims) if two_d else 1.0, jitter=0.1, seed=7, two_d=two_d)
    if shuffled:
        hm = renumber(hm, 3)
    rng = np.random.default_rng(11)
    dm = DeviceMesh(hm)
    T = neon.VolumeField(dm, 300.0 + rng.standard_normal(hm.n),
                         [("fixedValue", 400.0)] + [("zeroGradient", 0.0)] * (hm.npatch - 1))
    g = neon.SurfaceField(dm, np.exp(0.5 * rng.standard_normal(hm.nif + hm.nbf)))
    ls = neon.LinearSystem(dm)
    ls.assemble([neon.ddt(T.internal.clone()), neon.laplacian(g, -1.0)], dt, T)
    return hm, T, ls


DIMS = [
    ((5, 5, 5), False, False), ((16, 8, 1), False, True), ((127, 1, 1), False, False), ((129, 1, 1), False, False),
    ((16, 16, 8), False, False), ((13, 13, 13), True, False), ((64, 64, 1), False, True), ((17, 241, 1), False, True),
    ((1, 1, 1), False, False), ((7, 3, 1), False, False), ((11, 31, 3), False, False), ((32, 32, 1), False, True),
    ((25, 41, 1), False, True), ((19, 23, 29), False, False), ((17, 17, 17), True, False),
    ((47, 41, 17), False, False), ((32, 32, 32), False, False), ((36, 34, 31), True, False),
    ((128, 128, 19), False, False), ((512, 608, 1), False, True), ((129, 128, 19), False, False),
]


@pytest.mark.parametrize("dims,shuffled,two_d", DIMS)
@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED_IR])
def test_resident_equals_graph(cuda, dims, shuffled, two_d, precision):
    hm, T, ls = system(dims, shuffled, two_d)
    kw = dict(rel_tol=1e-9, max_iter=400, precision=precision, inner_rel_tol=0.1)
    out = []
    for mode in (1, 2, 2):
        x = T.internal.clone()
        st = ls.solve(x, kernel_mode=mode, **kw)
        out.append((x.cpu().numpy(), st.num_iter, st.num_outer, st.init_res_norm, st.final_res_norm, st.status))
    for o in out[1:]:
        assert o[1:] == out[0][1:]
        np.testing.assert_array_equal(o[0], out[0][0])


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED_IR])
def test_resident_stopping(cuda, precision):
    """Iteration caps 0 and 3, an absolute tolerance met at the start, the ||b|| baseline
    and a zero residual stop the resident solve where they stop the graph."""
    hm, T, ls = system((19, 23, 29))
    solved = T.internal.clone()
    ls.solve(solved, rel_tol=1e-12, max_iter=2000)
    for kw in (dict(rel_tol=1e-9, max_iter=0), dict(rel_tol=1e-9, max_iter=3), dict(rel_tol=0.0, abs_tol=1e30),
               dict(rel_tol=1e-6, flags=abi.SOLVE_RHS_BASELINE), dict(rel_tol=1e-30, max_iter=60)):
        for start in (T.internal, solved):
            out = []
            for mode in (1, 2):
                x = start.clone()
                st = ls.solve(x, kernel_mode=mode, precision=precision, max_outer=6, **kw)
                out.append((x.cpu().numpy(), st.num_iter, st.num_outer, st.init_res_norm, st.final_res_norm,
                            st.status))
            assert out[0][1:] == out[1][1:], kw
            np.testing.assert_array_equal(out[0][0], out[1][0])


def test_resident_solves_on_two_streams(cuda):
    """Two systems solved asynchronously on two streams give their own bits."""
    systems = [system((19, 23, 29)), system((47, 41, 17))]
    cfg = abi.SolverCfg(1e-9, 0.0, 400, abi.PREC_FP64, 0.1, 1000, 50, 2)
    want = []
    for _, T, ls in systems:
        x = T.internal.clone()
        ls.solve(x, rel_tol=1e-9, max_iter=400, kernel_mode=1)
        want.append(x.cpu().numpy())
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for _ in range(3):
        xs = [T.internal.clone() for _, T, _ in systems]
        torch.cuda.synchronize()
        for (_, _, ls), x, s in zip(systems, xs, streams):
            abi.check(abi.lib().fvgb_solve_async(ls.handle, abi.ptr(x), cfg, None, s.cuda_stream))
        torch.cuda.synchronize()
        for x, w in zip(xs, want):
            np.testing.assert_array_equal(x.cpu().numpy(), w)


@pytest.mark.parametrize("n", [257, 520, 1025, 1600, 2049, 3100])
def test_cluster_blocks_without_rows(cuda, n):
    """128-row units that do not fill a power-of-two cluster (3, 5, 9, 13 units, 17 and 25 two
    to a block): thousands of iterations beside other work on the device keep the graph's
    bits and end at once (a block that waits for a word already written over holds the
    solve for the seconds that bound a wait)."""
    hm, T, ls = system((n, 1, 1))
    kw = dict(rel_tol=1e-300, max_iter=4000, allow=(abi.ERR_NOT_CONVERGED, abi.ERR_BREAKDOWN))
    x0 = T.internal.clone()
    want = ls.solve(x0, kernel_mode=1, **kw)
    other = torch.cuda.Stream()
    load = torch.randn(1 << 22, device="cuda")
    for busy in (False, True, True):
        x = T.internal.clone()
        ls.solve(x.clone(), kernel_mode=2, **kw)
        torch.cuda.synchronize()
        if busy:
            with torch.cuda.stream(other):
                for _ in range(200):
                    load.mul_(1.0001)
        start = time.perf_counter()
        st = ls.solve(x, kernel_mode=2, **kw)
        assert time.perf_counter() - start < 1.0
        assert (st.num_iter, st.final_res_norm, st.status) == (want.num_iter, want.final_res_norm, want.status)
        assert torch.equal(x, x0)
        torch.cuda.synchronize()


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED_IR])
def test_first_resident_solve_waits_for_nothing(cuda, precision):
    """fvgb_solve_async returns while the stream is still busy with what was queued before,
    also for the first solve that takes the resident kernel, on a mesh of the host's and
    on one built on the device."""
    hm, T, ls = system((47, 41, 17))
    specs = (abi.BoxSpec * 2)(abi.BoxSpec(33, 31, 20, 1.0, 1.0, 1.0, 0.0, 0, 0), abi.BoxSpec(7, 5, 3, 1.0, 1.0, 1.0, 0.0, 0, 0))
    ranges, handle, lsd = np.zeros(4, np.int32), C.c_void_p(), C.c_void_p()
    L = abi.lib()
    abi.check(L.fvgb_mesh_create_boxes(specs, 2, C.byref(handle), abi.ptr(ranges), None))
    abi.check(L.fvgb_ls_create(handle, 1, C.byref(lsd)))
    sizes = (C.c_int64 * 5)()
    abi.check(L.fvgb_mesh_sizes(handle, sizes))
    n, nif, nbf = list(sizes)[:3]
    old = torch.rand(n, dtype=torch.float64, device="cuda")
    gamma, ref = torch.ones(nif + nbf, dtype=torch.float64, device="cuda"), torch.zeros(nbf, dtype=torch.float64, device="cuda")
    types = np.full(6, abi.BC_FIXED_GRADIENT, np.int32)
    bc = abi.BC(abi.ptr(types), abi.ptr(ref))
    terms = (abi.Term * 2)(abi.Term(abi.TERM_DDT, 0, 1.0, abi.ptr(old), None), abi.Term(abi.TERM_LAPLACIAN, 0, -1.0, None, abi.ptr(gamma)))
    abi.check(L.fvgb_assemble(lsd, terms, 2, 1e-4, C.byref(bc), abi.ptr(ref), None))
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    for handle_ls, x0 in ((ls.handle, T.internal), (lsd, old)):
        cfg = [abi.SolverCfg(1e-9, 0.0, 50, precision, 0.1, 1000, 50, mode, abi.SOLVE_NO_TUNE) for mode in (1, 2)]
        x1, x2 = x0.clone(), x0.clone()
        torch.cuda.synchronize()
        abi.check(L.fvgb_solve_async(handle_ls, abi.ptr(x1), C.byref(cfg[0]), None, stream.cuda_stream))  # workspaces
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            torch.cuda._sleep(1 << 30)   # half a second
        start = time.perf_counter()
        abi.check(L.fvgb_solve_async(handle_ls, abi.ptr(x2), C.byref(cfg[1]), None, stream.cuda_stream))
        waited = time.perf_counter() - start
        assert not stream.query() and waited < 0.2
        torch.cuda.synchronize()
        assert torch.equal(x1, x2)
    L.fvgb_ls_destroy(lsd)
    L.fvgb_mesh_destroy(handle)
