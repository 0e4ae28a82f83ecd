"""The V-cycle of every shape of hierarchy against the numpy restatement: one level
above the coarsest, several in the one-cluster tail, levels beyond it (residual and
restriction in one kernel over whole aggregates), ragged last slices and blocks, and
coarsest systems of odd sizes (the inverse dealt over the cluster's blocks).  Then the
CG with the FP64 and the FP32 V-cycle: the residual asked for, and the same bits twice.
The V-cycle's tolerance is that of tests/test_amg.py (rounding of an FP64 V-cycle with a
dense inverse of a system of condition 1e3 to 1e4, with two orders to spare)."""
import numpy as np
import pytest
import torch

from foamadapter_gb300 import abi
from oracle import amg as oamg
from test_amg import gpu_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(17, 16, 1), (23, 19, 1), (40, 40, 1), (13, 12, 11), (150, 130, 1), (33, 29, 27),
                                  (257, 255, 1), (64, 60, 33)])
def test_vcycle_and_cg(cuda, dims):
    s = gpu_system(cuda, dims, dt=1.0)
    levels = oamg.hierarchy(s["ro"], s["col"], s["v"])
    r = np.random.default_rng(4).standard_normal(s["hm"].n)
    rd = torch.tensor(r, dtype=torch.float64, device="cuda")
    zd = torch.zeros_like(rd)
    abi.check(abi.lib().fvgb_amg_apply(s["ls"].handle, abi.ptr(rd), abi.ptr(zd), None))
    want = oamg.vcycle(levels, r)
    assert np.linalg.norm(zd.cpu().numpy() - want) <= 1e-10 * np.linalg.norm(want)
    counts = []
    for prec in (abi.PREC_FP64, abi.PREC_MIXED_IR):
        out = []
        for _ in range(2):
            x = s["x0"].clone()
            st = s["ls"].solve(x, rel_tol=1e-10, max_iter=500, precision=prec, preconditioner=abi.PRECOND_MULTIGRID)
            assert st.status == abi.OK and st.final_res_norm <= 1e-10 * st.init_res_norm
            out.append((x, st.num_iter))
        assert out[0][1] == out[1][1] and torch.equal(out[0][0], out[1][0])
        counts.append(out[0][1])
    assert abs(counts[0] - counts[1]) <= 3
