"""gapk_nr_adjoint straight after an FP32 solve with refinement and reuse thresholds: the Jacobian is
refactorised at the solution and the transposed solve refined once, whatever the thresholds decided
in the solve's last iteration."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
BASE = 1e8


@pytest.mark.parametrize("n", [300, 3000])
@pytest.mark.parametrize("tol,status", [(1e-9, 0), (1e-17, 1)])
def test_adjoint_after_a_solve_with_thresholds(n, tol, status):
    """300 buses (the one-kernel loop) and 3,000; a converged solve, and one that ends at
    max_iter while it reuses its factors.  dL/dP and dL/dQ of a linear loss against an FP64 batch at
    the same voltages, to 1e-6 of the largest entry: one refinement squares the FP32 solve's relative
    error, which is 4e-5 to 4e-4 on such grids."""
    import torch

    from gap_b200 import _native as N
    from gap_b200 import synth
    from gap_b200.engine import NRBatch, NRPlan, YbusPlan, _dptr, _stream_ptr, branch_params, shunt_params

    scen = 11
    net = synth.transmission_grid(1, n=n)
    yp = YbusPlan.from_network(net)
    y = yp.assemble(torch.as_tensor(branch_params(net), device="cuda"),
                    torch.as_tensor(shunt_params(net), device="cuda"), mode=1,
                    scale=float(net.u_rated[0]) ** 2 / BASE)[0]
    plan = NRPlan(yp.row_ptr, yp.col_idx, net.bus_type, jacobian="exact")
    s = torch.as_tensor(synth.load_scenarios(net, scen, seed=3, base_power=BASE), device="cuda")
    w = torch.linspace(0.5, 1.5, n, device="cuda", dtype=torch.float64).repeat(scen, 1)

    def adjoint(b):
        dp, dq = torch.empty_like(w), torch.empty_like(w)
        N.check(N.lib().gapk_nr_adjoint(b._h, _dptr(w), _dptr(w), _dptr(dp), _dptr(dq), _stream_ptr()))
        return dp.cpu().numpy(), dq.cpu().numpy()

    b = NRBatch(plan, scen, precision="fp32", lanes=8)
    r = b.solve(y, s, v_init=torch.as_tensor(synth.dc_start(net, BASE), device="cuda"), tol=tol,
                max_iter=10, policy="newton", refine=2, refine_below=1e-2, reuse_below=1e-2)
    assert (r.status == status).all() and (r.final_mismatch < 1e-8).all()
    got = adjoint(b)
    exact = NRBatch(plan, scen, precision="fp64", lanes=8)
    exact.stage_load(y, s, v_init=r.v)
    for a, e in zip(got, adjoint(exact)):
        assert np.max(np.abs(a - e)) <= 1e-6 * np.max(np.abs(e))
