"""The factors that the one-kernel loop of small grids leaves in the batch, as a later stage or step
finds them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
BASE = 1e8


@pytest.mark.parametrize("n", [40, 300, 900])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_a_solve_that_does_not_iterate_keeps_the_factors(n, precision):
    """A second solve starts at its solution and ends at the first test: the batch still holds the
    first solve's factors, and a triangular solve takes them (bit for bit the correction of a batch
    that made only the first solve).  2 and 9 scenarios of a group, tails of 0 to 21 nodes."""
    import torch

    from gap_b200 import synth
    from gap_b200.engine import NRBatch, NRPlan, YbusPlan, branch_params, shunt_params

    net = synth.transmission_grid(1, n=n)
    yp = YbusPlan.from_network(net)
    y = yp.assemble(torch.as_tensor(branch_params(net), device="cuda"),
                    torch.as_tensor(shunt_params(net), device="cuda"), mode=1,
                    scale=float(net.u_rated[0]) ** 2 / BASE)[0]
    plan = NRPlan(yp.row_ptr, yp.col_idx, net.bus_type, jacobian="exact")
    vd = torch.as_tensor(synth.dc_start(net, BASE), device="cuda")
    refine = dict(refine=1) if precision == "fp32" else {}
    for scen in (2, 9):
        s = torch.as_tensor(synth.load_scenarios(net, scen, seed=3, base_power=BASE), device="cuda")
        got = []
        for second in (False, True):
            b = NRBatch(plan, scen, precision=precision, lanes=8)
            r = b.solve(y, s, v_init=vd, tol=1e-9, max_iter=20, policy="newton", **refine)
            assert (r.status == 0).all()
            if second:
                # another batch's factors in between, in the shared memory of every SM
                k = 592
                NRBatch(plan, k, precision=precision, lanes=8).solve(
                    50.0 * y, s[:1].expand(k, -1).contiguous(), v_init=vd, tol=1e-9, max_iter=1,
                    policy="newton", **refine)
                r2 = b.solve(y, s, v_init=r.v.clone(), tol=1e-6, max_iter=20, policy="newton", **refine)
                assert (r2.iterations == 1).all() and torch.equal(r2.v, r.v)
            b.stage_load(y, s, v_init=vd)
            b.stage("mismatch")
            b.stage("solve")
            got.append(b.correction().cpu().numpy())
        assert np.isfinite(got[0]).all() and np.array_equal(got[0], got[1])
