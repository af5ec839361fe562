"""A solve that starts from an earlier solution, as a time series makes it: its first mismatch is
already below reuse_below, so it must not take factors that it has not formed itself."""
import numpy as np
import pytest

from oracle import restate

pytestmark = pytest.mark.gpu
BASE = 1e8
KW = dict(tol=1e-9, max_iter=20, policy="newton", refine=2, refine_below=1e-2, reuse_below=1e-2)


@pytest.mark.parametrize("n", [300, 3000])
@pytest.mark.parametrize("scen,lanes", [(1, 1), (11, 8)])
def test_warm_start_below_the_reuse_threshold(n, scen, lanes):
    """300 buses (the one-kernel loop) and 3,000 (the separate kernels), FP32: loads changed by
    1e-4 and the voltages of the solve before, on a new batch, on the same batch right after that
    solve, and on it after a solve of another state (its factors are that state's).  All three
    bit for bit the same, within 1e-8 of the oracle."""
    import torch

    from gap_b200 import synth
    from gap_b200.engine import NRBatch, NRPlan, YbusPlan, branch_params, shunt_params

    net = synth.transmission_grid(1, n=n)
    v0 = synth.dc_start(net, BASE)
    yp = YbusPlan.from_network(net)
    y = yp.assemble(torch.as_tensor(branch_params(net), device="cuda"),
                    torch.as_tensor(shunt_params(net), device="cuda"), mode=1,
                    scale=float(net.u_rated[0]) ** 2 / BASE)[0]
    plan = NRPlan(yp.row_ptr, yp.col_idx, net.bus_type, jacobian="exact")
    s = torch.as_tensor(synth.load_scenarios(net, scen, seed=3, base_power=BASE), device="cuda")
    vd = torch.as_tensor(v0, device="cuda")
    batch = NRBatch(plan, scen, precision="fp32", lanes=lanes)
    first = batch.solve(y, s, v_init=vd, **KW)
    assert (first.status == 0).all()
    v1, s1 = first.v.clone(), s * (1.0 + 1e-4)
    # the start lies between the tolerance and the threshold
    rp, ci, va = restate.ybus_pi(net)
    ypu = va * float(net.u_rated[0]) ** 2 / BASE
    for k in range(scen):
        f = restate.mismatch(net.bus_type, restate.power_injections(rp, ci, ypu, v1[k].cpu().numpy()),
                             s1[k].cpu().numpy())
        assert 1e-9 < np.max(np.abs(f)) < 1e-2

    fresh = NRBatch(plan, scen, precision="fp32", lanes=lanes).solve(y, s1, v_init=v1, **KW)
    again = batch.solve(y, s1, v_init=v1, **KW)
    # one iteration of the same grid with all impedances 50 times smaller leaves its factors behind
    batch.solve(50.0 * y, s, v_init=vd, **dict(KW, max_iter=1))
    other = batch.solve(y, s1, v_init=v1, **KW)
    for r in (fresh, again, other):
        assert (r.status == 0).all() and torch.equal(r.v, fresh.v) and torch.equal(r.iterations, fresh.iterations)
    for k in {0, scen - 1}:
        o = restate.nr_solve(net, Y=restate.ybus_pi(net), tol=1e-12, max_iter=30, base_power=BASE,
                             policy="newton", jac="exact", s_spec=s1[k].cpu().numpy(), v0=v0)
        assert o["converged"] and np.max(np.abs(fresh.v[k].cpu().numpy() - o["v"])) < 1e-8
