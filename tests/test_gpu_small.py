"""The one-kernel Newton loop of small grids (k_nr_small) against the FP64 oracle, where its shapes
change: lanes per CTA and clusters, ragged scenario counts, the dense tail, refinement and reuse
thresholds, singular and unconverged scenarios, stepped solves, and outage batches with their own
admittances."""
import numpy as np
import pytest

from oracle import restate

pytestmark = pytest.mark.gpu
BASE = 1e8


def _grid(n, seed):
    from gap_b200 import synth

    net = synth.transmission_grid(seed, n=n)
    return net, synth.dc_start(net, BASE)


def _plan(net):
    import torch

    from gap_b200.engine import NRPlan, YbusPlan, branch_params, shunt_params

    yp = YbusPlan.from_network(net)
    y = yp.assemble(torch.as_tensor(branch_params(net), device="cuda"),
                    torch.as_tensor(shunt_params(net), device="cuda"), mode=1,
                    scale=float(net.u_rated[0]) ** 2 / BASE)[0]
    return NRPlan(yp.row_ptr, yp.col_idx, net.bus_type, jacobian="exact"), y


FP32 = dict(refine=2, refine_below=1e-2, reuse_below=1e-2)


@pytest.mark.parametrize("n", [2, 3, 40, 300, 900])
@pytest.mark.parametrize("scen,lanes,precision", [(1, 0, "fp64"), (11, 8, "fp64"), (19, 4, "fp32"),
                                                  (600, 8, "fp64"), (9, 1, "fp32")])
def test_small_grid_matches_oracle(n, scen, lanes, precision):
    """2 buses to a tail of 21 nodes (900 buses); voltages within 1e-8 of the oracle's."""
    import torch

    from gap_b200 import synth
    from gap_b200.engine import NRBatch

    if n == 900 and scen > 100:
        pytest.skip("more waves than the kernel is chosen for")
    net, v0 = _grid(n, 1)
    plan, y = _plan(net)
    s = synth.load_scenarios(net, scen, seed=3, base_power=BASE)
    b = NRBatch(plan, scen, precision=precision, lanes=lanes)
    kw = FP32 if precision == "fp32" else {}
    r = b.solve(y, torch.as_tensor(s, device="cuda"), v_init=torch.as_tensor(v0, device="cuda"),
                tol=1e-9, max_iter=20, policy="newton", **kw)
    assert (r.status.cpu().numpy() == 0).all()
    v = r.v.cpu().numpy()
    for k in {0, scen // 2, scen - 1}:
        o = restate.nr_solve(net, Y=restate.ybus_pi(net), tol=1e-12, max_iter=30, base_power=BASE,
                             policy="newton", jac="exact", s_spec=s[k], v0=v0)
        assert o["converged"] and np.max(np.abs(v[k] - o["v"])) < 1e-8


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_stepped_solve_is_the_solve(precision):
    """gapk_nr_step advances the same kernel one iteration at a time, with the factors reused
    below the threshold: bit for bit the one-launch solve."""
    import torch

    from gap_b200 import synth
    from gap_b200.engine import NRBatch

    net, v0 = _grid(300, 2)
    plan, y = _plan(net)
    s = torch.as_tensor(synth.load_scenarios(net, 13, seed=5, base_power=BASE), device="cuda")
    kw = dict(tol=1e-9, max_iter=20, policy="newton", v_init=torch.as_tensor(v0, device="cuda"))
    if precision == "fp32":
        kw.update(FP32)
    one = NRBatch(plan, 13, precision=precision, lanes=8).solve(y, s, **kw)
    r, states = NRBatch(plan, 13, precision=precision, lanes=8).solve_captured(y, s, **kw)
    assert torch.equal(one.v, r.v) and torch.equal(one.iterations, r.iterations)
    assert torch.equal(one.status, r.status) and len(states) == int(r.iterations.max())


def test_status_words_of_small_grids():
    """A scenario that does not converge, one whose mismatch is not finite and one that does, in
    one group; the unconverged one is at max_iter, and a batch that starts over converges."""
    import torch

    from gap_b200 import synth
    from gap_b200.engine import NRBatch

    net, v0 = _grid(120, 4)
    plan, y = _plan(net)
    s = synth.load_scenarios(net, 3, seed=1, base_power=BASE)
    s[1] *= 400.0
    s[2, 7] = np.nan
    b = NRBatch(plan, 3, precision="fp64", lanes=4)
    vd = torch.as_tensor(v0, device="cuda")
    r = b.solve(y, torch.as_tensor(s, device="cuda"), v_init=vd, tol=1e-9, max_iter=6, policy="clamped")
    st, it = r.status.cpu().numpy(), r.iterations.cpu().numpy()
    assert st[0] == 0 and st[1] == 1 and it[1] == 6 and st[2] == 3 and it[2] == 1
    assert np.array_equal(r.v[2].cpu().numpy(), v0)
    again = b.solve(y, torch.as_tensor(s[[0, 0, 0]], device="cuda"), v_init=vd, tol=1e-9, max_iter=20,
                    policy="clamped")
    assert (again.status.cpu().numpy() == 0).all() and torch.equal(again.v[0], r.v[0])


def test_outages_of_a_small_grid():
    """Per-scenario admittances (17 outages), FP32 factor, group thresholds across a cluster."""
    import torch

    from gap_b200 import studies, synth

    net, v0 = _grid(400, 6)
    outs = synth.n_minus_1(net, 17)
    st = studies.contingency_study("n-1", net, outs, net.specified_power(BASE), v0, base_power=BASE)
    r = st.make_batch().solve(st.y, st.s_spec, v_init=st.v0, tol=1e-9, max_iter=20, policy="newton", **FP32)
    torch.cuda.synchronize()
    assert (r.status.cpu().numpy() == 0).all()
    for k in (0, 8, 16):
        o = restate.nr_solve(net, Y=restate.ybus_pi(studies.outage_network(net, int(outs[k]))), tol=1e-12,
                             max_iter=30, base_power=BASE, policy="newton", jac="exact",
                             s_spec=net.specified_power(BASE), v0=v0)
        assert o["converged"] and np.max(np.abs(r.v[k].cpu().numpy() - o["v"])) < 1e-8
