"""What a solve leaves in the batch for the stage calls and the loop counter: the same after the
one-kernel loop of small grids as after the separate kernels."""
import pytest

pytestmark = pytest.mark.gpu
BASE = 1e8
FP32 = dict(refine=2, refine_below=1e-2, reuse_below=1e-2)


def _setup(n, scen):
    import torch

    from gap_b200 import synth
    from gap_b200.engine import NRPlan, YbusPlan, branch_params, shunt_params

    net = synth.transmission_grid(1, n=n)
    yp = YbusPlan.from_network(net)
    y = yp.assemble(torch.as_tensor(branch_params(net), device="cuda"),
                    torch.as_tensor(shunt_params(net), device="cuda"), mode=1,
                    scale=float(net.u_rated[0]) ** 2 / BASE)[0]
    s = torch.as_tensor(synth.load_scenarios(net, scen, seed=3, base_power=BASE), device="cuda")
    return (NRPlan(yp.row_ptr, yp.col_idx, net.bus_type, jacobian="exact"), y, s,
            torch.as_tensor(synth.dc_start(net, BASE), device="cuda"))


@pytest.mark.parametrize("n", [300, 3000])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("stepped", [False, True])
def test_stages_after_a_solve(n, precision, stepped):
    """300 buses (the one-kernel loop) and 3,000.  After a solve that converged no group solves: the
    Jacobian, factor and solve stages change nothing.  After one that ended at max_iter no group
    iterates: the mismatch stage changes nothing."""
    import torch

    from gap_b200.engine import NRBatch

    plan, y, s, v0 = _setup(n, 11)
    kw = dict(v_init=v0, tol=1e-9, policy="newton", **(FP32 if precision == "fp32" else {}))

    def solve(max_iter):
        b = NRBatch(plan, 11, precision=precision, lanes=8)
        if stepped:
            return b, b.solve_captured(y, s, max_iter=max_iter, **kw)[0]
        return b, b.solve(y, s, max_iter=max_iter, **kw)

    b, r = solve(20)
    assert (r.status == 0).all() and b.loop_count() == int(r.iterations.max())
    dx = b.correction()
    for stage in ("jacobian", "factor", "solve"):
        b.stage(stage)
    assert torch.equal(b.correction(), dx)
    b, r = solve(2)
    assert (r.status == 1).all() and b.loop_count() == 2
    f = b.mismatch()
    b.stage("mismatch")
    assert torch.equal(b.mismatch(), f)


def test_loop_count_after_a_retry():
    """A start of 0.45 pu, which the clamped policy's floor keeps from converging and the retry with
    full steps solves: the loop counter is the retry's, for grids of 120 and 3,000 buses in one
    launch."""
    import torch

    from gap_b200 import studies, synth

    sts = []
    for n in (120, 3000):
        net = synth.transmission_grid(1, n=n)
        sts.append(studies.load_study(f"g{n}", net, synth.load_scenarios(net, 9, seed=3, base_power=BASE),
                                      0.45 * synth.dc_start(net, BASE), base_power=BASE, precision="fp64"))
    res = studies.solve_mixed(sts, policy="clamped", retry="newton", max_iter=12, refine=0)
    torch.cuda.synchronize()
    for st, r in zip(sts, res):
        assert (r.status == 0).all() and int(r.iterations.max()) < 12
        assert st.batch.loop_count() == int(r.iterations.max())
