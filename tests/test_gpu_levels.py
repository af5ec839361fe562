"""The level-scheduled kernels over clusters of CTAs: results against the FP64 oracle for batches
of one to many groups, and bit for bit the same whatever the cluster's size, in a mix of studies
and in the adjoint."""
import numpy as np
import pytest

from oracle import restate

pytestmark = pytest.mark.gpu
BASE = 1e8


def _setup(n, seed):
    import torch

    from gap_b200 import synth
    from gap_b200.engine import NRPlan, YbusPlan, branch_params, shunt_params

    net = synth.transmission_grid(seed, n=n)
    yp = YbusPlan.from_network(net)
    y = yp.assemble(torch.as_tensor(branch_params(net), device="cuda"),
                    torch.as_tensor(shunt_params(net), device="cuda"), mode=1,
                    scale=float(net.u_rated[0]) ** 2 / BASE)[0]
    return net, NRPlan(yp.row_ptr, yp.col_idx, net.bus_type, jacobian="exact"), y, synth.dc_start(net, BASE)


@pytest.mark.parametrize("scen,lanes,threads", [(1, 1, 0), (1, 1, 64), (5, 4, 96), (9, 8, 0), (150, 8, 0),
                                                (296, 2, 256)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_groups_and_cluster_sizes(scen, lanes, threads, precision):
    """Clusters of 8, 8, 8, 8, 4 and 1 CTAs; CTAs of 64 and 96 threads leave levels in several
    rounds.  2,500 buses (a tail of 47 nodes), voltages within 1e-8 of the oracle's."""
    import torch

    from gap_b200 import synth
    from gap_b200.engine import NRBatch

    net, plan, y, v0 = _setup(2500, 2)
    s = synth.load_scenarios(net, scen, seed=4, base_power=BASE)
    kw = dict(refine=2, refine_below=1e-2, reuse_below=1e-2) if precision == "fp32" else {}
    r = NRBatch(plan, scen, precision=precision, lanes=lanes, threads=threads).solve(
        y, torch.as_tensor(s, device="cuda"), v_init=torch.as_tensor(v0, device="cuda"), tol=1e-9,
        max_iter=20, policy="newton", **kw)
    assert (r.status.cpu().numpy() == 0).all()
    for k in {0, scen - 1}:
        o = restate.nr_solve(net, Y=restate.ybus_pi(net), tol=1e-12, max_iter=30, base_power=BASE,
                             policy="newton", jac="exact", s_spec=s[k], v0=v0)
        assert o["converged"] and np.max(np.abs(r.v[k].cpu().numpy() - o["v"])) < 1e-8


def test_mix_keeps_the_batches_bits():
    """Twelve studies in one launch take smaller clusters than each alone; same bits."""
    import torch

    from gap_b200 import studies, synth

    kw = dict(refine=2, refine_below=1e-2, reuse_below=1e-2)
    sts = []
    for i in range(12):
        net = synth.transmission_grid(60 + i, n=2000 + 37 * i)
        sts.append(studies.load_study(f"g{i}", net, synth.load_scenarios(net, 3 + i, seed=i, base_power=BASE),
                                      synth.dc_start(net, BASE), base_power=BASE))
    res = [r.v.clone() for r in studies.solve_mixed(sts, retry=None, **kw)]
    torch.cuda.synchronize()
    for st, v in zip(sts, res):
        alone = st.batch.solve(st.y, st.s_spec, v_init=st.v0, policy="newton", **kw)
        assert (alone.status == 0).all() and torch.equal(alone.v, v)


@pytest.mark.parametrize("scen", [1, 20])
def test_adjoint_solves(scen):
    """dL/dP and dL/dQ through the transposed sweeps (one kernel with the plain ones) against the
    oracle's implicit-function gradient, to 1e-6 of the largest entry."""
    import torch

    from gap_b200 import synth
    from gap_b200.autograd import DifferentiablePowerFlow

    net = synth.transmission_grid(5, n=1500)
    s = synth.load_scenarios(net, scen, seed=2, base_power=BASE)
    model = DifferentiablePowerFlow(net, scen, base_power=BASE)
    p = torch.tensor(s.real, device="cuda", requires_grad=True)
    q = torch.tensor(s.imag, device="cuda", requires_grad=True)
    w = torch.linspace(0.5, 1.5, net.n_bus, device="cuda", dtype=torch.float64)
    vm, va = model(p, q)
    ((vm * w).sum() + (va * w.flip(0)).sum()).backward()
    k = scen - 1
    o = restate.nr_solve(net, Y=restate.ybus_pi(net), tol=1e-12, max_iter=30, base_power=BASE,
                         policy="newton", jac="exact", s_spec=s[k], v0=synth.dc_start(net, BASE))
    rp, ci, va_ = restate.ybus_pi(net)
    zb = float(net.u_rated[0]) ** 2 / BASE
    import scipy.sparse as sp
    import scipy.sparse.linalg as spla

    J = restate.jacobian(rp, ci, va_ * zb, o["v"], net.bus_type, mode="exact", drop=False)
    J = sp.csc_matrix(J[0] if isinstance(J, tuple) else J)
    ang, mag, peq, qeq, _ = restate.var_maps(net.bus_type)
    wn = w.cpu().numpy()
    g = np.zeros(J.shape[0])
    g[ang[ang >= 0]], g[mag[mag >= 0]] = wn[::-1][ang >= 0], wn[mag >= 0]
    lam = spla.spsolve(J.T.tocsc(), g)
    want_p = np.where(peq >= 0, lam[peq], 0.0)
    want_q = np.where(qeq >= 0, lam[qeq], 0.0)
    for got, want in ((p.grad[k], want_p), (q.grad[k], want_q)):
        assert np.max(np.abs(got.cpu().numpy() - want)) <= 1e-6 * np.max(np.abs(want))


@pytest.mark.parametrize("n,scen", [(700, 1), (300, 9)])
def test_more_levels_than_the_bounds_buffer(n, scen):
    """A line of buses eliminated in natural order: n - 1 levels of one node each, past and below
    the 256 level bounds kept in shared memory plus one; FP64 flat start against the oracle."""
    import torch

    from gap_b200 import _native as N
    from gap_b200.engine import NRBatch, NRPlan, YbusPlan, branch_params, shunt_params
    from gap_b200.network import PQ, SLACK, Network

    bt = np.full(n, PQ, np.int32)
    bt[-1] = SLACK
    p = np.full(n, -1e3)
    p[-1] = 0.0
    net = Network.build(bus_id=np.arange(n), u_rated=np.full(n, 10e3), bus_type=bt, p=p, q=0.3 * p,
                        from_id=np.arange(n - 1), to_id=np.arange(1, n), r1=np.full(n - 1, 0.02),
                        x1=np.full(n - 1, 0.02))
    yp = YbusPlan.from_network(net)
    y = yp.assemble(torch.as_tensor(branch_params(net), device="cuda"),
                    torch.as_tensor(shunt_params(net), device="cuda"), mode=N.YBUS_REFERENCE,
                    scale=10e3 ** 2 / 1e6)[0]
    plan = NRPlan(yp.row_ptr, yp.col_idx, net.bus_type, jacobian="exact", ordering="natural", dense_min=-1)
    assert plan.info["n_levels"] == n - 1
    s = np.repeat(net.specified_power(1e6)[None], scen, axis=0)
    b = NRBatch(plan, scen, precision="fp64", use_graph=False)
    sd = torch.as_tensor(s, device="cuda")
    v0 = torch.ones(n, dtype=torch.complex128, device="cuda")
    b.stage_load(y, sd, v_init=v0)
    for stage in ("mismatch", "jacobian", "factor", "solve"):
        b.stage(stage)
    dx = b.correction().cpu().numpy()
    import scipy.sparse.linalg as spla

    rp, ci, va = restate.ybus_reference(net)
    ypu = va * (10e3 ** 2 / 1e6)
    one = np.ones(n, complex)
    J = restate.jacobian(rp, ci, ypu, one, net.bus_type, mode="exact", drop=False).tocsc()
    want = spla.spsolve(J, -restate.mismatch(net.bus_type, restate.power_injections(rp, ci, ypu, one), s[0]))
    assert np.max(np.abs(dx[-1] - want)) <= 1e-8 * np.max(np.abs(want))  # condition ~ n^2 ~ 5e5
