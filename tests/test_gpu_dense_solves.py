"""The dense tail's substitutions with a cluster of CTAs per scenario, and the transposed ones of
the adjoint: tail orders around the blocks of 32, cluster sizes 8 to 1."""
import numpy as np
import pytest

from oracle import restate

pytestmark = pytest.mark.gpu
BASE = 1e8


@pytest.mark.parametrize("n,seed", [(900, 1), (1467, 100), (2500, 2), (6000, 3), (10000, 0)])
@pytest.mark.parametrize("scen,precision", [(1, "fp64"), (13, "fp64"), (40, "fp64")])
def test_newton_correction_of_few_scenarios(n, seed, scen, precision):
    """Tails of 21 to 253 nodes (orders 42 to 506: full and partial last blocks) with clusters of
    8, 8 and 2 CTAs: the first Newton correction against scipy's, to 1e-10 of the largest entry."""
    import scipy.sparse.linalg as spla
    import torch

    from gap_b200 import synth
    from gap_b200.engine import NRBatch, NRPlan, YbusPlan, branch_params, shunt_params

    net = synth.transmission_grid(seed, n=n)
    yp = YbusPlan.from_network(net)
    y = yp.assemble(torch.as_tensor(branch_params(net), device="cuda"),
                    torch.as_tensor(shunt_params(net), device="cuda"), mode=1,
                    scale=float(net.u_rated[0]) ** 2 / BASE)[0]
    plan = NRPlan(yp.row_ptr, yp.col_idx, net.bus_type, jacobian="exact")
    assert plan.info["n_tail"] >= 16
    s = synth.load_scenarios(net, scen, seed=3, base_power=BASE)
    v0 = synth.dc_start(net, BASE)
    b = NRBatch(plan, scen, precision=precision)
    b.stage_load(y, torch.as_tensor(s, device="cuda"), v_init=torch.as_tensor(v0, device="cuda"))
    for stage in ("mismatch", "jacobian", "factor", "solve"):
        b.stage(stage)
    dx = b.correction().cpu().numpy()
    rp, ci, va = restate.ybus_pi(net)
    ypu = va * float(net.u_rated[0]) ** 2 / BASE
    J = restate.jacobian(rp, ci, ypu, v0, net.bus_type, mode="exact", drop=False).tocsc()
    lu = spla.splu(J)
    calc = restate.power_injections(rp, ci, ypu, v0)
    for k in {0, scen - 1}:
        want = lu.solve(-restate.mismatch(net.bus_type, calc, s[k]))
        assert np.max(np.abs(dx[k] - want)) <= 1e-10 * np.max(np.abs(want))


@pytest.mark.parametrize("scen", [1, 30, 160])
def test_transposed_dense_solve(scen):
    """Gradients of a linear loss on a 4,000-bus grid (clusters of 8, 4 and 1) are the same for a
    scenario whatever the batch around it, to 1e-10 of the largest entry, and the first one's
    directional derivative matches central differences of the solve to 1e-6."""
    import torch

    from gap_b200 import synth
    from gap_b200.autograd import DifferentiablePowerFlow

    net = synth.transmission_grid(9, n=4000)
    s = synth.load_scenarios(net, scen, seed=2, base_power=BASE)
    w = torch.linspace(-1.0, 1.0, net.n_bus, device="cuda", dtype=torch.float64)

    def grads(spec):
        model = DifferentiablePowerFlow(net, spec.shape[0], base_power=BASE)
        p, q = (torch.tensor(a, device="cuda", requires_grad=True) for a in (spec.real, spec.imag))
        vm, va = model(p, q)
        ((vm + va) * w).sum().backward()
        return p.grad.cpu().numpy(), q.grad.cpu().numpy()

    gp, gq = grads(s)
    one = grads(s[-1:])
    for a, b in ((gp[-1], one[0][0]), (gq[-1], one[1][0])):
        assert np.max(np.abs(a - b)) <= 1e-10 * np.max(np.abs(b))
    rng = np.random.default_rng(0)
    d = rng.normal(size=net.n_bus)
    h = 1e-4

    def loss(step):
        spec = s[:1] + step * d[None]
        model = DifferentiablePowerFlow(net, 1, base_power=BASE, tol=1e-12)
        vm, va = model(*(torch.tensor(a, device="cuda") for a in (spec.real, spec.imag)))
        return float(((vm + va) * w).sum())

    fd = (8 * (loss(h) - loss(-h)) - (loss(2 * h) - loss(-2 * h))) / (12 * h)
    assert abs(fd - gp[0] @ d) <= 1e-6 * abs(gp[0] @ d)
