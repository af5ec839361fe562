"""The CTA size that a batch of many lane groups takes by itself."""
import pytest

pytestmark = pytest.mark.gpu
BASE = 1e8


@pytest.mark.parametrize("n,scen,precision,few", [(500, 4096, "fp64", 256), (1000, 4096, "fp32", 256),
                                                  (500, 5920, "fp32", 192)])
def test_many_groups_keep_small_ctas(n, scen, precision, few):
    """512 and 740 groups: the default is as fast as the threads that hold all groups on the GPU at
    once (larger CTAs, which leave the groups to several waves, take 1.28 to 1.36 times as long)."""
    import torch

    from gap_b200 import synth
    from gap_b200.engine import NRBatch, NRPlan, YbusPlan, branch_params, shunt_params

    net = synth.transmission_grid(1, n=n)
    yp = YbusPlan.from_network(net)
    y = yp.assemble(torch.as_tensor(branch_params(net), device="cuda"),
                    torch.as_tensor(shunt_params(net), device="cuda"), mode=1,
                    scale=float(net.u_rated[0]) ** 2 / BASE)[0]
    plan = NRPlan(yp.row_ptr, yp.col_idx, net.bus_type, jacobian="exact")
    s = torch.as_tensor(synth.load_scenarios(net, scen, seed=3, base_power=BASE), device="cuda")
    kw = dict(v_init=torch.as_tensor(synth.dc_start(net, BASE), device="cuda"), tol=1e-8, max_iter=20,
              policy="newton")
    if precision == "fp32":
        kw.update(refine=2, refine_below=1e-2, reuse_below=1e-2)
    batches = [NRBatch(plan, scen, precision=precision, threads=t) for t in (0, few)]
    best = [float("inf")] * 2
    for _ in range(6):
        for i, b in enumerate(batches):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            r = b.solve(y, s, **kw)
            e1.record()
            torch.cuda.synchronize()
            assert (r.status == 0).all()
            best[i] = min(best[i], e0.elapsed_time(e1))
    assert best[0] < 1.15 * best[1]
