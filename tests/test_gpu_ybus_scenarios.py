"""Y-bus assembly with one and with four scenarios per CTA: the same values on both sides of the
line between them."""
import numpy as np
import pytest

from oracle import restate
from test_gpu_ybus_tiles import _scenarios, _star, _with

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spokes,tail,scen", [(3, 1, 1024), (3, 1, 1027), (300, 70, 259), (192, 255, 403)])
@pytest.mark.parametrize("aligned", [True, False])
def test_many_scenarios_as_few_at_a_time(spokes, tail, scen, aligned):
    """1 tile x 1,024 scenarios is the last size with one scenario per CTA; the others have four,
    with 3 scenarios in the last one, and a row longer than a tile in the second and third grid.
    Without taps bit for bit the assembly of 100 scenarios at a time, with taps within 4 roundings
    per term."""
    import torch

    from gap_b200.engine import YbusPlan, shunt_params

    net = _star(spokes, tail)
    plan = YbusPlan.from_network(net)
    br, dev = _scenarios(net, scen, aligned)
    sh = torch.as_tensor(shunt_params(net), device="cuda")
    for mode in (0, 1):
        got = plan.assemble(dev, sh, mode=mode, scale=2.0).cpu().numpy()
        few = np.concatenate([plan.assemble(dev[a:a + 100], sh, mode=mode, scale=2.0).cpu().numpy()
                              for a in range(0, scen, 100)])
        if mode == 0:
            assert np.array_equal(got, few)
        rows = np.repeat(np.arange(net.n_bus), np.diff(plan.row_ptr))
        size = np.zeros((scen, net.n_bus))
        np.add.at(size, (slice(None), rows), np.abs(few))
        assert np.all(np.abs(got - few) <= 2 * 8 * 2.0 ** -52 * 4 * size[:, rows])
    assert np.array_equal(plan.assemble(dev, sh, mode=0).cpu().numpy()[-1],
                          restate.ybus_reference(_with(net, br[-1]))[2])
