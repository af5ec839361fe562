"""Y-bus assembly and branch results where their kernels' tiles end: rows longer than a tile,
scenario counts and branch counts that leave a remainder, branch rows off a 16-byte boundary."""
import numpy as np
import pytest

from gap_b200.network import PQ, SLACK, Network
from oracle import restate

pytestmark = pytest.mark.gpu


def _star(spokes, tail, seed=0):
    """A hub with `spokes` neighbours (two parallel branches to each third one) and a line of
    `tail` buses behind the last spoke; a third of the branches tapped."""
    rng = np.random.default_rng(seed)
    frm = [0] * spokes + [0 for k in range(0, spokes, 3)] + list(range(spokes, spokes + tail))
    to = list(range(1, spokes + 1)) + [k + 1 for k in range(0, spokes, 3)] + \
        list(range(spokes + 1, spokes + tail + 1))
    m, n = len(frm), spokes + tail + 1
    tap = rng.random(m) < 0.33
    bt = np.full(n, PQ, np.int32)
    bt[0] = SLACK
    return Network.build(bus_id=np.arange(n), u_rated=np.full(n, 10e3), bus_type=bt,
                         from_id=frm, to_id=to, r1=rng.uniform(0.05, 0.5, m),
                         x1=rng.uniform(0.05, 0.4, m), b1=rng.uniform(0, 1e-5, m),
                         g1=rng.uniform(0, 1e-6, m), k=np.where(tap, rng.uniform(0.95, 1.05, m), 1.0),
                         theta=np.where(tap, rng.uniform(-0.2, 0.2, m), 0.0))


def _scenarios(net, scen, aligned, seed=1):
    """Branch rows [scen, m, 6] with r, x, b spread by 10 %, on the device; with aligned=False
    the first row starts 8 bytes past a 16-byte boundary."""
    import torch

    from gap_b200.engine import branch_params

    rng = np.random.default_rng(seed)
    br = np.repeat(branch_params(net)[None], scen, axis=0)
    br[:, :, [0, 1, 3]] *= rng.uniform(0.9, 1.1, size=br.shape[:2] + (3,))
    off = 0 if aligned else 1
    buf = torch.empty(br.size + off, dtype=torch.float64, device="cuda")
    dev = buf[off:].view(br.shape)
    dev.copy_(torch.as_tensor(br))
    assert dev.is_contiguous() and (dev.data_ptr() % 16 == 0) == aligned
    return br, dev


def _with(net, row):
    import dataclasses

    return dataclasses.replace(net, r1=row[:, 0].copy(), x1=row[:, 1].copy(), b1=row[:, 3].copy())


@pytest.mark.parametrize("spokes,tail", [(3, 1), (191, 4), (192, 255), (300, 70)])
@pytest.mark.parametrize("scen,aligned", [(1, True), (5, False), (8, True)])
def test_ybus_tile_edges(spokes, tail, scen, aligned):
    """The hub's row holds 2/3 spokes parallel pairs: 256, 257 and 401 slots around the tile of
    256.  Without taps bit for bit the oracle's; with taps within 4 roundings per term."""
    import torch

    from gap_b200.engine import YbusPlan, shunt_params

    net = _star(spokes, tail)
    plan = YbusPlan.from_network(net)
    br, dev = _scenarios(net, scen, aligned)
    sh = torch.as_tensor(shunt_params(net), device="cuda")
    ref = plan.assemble(dev, sh, mode=0).cpu().numpy()
    pi = plan.assemble(dev, sh, mode=1).cpu().numpy()
    rows = np.repeat(np.arange(net.n_bus), np.diff(plan.row_ptr))
    for s in range(scen):
        one = _with(net, br[s])
        assert np.array_equal(ref[s], restate.ybus_reference(one)[2])
        want = restate.ybus_pi(one)[2]
        size = np.zeros(net.n_bus)  # sum of |entries| of each row bounds its rounding errors
        np.add.at(size, rows, np.abs(want))
        assert np.all(np.abs(pi[s] - want) <= 8 * 2.0 ** -52 * 4 * size[rows])


@pytest.mark.parametrize("scen", [1, 8, 9])
@pytest.mark.parametrize("shared", [True, False])
def test_branch_flow_tile_edges(scen, shared):
    """301 branches (two tiles of 128 and 45), one of them out of service, and scenario counts at
    and past the 8 of a CTA; branch data shared by the scenarios or their own."""
    import torch

    from gap_b200.engine import branch_flows

    net = _star(200, 34)
    assert net.n_branch == 301
    net.status[130] = 0
    br, dev = _scenarios(net, scen, True)
    rng = np.random.default_rng(5)
    v = rng.uniform(0.9, 1.1, (scen, net.n_bus)) * np.exp(1j * rng.uniform(-0.2, 0.2, (scen, net.n_bus)))
    i_n = np.full(net.n_branch, 100.0)
    out = branch_flows(net, torch.as_tensor(v, device="cuda"), 1e6, i_n=i_n,
                       branch=None if shared else dev).cpu().numpy()
    for s in range(scen):
        one = net if shared else _with(net, br[s])
        want, idx = restate.branch_flows(one, v[s], 1e6, i_n=i_n)
        assert len(idx) == 300 and np.all(out[s, 130] == 0.0)
        assert np.max(np.abs(out[s, idx] - want) / np.abs(want).max(axis=0)) <= 1e-12
