"""Dense tails with more blocks than the clustered solves fetch ahead, and with a vector that needs
more shared memory than a launch gets without opting in."""
import functools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@functools.lru_cache(maxsize=None)
def _complete(n):
    """A grid with a branch between every two of n buses (admittances for 1 pu in all per bus), one
    dense tail of order 2 n - 2: its plan, admittances, powers, voltages around 1 pu, exact Jacobian
    and mismatch."""
    from gap_b200.engine import NRPlan
    from oracle import restate

    rng = np.random.default_rng(0)
    y = (rng.uniform(0.1, 0.2, (n, n)) - 1j * rng.uniform(0.5, 1.5, (n, n))) / n
    y = np.triu(y, 1)
    y = y + y.T
    ybus = (np.diag(y.sum(axis=1)) - y).ravel()
    rp, ci = np.arange(n + 1) * n, np.tile(np.arange(n), n)
    bt = np.zeros(n, np.int32)
    bt[0] = 2
    v = 1.0 + 0.02 * rng.normal(size=n) + 0.02j * rng.normal(size=n)
    s = 0.1 * (rng.normal(size=n) + 1j * rng.normal(size=n))
    J = restate.jacobian(rp, ci, ybus, v, bt, mode="exact", drop=False).toarray()
    f = restate.mismatch(bt, restate.power_injections(rp, ci, ybus, v), s)
    plan = NRPlan(rp, ci, bt, jacobian="exact", ordering="natural")
    assert plan.info["n_tail"] == n - 1
    return plan, ybus, s, v, bt, J, f


def _loaded(n, fused):
    import torch

    from gap_b200.engine import NRBatch

    plan, y, s, v, _, _, _ = _complete(n)
    b = NRBatch(plan, 1, precision="fp64", dense_fused=fused)
    y, s, v = (torch.as_tensor(a, device="cuda") for a in (y, s[None], v[None]))
    b.stage_load(y, s, v_init=v)
    return b, (y, s, v)


@pytest.mark.parametrize("n,fused", [(2560, False), (2560, True), (1100, False)])
def test_correction_with_a_large_tail(n, fused):
    """Orders 5,118 (40 KB in FP64) and 2,198 (69 blocks, the last one of 22); one scenario by a
    cluster of 8 CTAs, and as one of several concurrent batches by one CTA: to 1e-10 of the largest
    entry."""
    plan, y, s, v, bt, J, f = _complete(n)
    want = np.linalg.solve(J, -f)
    b, keep = _loaded(n, fused)
    for stage in ("mismatch", "jacobian", "factor", "solve"):
        b.stage(stage)
    got = b.correction().cpu().numpy()[0]
    assert np.max(np.abs(got - want)) <= 1e-10 * np.max(np.abs(want))


@pytest.mark.parametrize("n,fused", [(2560, False), (2560, True), (1100, False)])
def test_transposed_solve_with_a_large_tail(n, fused):
    """The adjoint of a linear loss, clusters of 8 CTAs and one CTA: to 1e-10 of the largest entry."""
    import torch

    from gap_b200 import _native as N
    from gap_b200.engine import _dptr, _stream_ptr
    from oracle import restate

    plan, y, s, v, bt, J, f = _complete(n)
    b, keep = _loaded(n, fused)
    w = torch.linspace(0.5, 1.5, n, device="cuda", dtype=torch.float64)[None].contiguous()
    dp, dq = torch.empty_like(w), torch.empty_like(w)
    N.check(N.lib().gapk_nr_adjoint(b._h, _dptr(w), _dptr(w), _dptr(dp), _dptr(dq), _stream_ptr()))
    ang, mag, peq, qeq, _ = restate.var_maps(bt)
    g, wn = np.zeros(J.shape[0]), w.cpu().numpy()[0]
    g[ang[ang >= 0]], g[mag[mag >= 0]] = wn[ang >= 0], wn[mag >= 0]
    lam = np.linalg.solve(J.T, g)
    for got, eq in ((dp, peq), (dq, qeq)):
        want = np.where(eq >= 0, lam[eq], 0.0)
        assert np.max(np.abs(got.cpu().numpy()[0] - want)) <= 1e-10 * np.max(np.abs(lam))
