"""The work that this framework is timed on: its public entry points over their real range.

Every case is a dict of plain values whose "kind" names the call that a user's program makes:

* "api"      NewtonRaphson.solve_power_flow on one network, the call a program written for the
             reference's solver interface makes; the whole call, host work included.
* "solve"    NRBatch.solve: load scenarios of one grid (one shared Y), or its N-1 outages (one Y
             value set per scenario), on device tensors.
* "mix"      studies.solve_mixed: load scenarios, outages and independent grids in one launch.
* "gradient" DifferentiablePowerFlow forward and backward (voltages, then dL/dP, dL/dQ, dL/dr, dL/dx).
* "pipeline" HostPipeline.solve from and to pinned host memory.
* "lu"       SparseLU.factorize and one solve of a complex admittance system.
* "ybus"     YbusPlan.assemble with branch data per scenario.
* "flows"    branch_flows: the branch results of solved scenarios.

Grids are the repository's synthetic ones (gap_b200.synth); a case names its grid, the seed
draws the loads.  A solve's final mismatch is left out of the outputs: once converged it is the
rounding noise of the residual.  Voltages come whole, with the iteration counts and statuses.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from gap_b200 import _native as N
from gap_b200 import studies, synth, workloads
from gap_b200.api import NewtonRaphson, PowerFlowConfig
from gap_b200.autograd import DifferentiablePowerFlow, branch_losses_mw
from gap_b200.engine import (HostPipeline, NRBatch, NRPlan, SparseLU, YbusPlan, branch_flows,
                             branch_params, shunt_params)

SIGMA = 0.1  # lognormal spread of the loads between scenarios
MIXED = dict(refine=2, refine_below=1e-2, reuse_below=1e-2)  # the benchmark's FP32 settings


def listed():
    return [
        # the smallest call: one 200-bus feeder through the reference-shaped interface
        {"name": "feeder api", "kind": "api", "grid": "feeder", "n": 200, "grid_seed": 0},
        # a distribution utility's load study: the same feeder, 1024 load scenarios, FP64
        {"name": "feeder batch", "kind": "solve", "grid": "feeder", "n": 200, "grid_seed": 0,
         "scen": 1024, "precision": "fp64", "policy": "reference", "lanes": 8, "threads": 512},
        # one transmission-grid power flow in plain FP64: latency
        {"name": "grid single", "kind": "solve", "grid": "transmission", "n": 10000,
         "grid_seed": 0, "scen": 1, "precision": "fp64", "policy": "newton", "lanes": 1,
         "threads": 512},
        # the benchmark's headline batch: FP32 factor refined in FP64
        {"name": "grid batch", "kind": "solve", "grid": "transmission", "n": 10000,
         "grid_seed": 0, "scen": 1024, "precision": "fp32", "policy": "newton", "lanes": 8,
         "threads": 1024},
        # an ordinary study of odd size with the default launch shape
        {"name": "odd batch", "kind": "solve", "grid": "transmission", "n": 3001,
         "grid_seed": 3, "scen": 333, "precision": "fp32", "policy": "clamped", "lanes": 0,
         "threads": 0},
        # the largest grid: few scenarios, a dense tail that no single block can hold
        {"name": "large grid", "kind": "solve", "grid": "transmission", "n": 30000,
         "grid_seed": 0, "scen": 8, "precision": "fp32", "policy": "clamped", "lanes": 8,
         "threads": 1024},
        # operational planning: load scenarios, N-1 outages and neighbouring grids in one launch
        {"name": "mixed studies", "kind": "mix", "n": 2000, "grid_seed": 0, "scen": 256,
         "outages": 64, "grids": 8},
        # optimisation through the power flow: forward and adjoint in FP64
        {"name": "gradient", "kind": "gradient", "n": 10000, "grid_seed": 0, "scen": 256,
         "precision": "fp64"},
        # a serving process: inputs and results in pinned host memory
        {"name": "host pipeline", "kind": "pipeline", "n": 10000, "grid_seed": 0, "scen": 512,
         "chunks": 4},
        # the general complex LU (the reference's ILUSolver)
        {"name": "sparse lu", "kind": "lu", "n": 3000, "grid_seed": 0},
        # admittances of 512 parameter scenarios (taps and phase shifts applied)
        {"name": "ybus scenarios", "kind": "ybus", "n": 10000, "grid_seed": 0, "scen": 512,
         "taps": True},
        # branch results (power, current, loading) of 512 solved scenarios
        {"name": "branch results", "kind": "flows", "n": 10000, "grid_seed": 0, "scen": 512,
         "taps": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges: grids of 50 to 12,000 buses (log-uniform, odd sizes
    as they come), 1 to 1024 scenarios, bounded by what the headline batch holds."""
    kind = rng.choice(["api", "solve", "solve", "solve", "solve", "feeder", "feeder", "mix",
                       "gradient", "pipeline", "lu", "ybus", "flows"])
    seed = rng.randrange(8)
    if kind == "api":
        return {"kind": "api", "grid": "feeder", "n": _log(rng, 20, 300), "grid_seed": seed}
    if kind == "feeder":
        return {"kind": "solve", "grid": "feeder", "n": _log(rng, 20, 300), "grid_seed": seed,
                "scen": _log(rng, 1, 1024), "precision": "fp64", "policy": "reference",
                "lanes": 0, "threads": 0}
    if kind == "solve":
        n = _log(rng, 50, 12000)
        precision = rng.choice(["fp32", "fp32", "fp64"])
        most = (6_000_000 if precision == "fp32" else 1_500_000) // n
        case = {"kind": "solve", "grid": "transmission", "n": n, "grid_seed": seed,
                "scen": _log(rng, 1, min(1024, most)), "precision": precision,
                "policy": rng.choice(["newton", "clamped"]), "lanes": 0, "threads": 0}
        if n >= 200 and rng.random() < 0.3:
            case["outages"] = True
            case["scen"] = min(case["scen"], n // 10, 256)
        return case
    if kind == "mix":
        return {"kind": "mix", "n": _log(rng, 500, 3000), "grid_seed": seed,
                "scen": _log(rng, 16, 512), "outages": _log(rng, 8, 32),
                "grids": rng.randrange(1, 9)}
    if kind == "gradient":
        n = _log(rng, 100, 10000)
        return {"kind": "gradient", "n": n, "grid_seed": seed,
                "scen": _log(rng, 1, min(256, 1_000_000 // n)),
                "precision": rng.choice(["fp64", "fp32"])}
    if kind == "pipeline":
        n = _log(rng, 500, 10000)
        return {"kind": "pipeline", "n": n, "grid_seed": seed,
                "scen": _log(rng, 32, min(1024, 4_000_000 // n)), "chunks": rng.randrange(1, 5)}
    if kind == "lu":
        return {"kind": "lu", "n": _log(rng, 50, 8000), "grid_seed": seed}
    n = _log(rng, 100, 12000)
    return {"kind": kind, "n": n, "grid_seed": seed,
            "scen": _log(rng, 1, min(1024, 6_000_000 // n)), "taps": rng.random() < 0.7}


# ----------------------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------------------

def _base(case):
    return 1e6 if case.get("grid") == "feeder" else workloads.BASE


@functools.lru_cache(maxsize=64)
def _network(grid, seed, n):
    if grid == "feeder":
        return synth.feeder_grid(seed, n=n)
    # above 10,000 buses the generator's loading has no solution for every scenario; half of it
    # has (as in the benchmark's large workload)
    return synth.transmission_grid(seed, n=n, load_scale=0.05 if n <= 10000 else 0.025)


def _net(case):
    return _network(case.get("grid", "transmission"), case["grid_seed"], case["n"])


@functools.lru_cache(maxsize=64)
def _start(seed, n):
    return synth.dc_start(_network("transmission", seed, n), workloads.BASE)


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _loads(case, seed, scen, stream=0):
    """S_spec complex128 [scen, n]: every load scaled by its own lognormal factor."""
    net, dev = _net(case), _device()
    s0 = torch.as_tensor(net.specified_power(_base(case)), device=dev)
    load = torch.complex(s0.real.clamp(max=0.0), s0.imag.clamp(max=0.0))
    g = torch.Generator(device=dev).manual_seed(int(seed) * 4 + stream)
    f = torch.randn((scen, net.n_bus), dtype=torch.float64, device=dev, generator=g).mul_(SIGMA).exp_()
    return (s0 - load) + f * load


def _branches(case, seed, scen):
    """Branch data [scen, m, 6]: r, x and b each within 10 % of the grid's."""
    net, dev = _net(case), _device()
    br = torch.as_tensor(branch_params(net), device=dev)
    g = torch.Generator(device=dev).manual_seed(int(seed) * 4 + 1)
    f = torch.rand((scen, br.shape[0], 3), dtype=torch.float64, device=dev, generator=g)
    out = br.expand(scen, -1, -1).clone()
    out[:, :, 0:2] *= 0.9 + 0.2 * f[:, :, :2]
    out[:, :, 3] *= 0.9 + 0.2 * f[:, :, 2]
    return out


def _mode(taps):
    return N.YBUS_TAPS if taps else N.YBUS_REFERENCE


def _zb(case):
    return float(_net(case).u_rated[0]) ** 2 / _base(case)


def _outage_list(case, count):
    return synth.n_minus_1(_net(case), count, seed=2 + case["grid_seed"])


def _neighbours(case):
    """The independent grids of a mix: sizes from 500 to 6,000 buses, one scenario each."""
    sizes = synth.grid_sizes(case["grids"], lo=500, hi=6000, seed=3 + case["grid_seed"])
    return [{"kind": "solve", "grid": "transmission", "n": int(n),
             "grid_seed": 100 + case["grid_seed"] + i} for i, n in enumerate(sizes)]


def _voltages(case, seed, scen):
    """Voltages as a solved grid has them: the DC start with a spread in angle and magnitude."""
    v0 = torch.as_tensor(_start(case["grid_seed"], case["n"]), device=_device())
    g = torch.Generator(device=v0.device).manual_seed(int(seed) * 4 + 2)
    f = torch.randn((2, scen, v0.numel()), dtype=torch.float64, device=v0.device, generator=g)
    return v0 * torch.polar(1.0 + 0.01 * f[0], 0.02 * f[1])


def prepare(case, seed):
    kind, net = case["kind"], _net(case)
    if kind == "api":
        import dataclasses

        s = _loads(case, seed, 1)[0].cpu().numpy() * _base(case)
        one = dataclasses.replace(net, p=np.ascontiguousarray(s.real), q=np.ascontiguousarray(s.imag))
        cfg = PowerFlowConfig(tolerance=1e-8, max_iterations=20, base_power=_base(case))
        return {"kind": kind, "solver": NewtonRaphson(), "net": one, "config": cfg}
    if kind == "ybus":
        return {"kind": kind, "plan": YbusPlan.from_network(net), "mode": _mode(case["taps"]),
                "branch": _branches(case, seed, case["scen"]), "zb": _zb(case),
                "shunt": torch.as_tensor(shunt_params(net), device="cuda")}
    if kind == "flows":
        return {"kind": kind, "net": net, "v": _voltages(case, seed, case["scen"]),
                "taps": case["taps"], "i_n": np.full(net.n_branch, 400.0)}
    if kind == "lu":
        plan = YbusPlan.from_network(net)
        br = _branches(case, seed, 1)[0]
        y = plan.assemble(br, torch.as_tensor(shunt_params(net), device="cuda"),
                          mode=N.YBUS_TAPS, scale=_zb(case))[0]
        # the loads as constant admittances on the diagonal, which also ground the grid
        s = _loads(case, seed, 1)[0]
        rows = torch.as_tensor(np.repeat(np.arange(net.n_bus), np.diff(plan.row_ptr)), device="cuda")
        diag = torch.nonzero(rows == torch.as_tensor(plan.col_idx, device="cuda"))[:, 0]
        y[diag] += s[rows[diag]].abs() + 0.01
        return {"kind": kind, "lu": SparseLU(plan.row_ptr, plan.col_idx), "y": y,
                "b": _voltages(case, seed, 1)[0]}
    if kind == "mix":
        v0 = _start(case["grid_seed"], case["n"])
        load = studies.load_study("load", net, _loads(case, seed, case["scen"]).cpu().numpy(), v0)
        outs = _outage_list(case, case["outages"])
        cont = studies.contingency_study("n-1", net, outs, _loads(case, seed, 1, 3)[0].cpu().numpy(),
                                         v0, plan=load.plan)
        every = [load, cont]
        for c in _neighbours(case):
            every.append(studies.load_study("grid", _net(c), _loads(c, seed, 1).cpu().numpy(),
                                            _start(c["grid_seed"], c["n"])))
        for st in every:
            st.make_batch()
        return {"kind": kind, "studies": every}
    if kind == "gradient":
        model = DifferentiablePowerFlow(net, case["scen"], base_power=_base(case),
                                        precision=case["precision"],
                                        v_init=_start(case["grid_seed"], case["n"]))
        s = _loads(case, seed, case["scen"])
        leaf = [s.real.contiguous(), s.imag.contiguous(), model.branch[:, 0].clone(),
                model.branch[:, 1].clone()]
        return {"kind": kind, "model": model, "leaf": [t.requires_grad_(True) for t in leaf]}
    # "solve" and "pipeline": one plan with its batch
    yp = YbusPlan.from_network(net)
    feeder = case.get("grid") == "feeder"
    y = yp.assemble(torch.as_tensor(branch_params(net), device="cuda"),
                    torch.as_tensor(shunt_params(net), device="cuda"), mode=_mode(not feeder),
                    scale=_zb(case))
    plan = NRPlan(yp.row_ptr, yp.col_idx, net.bus_type,
                  jacobian="reference" if feeder else "exact")
    s = _loads(case, seed, case["scen"])
    if kind == "pipeline":
        host = s.cpu().pin_memory()
        v0 = torch.as_tensor(_start(case["grid_seed"], case["n"])).pin_memory()
        pipe = HostPipeline(plan, case["scen"], chunks=case["chunks"], precision="fp32",
                            lanes=workloads.LANES, threads=workloads.THREADS)
        out = torch.empty_like(host).pin_memory()
        word = [torch.empty(case["scen"], dtype=torch.int32).pin_memory() for _ in range(2)]
        return {"kind": kind, "pipe": pipe, "y": y[0], "s": host, "v0": v0, "out": out,
                "status": word[0], "iterations": word[1], "kw": workloads.solve_kwargs()}
    if case.get("outages"):
        st = studies.contingency_study("n-1", net, _outage_list(case, case["scen"]),
                                       s.cpu().numpy(), _start(case["grid_seed"], case["n"]),
                                       plan=plan)
        y = st.y
    batch = NRBatch(plan, s.shape[0], precision=case["precision"], lanes=case["lanes"],
                    threads=case["threads"], y_shared=not case.get("outages"))
    kw = dict(tol=1e-8, max_iter=30, policy=case["policy"])
    if feeder:
        kw["u_pu"] = torch.as_tensor(net.u_pu.astype(np.float64), device="cuda")
    else:
        kw["v_init"] = torch.as_tensor(_start(case["grid_seed"], case["n"]), device="cuda")
    if case["precision"] == "fp32":
        kw.update(MIXED)
    return {"kind": kind, "batch": batch, "y": y if case.get("outages") else y[0], "s": s, "kw": kw}


def run(state):
    kind = state["kind"]
    if kind == "api":
        r = state["solver"].solve_power_flow(state["net"], None, state["config"])
        return {"v": r.bus_voltages, "s": r.bus_injections, "iterations": r.iterations,
                "converged": r.converged}
    if kind == "solve":
        r = state["batch"].solve(state["y"], state["s"], **state["kw"])
        return {"v": r.v, "iterations": r.iterations, "status": r.status}
    if kind == "mix":
        res = studies.solve_mixed(state["studies"], retry="clamped", **MIXED)
        return [{"v": r.v, "iterations": r.iterations, "status": r.status} for r in res]
    if kind == "gradient":
        model, (p, q, r, x) = state["model"], state["leaf"]
        vm, va = model(p, q, r, x)
        loss = ((vm - 1.0) ** 2).sum() + branch_losses_mw(vm, va, r, x, model).sum()
        grads = torch.autograd.grad(loss, (p, q, r, x))
        return {"vm": vm.detach(), "va": va.detach(), "loss": loss.detach(),
                "dp": grads[0], "dq": grads[1], "dr": grads[2], "dx": grads[3]}
    if kind == "pipeline":
        state["pipe"].solve(state["y"], state["s"], state["v0"], state["out"],
                            out_status=state["status"], out_iterations=state["iterations"],
                            **state["kw"])
        return {"v": state["out"], "iterations": state["iterations"], "status": state["status"]}
    if kind == "lu":
        ok = state["lu"].factorize(state["y"])
        return {"x": state["lu"].solve(state["b"]), "ok": ok}
    if kind == "ybus":
        return state["plan"].assemble(state["branch"], state["shunt"], mode=state["mode"],
                                      scale=state["zb"])
    return branch_flows(state["net"], state["v"], workloads.BASE, taps=state["taps"],
                        i_n=state["i_n"])


# ----------------------------------------------------------------------------------------
# what the work needs
# ----------------------------------------------------------------------------------------

@functools.lru_cache(maxsize=64)
def _newton_flops(grid, seed, n):
    """Operations of one Newton iteration of one scenario: the sparse block factorisation (a
    2x2 block product is 16), its dense trailing part, the triangular solves, the mismatch and
    the Jacobian."""
    net = _network(grid, seed, n)
    yp = YbusPlan.from_network(net)
    i = NRPlan(yp.row_ptr, yp.col_idx, net.bus_type).info
    tail = 2.0 * i["n_tail"]
    return (16.0 * i["n_pairs"] + 2.0 / 3.0 * tail ** 3 + 16.0 * i["nnz_l_blocks"] +
            2.0 * tail ** 2 + 60.0 * yp.nnz), yp.nnz, net.n_branch


def work(case):
    kind, n, scen = case["kind"], case["n"], case.get("scen", 1)
    flops, nnz, m = _newton_flops(case.get("grid", "transmission"), case["grid_seed"], n)
    if kind == "ybus":
        return {"bytes": scen * (48.0 * m + 16.0 * nnz), "flops": scen * 40.0 * m}
    if kind == "flows":
        return {"bytes": scen * (16.0 * n + 72.0 * m) + 48.0 * m, "flops": scen * 80.0 * m}
    if kind == "lu":
        return {"bytes": 16.0 * nnz + 32.0 * n, "flops": flops}
    if kind == "mix":
        parts = [(scen + case["outages"], n, flops, nnz)]
        for c in _neighbours(case):
            f, z, _ = _newton_flops("transmission", c["grid_seed"], c["n"])
            parts.append((1, c["n"], f, z))
        return {"bytes": sum(48.0 * k * s + 16.0 * z for s, k, _, z in parts) +
                case["outages"] * 16.0 * nnz, "flops": sum(6.0 * s * f for s, _, f, _ in parts)}
    steps = {"reference": 10, "clamped": 10}.get(case.get("policy"), 6)
    if kind == "api":
        steps = 10
    per = 32.0 * n + (16.0 * nnz if case.get("outages") else 0.0)
    extra = scen * 64.0 * n if kind == "gradient" else 0.0
    return {"bytes": scen * per + 16.0 * nnz + extra, "flops": scen * steps * flops}


# ----------------------------------------------------------------------------------------
# what the outputs are, in 64 bits, by plain torch on dense matrices
# ----------------------------------------------------------------------------------------

def _stamps(br, taps):
    """(ff, tt, ft, tf) of branch rows [..., 6] = (r, x, g, b, k, theta)."""
    y = 1.0 / torch.complex(br[..., 0], br[..., 1])
    end = y + torch.complex(br[..., 2], br[..., 3] / 2.0)
    if not taps:
        return end, end, -y, -y
    t = torch.polar(br[..., 4], br[..., 5])
    return end / br[..., 4] ** 2, end, -y / t.conj(), -y / t


class _Plain:
    """One grid's admittances as triplets (diagonal stamps kept apart), and its Newton solve."""

    def __init__(self, case, br, taps):
        net, dev = _net(case), br.device
        f, t, valid = net.branch_index()
        assert bool(np.all(valid))
        sb, sg, sbb = net.shunt_index()
        self.f, self.t = (torch.as_tensor(np.asarray(a), device=dev).long() for a in (f, t))
        self.n, self.zb, self.taps = net.n_bus, _zb(case), taps
        bt = torch.as_tensor(np.asarray(net.bus_type), device=dev)
        self.free = torch.nonzero(bt != 2)[:, 0]
        self.pq = torch.nonzero(bt == 0)[:, 0]
        self.sh = torch.zeros(self.n, dtype=torch.complex128, device=dev)
        if len(sb):
            self.sh.index_add_(0, torch.as_tensor(np.asarray(sb), device=dev).long(),
                               torch.complex(*(torch.as_tensor(np.asarray(a, np.float64), device=dev)
                                               for a in (sg, sbb))))
        self.stamp(br)

    def stamp(self, br):
        self.br = br
        self.y = [s * self.zb for s in _stamps(br, self.taps)]
        return self

    def current(self, v):
        """I = Y V for v [S, n]."""
        ff, tt, ft, tf = self.y
        out = v * (self.sh * self.zb)
        vf, vt = v[:, self.f], v[:, self.t]
        out.index_add_(1, self.f, ff * vf + ft * vt)
        return out.index_add_(1, self.t, tf * vf + tt * vt)

    def dense(self, s):
        """Y [n, n] of scenario s."""
        ff, tt, ft, tf = [a if a.dim() == 1 else a[s] for a in self.y]
        m = torch.diag(self.sh * self.zb)
        for r, c, a in ((self.f, self.f, ff), (self.t, self.t, tt), (self.f, self.t, ft), (self.t, self.f, tf)):
            m.index_put_((r, c), a, accumulate=True)
        return m

    def jacobian(self, v, s):
        """d(P, Q) / d(theta, |V|) at v [n] over the free angles and the PQ magnitudes."""
        y = self.dense(s)
        i = y @ v
        a = 1j * v[:, None] * (torch.diag(i) - y * v).conj()
        b = v[:, None] * (y * (v / v.abs())).conj() + torch.diag(i.conj() * v / v.abs())
        fr, pq = self.free, self.pq
        return torch.cat([torch.cat([a.real[fr][:, fr], b.real[fr][:, pq]], 1),
                          torch.cat([a.imag[pq][:, fr], b.imag[pq][:, pq]], 1)], 0)

    def residual(self, v, spec):
        d = v * self.current(v).conj() - spec
        return torch.cat([d.real[:, self.free], d.imag[:, self.pq]], 1)

    def step(self, v, dx):
        a, m = torch.angle(v), v.abs()
        a[:, self.free] -= dx[:, : self.free.numel()]
        m[:, self.pq] -= dx[:, self.free.numel():]
        return torch.polar(m, a)

    def solve(self, spec, v0):
        """Scenario 0 by Newton, then all of them with its factors, and the ones that this does
        not bring to 1e-13 by Newton of their own; None when some do not get there."""
        v = v0.expand(spec.shape[0], -1).clone()
        one = _Plain.__new__(_Plain)
        one.__dict__.update(self.__dict__)
        one.y = [a if a.dim() == 1 else a[:1] for a in self.y]
        w = v[:1]
        for _ in range(30):
            f = one.residual(w, spec[:1])
            if float(f.abs().max()) < 1e-11:
                break
            w = one.step(w, _limit(torch.linalg.solve(self.jacobian(w[0], 0), f[0])[None]))
        lu = torch.linalg.lu_factor(self.jacobian(w[0], 0))
        v = w.abs() * torch.exp(1j * torch.angle(w)) * torch.ones_like(v)
        best = None
        for _ in range(60):
            f = self.residual(v, spec)
            worst = f.abs().amax(1)
            if not bool(torch.isfinite(worst).all()) or float(worst.max()) < 1e-13 or (
                    best is not None and float(worst.max()) < 1e-10 and float(worst.max()) > 0.7 * best):
                break
            best = float(worst.max())
            v = self.step(v, torch.linalg.lu_solve(*lu, f.T).T)
        late = torch.nonzero(~(self.residual(v, spec).abs().amax(1) < 1e-9))[:, 0].tolist()
        if len(late) > 64 or self.n > 4000 and late:
            return None
        for s in late:
            self_y, u = self.y, v0.reshape(-1, self.n)[:1].clone()
            self.y = [a if a.dim() == 1 else a[s:s + 1] for a in self_y]
            for _ in range(30):
                f = self.residual(u, spec[s:s + 1])
                if float(f.abs().max()) < 1e-12:
                    break
                u = self.step(u, _limit(torch.linalg.solve(self.jacobian(u[0], 0), f[0])[None]))
            self.y = self_y
            v[s] = u[0]
        return v if bool((self.residual(v, spec).abs().amax(1) < 1e-9).all()) else None


def _limit(dx):
    return dx.clamp(-0.5, 0.5)


def _plain(case, taps=True):
    br = torch.as_tensor(branch_params(_net(case)), device=_device())
    return _Plain(case, br, taps)


def _solved(case, spec, outages=None, v0=None):
    g = _plain(case, taps=case.get("grid") != "feeder")
    if outages is not None:
        # an outage is the branch without its stamps
        keep = torch.ones((len(outages), g.br.shape[0]), dtype=torch.float64, device=spec.device)
        keep[torch.arange(len(outages)), torch.as_tensor(np.asarray(outages), device=spec.device)] = 0.0
        g.y = [a * keep for a in g.y]
    if v0 is None:
        net = _net(case)
        v0 = (torch.as_tensor(np.where(net.bus_type == 0, 1.0, net.u_pu), device=spec.device) + 0j
              if case.get("grid") == "feeder" else
              torch.as_tensor(_start(case["grid_seed"], case["n"]), device=spec.device))
    return g, g.solve(spec, v0)


def _exact_gradient(case, seed):
    spec = _loads(case, seed, case["scen"])
    g, v = _solved(case, spec)
    if v is None:
        return None
    r, x = (g.br[:, i].clone().requires_grad_(True) for i in (0, 1))
    br = torch.cat([r[:, None], x[:, None], g.br[:, 2:]], 1)
    vm, va = v.abs().requires_grad_(True), torch.angle(v).requires_grad_(True)
    g.stamp(br)

    def loss_of(vm, va):
        u = torch.polar(vm, va)
        uf, ut = u[:, g.f], u[:, g.t]
        ff, tt, ft, tf = g.y
        loss = uf * (ff * uf + ft * ut).conj() + ut * (tf * uf + tt * ut).conj()
        return ((vm - 1.0) ** 2).sum() + loss.real.sum() * (_base(case) / 1e6)

    loss = loss_of(vm, va)
    gm, ga, lr, lx = torch.autograd.grad(loss, (vm, va, r, x), retain_graph=True)
    rhs = torch.cat([ga[:, g.free], gm[:, g.pq]], 1)
    # J^T lam = dL/d(theta, |V|): scenario 0's factors as a preconditioner of each one's own J^T
    at = torch.polar(vm.detach(), va.detach())
    lu = torch.linalg.lu_factor(g.jacobian(at[0], 0).detach())
    lam = torch.zeros_like(rhs)
    res = g.residual(torch.polar(vm, va), spec)
    for k in range(80):
        jt = torch.autograd.grad(res, (va, vm), lam, retain_graph=True)
        d = rhs - torch.cat([jt[0][:, g.free], jt[1][:, g.pq]], 1)
        if float(d.abs().max()) < 1e-13 * float(rhs.abs().max()):
            break
        lam = lam + torch.linalg.lu_solve(*lu, d.T, adjoint=True).T
    if float(d.abs().max()) > 1e-9 * float(rhs.abs().max()):
        return None
    jr, jx = torch.autograd.grad(res, (r, x), lam)
    dp, dq = torch.zeros_like(vm), torch.zeros_like(vm)
    dp[:, g.free] = lam[:, : g.free.numel()]
    dq[:, g.pq] = lam[:, g.free.numel():]
    return {"vm": vm.detach(), "va": va.detach(), "loss": loss.detach(), "dp": dp.detach(),
            "dq": dq.detach(), "dr": lr - jr, "dx": lx - jx}


def exact(case, seed):
    """What run() returns, in 64 bits; None where the dense matrices would take too long."""
    kind, n = case["kind"], case["n"]
    if n > 12000:
        return None  # a dense Jacobian of the 30,000-bus grid does not fit a card's time
    torch.set_grad_enabled(kind == "gradient")
    try:
        if kind == "ybus":
            return _exact_ybus(case, seed)
        if kind == "flows":
            return _exact_flows(case, seed)
        if kind == "lu":
            g = _plain(case).stamp(_branches(case, seed, 1)[0])
            a = g.dense(0) + torch.diag(_loads(case, seed, 1)[0].abs() + 0.01)
            return {"x": torch.linalg.solve(a, _voltages(case, seed, 1)[0]), "ok": None}
        if kind == "gradient":
            return _exact_gradient(case, seed)
        if kind == "mix":
            parts = [_solved(case, _loads(case, seed, case["scen"]))[1],
                     _solved(case, _loads(case, seed, 1, 3).expand(case["outages"], -1),
                             _outage_list(case, case["outages"]))[1]]
            parts += [_solved(c, _loads(c, seed, 1))[1] for c in _neighbours(case)]
            return [{"v": v, "iterations": None, "status": None} for v in parts]
        scen = case.get("scen", 1)
        g, v = _solved(case, _loads(case, seed, scen),
                       _outage_list(case, scen) if case.get("outages") else None)
        if v is None:
            return None
        if kind == "api":
            s = v * g.current(v).conj()
            return {"v": v[0], "s": s[0], "iterations": None, "converged": None}
        return {"v": v, "iterations": None, "status": None}
    finally:
        torch.set_grad_enabled(True)


def _exact_ybus(case, seed):
    g, br = _plain(case, case["taps"]), _branches(case, seed, case["scen"])
    # one slot per entry, by row and column: the generator's grids have no parallel branches
    bus = torch.arange(g.n, device=br.device)
    entries = [a * g.n + b for a, b in ((g.f, g.f), (g.t, g.t), (g.f, g.t), (g.t, g.f), (bus, bus))]
    key = torch.unique(torch.cat(entries))
    where = [torch.searchsorted(key, e) for e in entries]
    out = torch.zeros((case["scen"], key.numel()), dtype=torch.complex128, device=br.device)
    out[:, where.pop()] += g.sh
    for w, a in zip(where, _stamps(br, case["taps"])):
        out.index_add_(1, w, a)
    return out * g.zb


def _exact_flows(case, seed):
    net, g = _net(case), _plain(case, case["taps"])
    v = _voltages(case, seed, case["scen"])
    ff, tt, ft, tf = g.y
    vf, vt = v[:, g.f], v[:, g.t]
    out = torch.zeros((case["scen"], net.n_branch, 9), dtype=torch.float64, device=v.device)
    for c, (u, i) in enumerate(((vf, ff * vf + ft * vt), (vt, tf * vf + tt * vt))):
        s = u * i.conj() * workloads.BASE
        amp = s.abs() / (math.sqrt(3.0) * float(net.u_rated[0]) * u.abs())
        for k, a in enumerate((s.real, s.imag, amp, s.abs())):
            out[:, :, 4 * c + k] = a
    out[:, :, 8] = torch.maximum(out[:, :, 2], out[:, :, 6]) / 400.0
    return out
