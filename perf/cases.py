"""Workloads of the batched GGA solver and its implicit adjoint, one function
per step of a measurement: `listed` and `draw` name the cases, `prepare` makes
what a program holds before the call (network, solver with its plan, inputs on
the GPU), `run` is one pass through the public entry points, `work` the bytes
and operations the pass cannot do without, and `exact` the same results from
plain dense torch in 64 bits.

Kinds of case, each with the range its cases are drawn from:

* steady       `GGASolver.solve`: a hydraulic solve at EPANET's own accuracy,
               one network state up to a few thousand (31 to 3000 junctions).
* implicit     `implicit_solve` and its backward: calibration and control
               steps, gradients of measured heads and flows w.r.t. demands,
               emitters and resistances; looped networks, networks with
               pressure reducing valves or throttle control valves; 1 to
               16384 scenarios.  (The opt-in FP32 factor has no case: on
               these networks it is refused for some of every few hundred
               scenarios.)
* pumps        the same with pump speeds and curve coefficients as parameters.
* multi        `implicit_solve_multi`: networks of four sizes in one launch.
* unrolled     `solve_unrolled` and its backward: K fixed iterations.
* sensitivity  `sensitivity_matrix`: every sensor of several frames.
* eps          `eps_solve` and its backward: hourly frames of a district-size
               network with tanks and pumps.
"""
from functools import lru_cache
from math import exp, log, log2

import numpy as np
import torch

from wdsgpu_b200 import synth
from wdsgpu_b200.autodiff import implicit_solve, solve_unrolled
from wdsgpu_b200.eps import eps_solve
from wdsgpu_b200.multi import implicit_solve_multi
from wdsgpu_b200.sensitivity import sensitivity_matrix
from wdsgpu_b200.solver import GGASolver

DEV = "cuda"
N_SENSORS = 30


# ---------------------------------------------------------------- cases
def listed():
    case = lambda name, kind, **k: dict(name=name, kind=kind, **k)
    return [
        # one state of a small village network: the smallest call there is
        case("steady_31_b1", "steady", net="looped", junctions=31, batch=1, accuracy=1e-3),
        # a Monte-Carlo of demands on a town network, heads and flows only
        case("steady_782_b256", "steady", net="looped", junctions=782, batch=256, accuracy=1e-3),
        # one gradient of one state: an optimiser that steps through a day
        case("implicit_100_b1", "implicit", net="looped", junctions=100, batch=1, accuracy=1e-6,
             meters=4),
        # the benchmark's step: 1024 scenarios of the 782-junction network with 3 PRVs
        case("implicit_782_b1024", "implicit", net="prv", junctions=782, batch=1024,
             accuracy=1e-6, meters=0),
        # the same network as a large ensemble
        case("implicit_782_b16384", "implicit", net="prv", junctions=782, batch=16384,
             accuracy=1e-6, meters=0),
        # a network whose state is too large for shared memory, an odd batch
        case("implicit_3000_b33", "implicit", net="looped", junctions=3000, batch=33,
             accuracy=1e-6, meters=8),
        # throttle control valves, a batch smaller than the GPU
        case("implicit_542_b97", "implicit", net="tcv", junctions=542, batch=97, accuracy=1e-7,
             meters=5),
        # pump schedules of a supply zone: per-scenario speeds, gradients of the curves
        case("pumps_301_b96", "pumps", junctions=301, batch=96, accuracy=1e-8, meters=4),
        # 256 instances of four networks (100 to 3000 junctions) in one launch per pass
        case("multi_256", "multi", junctions=3000, batch=256, accuracy=1e-6),
        # fixed iterations differentiated through: learned models that unroll the solver
        case("unrolled_782_b513", "unrolled", junctions=782, batch=513, iterations=14),
        # sensor placement: 30 sensors of 16 demand frames
        case("sensitivity_782_t16", "sensitivity", junctions=782, batch=16, accuracy=1e-8),
        # a quarter of a day of a district with 20 000 junctions, 64 scenarios
        case("eps_20000_b64", "eps", junctions=20000, batch=64, periods=6, accuracy=1e-6),
    ]


def _log(rng, lo, hi):
    return int(round(exp(rng.uniform(log(lo), log(hi)))))


def draw(rng):
    kind = rng.choice(["steady", "implicit", "implicit", "implicit", "pumps", "multi",
                       "unrolled", "sensitivity", "eps"])
    c = dict(kind=kind)
    if kind == "eps":
        c["junctions"] = _log(rng, 5000, 20000)
        c["batch"] = min(_log(rng, 4, 64), 1200000 // c["junctions"])
        c.update(periods=rng.randint(3, 6), accuracy=1e-6)
        return c
    c["junctions"] = _log(rng, 31, 3000)
    # networks above about a thousand junctions run from global memory: fewer scenarios
    cap = 16384 if c["junctions"] <= 800 else 64
    if kind == "multi":
        c["junctions"] = _log(rng, 1000, 3000)
        c.update(batch=_log(rng, 16, 256), accuracy=1e-6)
    elif kind == "unrolled":
        c["junctions"] = _log(rng, 31, 800)
        c.update(batch=_log(rng, 1, 513), iterations=rng.randint(4, 14))
    elif kind == "sensitivity":
        c["junctions"] = _log(rng, 100, 800)
        c.update(batch=_log(rng, 1, 24), accuracy=1e-8)
    elif kind == "pumps":
        c["junctions"] = _log(rng, 60, 800)
        c.update(batch=_log(rng, 1, 512), accuracy=10.0 ** -rng.randint(6, 8), meters=rng.randint(0, 6))
    elif kind == "steady":
        c.update(net="looped", batch=_log(rng, 1, min(cap, 4096)), accuracy=10.0 ** -rng.randint(3, 6))
    else:
        c["net"] = rng.choice(["looped", "prv", "tcv"]) if c["junctions"] >= 300 else "looped"
        c.update(batch=_log(rng, 1, cap), accuracy=10.0 ** -rng.randint(6, 8),
                 meters=rng.randint(0, 8))
    return c


# ---------------------------------------------------------------- networks
@lru_cache(maxsize=None)
def _network(shape, n):
    """The network of a case: fixed by its shape and number of junctions (the
    benchmark's own at 782 junctions with PRVs)."""
    if shape == "prv":
        if n == 782:
            return synth.config2_network()
        for n_prv in (3, 2, 1, 0):  # as many pressure zones as the graph has room for
            try:
                return synth.looped_network(2, n, 2, round(1.157 * n), n_prv=n_prv,
                                            zone_size=(n // 31, n // 11), n_emitters=n // 39)
            except RuntimeError:
                continue
    if shape == "tcv":
        return synth.tcv_network(4, n_junc=n, n_links=round(1.022 * n), n_tcv=n // 7)
    if shape == "pumps":
        return synth.eps_network(7, n_junc=n, n_pipes=round(1.2 * n))
    return synth.looped_network(3, n, 1 if n < 300 else 2, round(1.2 * n),
                                n_emitters=min(20, n // 20))


@lru_cache(maxsize=None)
def _eps_network(n):
    """District network whose tanks sit on the grade line of a steady solve
    with the tanks as junctions, as an operator's model has them."""
    size = dict(seed=5, n_junc=n, n_pipes=round(1.15 * n), base_lps=(0.02, 0.08), spacing_m=120.0)
    net0 = synth.eps_network(**size)
    pre = synth.tanks_as_junctions(net0)
    o = GGASolver(pre, device=DEV, dense_status_machine=True).solve(
        pre.demand_cfs_at(0)[None] * synth.diurnal(0.0),
        np.nan_to_num(pre.fixed_head_ft_at(0))[None], status_machine=True, accuracy=1e-8)
    centre = o["head_ft"][0].cpu().numpy()[np.asarray(net0.tank_node)]
    return synth.eps_network(tank_center_ft=centre, **size)


def _multi_networks(n):
    return [_network("looped", 100), _network("tcv", 542), _network("prv", 782),
            _network("looped", n)]


def _demands(net, batch, seed, sigma):
    """Base demands times a lognormal factor per scenario and node, [B, N]."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    base = torch.as_tensor(net.demand_cfs_at(0), device=DEV)
    z = torch.randn(batch, net.N, generator=g, device=DEV, dtype=torch.float64)
    return base * torch.exp(sigma * z)


def _fixed(net, batch):
    rh = torch.as_tensor(np.nan_to_num(net.fixed_head_ft_at(0)), device=DEV)
    return rh.expand(batch, -1).contiguous()


def _inputs(case, seed):
    """Networks and device inputs of a case (no solver), for prepare and exact."""
    kind, B = case["kind"], case["batch"]
    if kind == "eps":
        net = _eps_network(case["junctions"])
        g = torch.Generator(device=DEV).manual_seed(seed)
        base = torch.as_tensor(net.demand_cfs_at(0), device=DEV)
        P = case["periods"]
        day = torch.as_tensor(synth.diurnal(np.arange(P)), device=DEV)[:, None, None]
        z = torch.randn(P, B, net.N, generator=g, device=DEV, dtype=torch.float64)
        return [net], dict(d=base * day * torch.exp(0.15 * z))
    if kind == "multi":
        nets = _multi_networks(case["junctions"])
        counts = [max(1, B // 4 + (1 if i < B % 4 else 0)) for i in range(4)]
        return nets, dict(d=[_demands(m, c, 7 * seed + i, 0.3)
                             for i, (m, c) in enumerate(zip(nets, counts))],
                          rh=[_fixed(m, c) for m, c in zip(nets, counts)])
    net = _network("pumps" if kind == "pumps" else case.get("net", "looped"), case["junctions"])
    s = dict(d=_demands(net, B, seed, 0.2), rh=_fixed(net, B),
             ke=torch.as_tensor(net.node_ke, device=DEV),
             r=torch.as_tensor(net.r_hw, device=DEV),
             sens=torch.as_tensor(_sensors(net), device=DEV),
             meters=torch.as_tensor(_meters(net, case.get("meters", 0)), device=DEV))
    if kind == "pumps":
        g = torch.Generator(device=DEV).manual_seed(seed + 1)
        pl = torch.as_tensor(np.asarray(net.pump_link, dtype=np.int64), device=DEV)
        row = lambda v: torch.zeros(net.L, dtype=torch.float64, device=DEV).index_put_(
            (pl,), torch.as_tensor(v, device=DEV))
        speed = torch.as_tensor(_settings(net), device=DEV).expand(B, -1).clone()
        u = torch.rand(B, pl.numel(), generator=g, device=DEV, dtype=torch.float64)
        speed[:, pl] = 0.95 + 0.1 * u
        s.update(speed=speed, h0=row(net.pump_h0), pr=row(net.pump_r))
    return [net], s


def _settings(net):
    """Link settings as the solver holds them: pump speeds, missing elsewhere."""
    return GGASolver(net, device=DEV, dense_status_machine=True).init_setting


def _sensors(net):
    n = int((np.asarray(net.node_type) == synth.JUNCTION).sum())
    return synth.sensor_nodes(net, min(N_SENSORS, n // 3))


def _meters(net, n):
    rng = np.random.default_rng(1)
    return np.sort(rng.choice(np.flatnonzero(np.asarray(net.link_type) == synth.PIPE), n,
                              replace=False))


def prepare(case, seed):
    nets, s = _inputs(case, seed)
    kind = case["kind"]
    solvers = []
    for i, net in enumerate(nets):
        g = GGASolver(net, device=DEV, dense_status_machine=kind not in ("steady", "unrolled"))
        g.plan(s["d"][i].shape[0] if kind == "multi" else case["batch"])
        solvers.append(g)
    if kind == "multi":
        s["sens"] = [torch.as_tensor(_sensors(m), device=DEV) for m in nets]
    if kind == "eps":
        s["sens"] = torch.arange(0, nets[0].N, 200, device=DEV)
    if kind == "sensitivity":
        s["sensors"] = _sensors(nets[0])
    s.update(case=case, solvers=solvers)
    return s


# ---------------------------------------------------------------- one pass
def _leaf(x):
    return x.detach().requires_grad_(True)


def _loss(s, head, flow):
    """Squared heads at the sensors and squared flows at the meters."""
    loss = (head.index_select(1, s["sens"]) ** 2).sum()
    if s["meters"].numel():
        loss = loss + (flow.index_select(1, s["meters"]) ** 2).sum()
    return loss


def run(s):
    case, g = s["case"], s["solvers"][0]
    kind = case["kind"]
    if kind == "steady":
        # relerr and the condition proxy are left out: the size of a last
        # correction is noise once the solve has converged
        o = g.solve(s["d"], s["rh"], accuracy=case["accuracy"])
        return {k: o[k] for k in ("head_ft", "flow_cfs", "emitter_cfs", "iters")}
    if kind == "implicit":
        x = [_leaf(s[k]) for k in ("d", "rh", "ke", "r")]
        out = implicit_solve(g, x[0], x[1], ke=x[2], r_hw=x[3], accuracy=case["accuracy"])
        return dict(out=_plain(out), grads=torch.autograd.grad(_loss(s, *out[:2]), x))
    if kind == "pumps":
        x = [_leaf(s[k]) for k in ("d", "rh", "r", "speed", "h0", "pr")]
        out = implicit_solve(g, x[0], x[1], r_hw=x[2], speed=x[3], pump_h0=x[4], pump_r=x[5],
                             accuracy=case["accuracy"])
        return dict(out=_plain(out), grads=torch.autograd.grad(_loss(s, *out[:2]), x))
    if kind == "multi":
        x = [_leaf(d) for d in s["d"]]
        r = [_leaf(p.r_hw) for p in s["solvers"]]
        outs = implicit_solve_multi(s["solvers"], x, s["rh"], r_hws=r, accuracy=case["accuracy"])
        loss = sum((o[0].index_select(1, k) ** 2).sum() for o, k in zip(outs, s["sens"]))
        return dict(out=[_plain(o) for o in outs], grads=torch.autograd.grad(loss, x + r))
    if kind == "unrolled":
        x = [_leaf(s[k]) for k in ("d", "rh", "ke", "r")]
        o = solve_unrolled(g, x[0], x[1], ke=x[2], r_hw=x[3], K=case["iterations"])
        out = (o["head_ft"], o["flow_cfs"], o["emitter_cfs"])
        return dict(out=_plain(out), grads=torch.autograd.grad(_loss(s, *out[:2]), x))
    if kind == "sensitivity":
        return sensitivity_matrix(g, s["d"], s["rh"], s["r"], s["sensors"], wrt="r",
                                  accuracy=case["accuracy"])
    x = [_leaf(s["d"])]
    o = eps_solve(g, x[0], accuracy=case["accuracy"])
    loss = (o["head"].index_select(2, s["sens"]) ** 2).sum() + (o["tank_head"][-1] ** 2).sum()
    grad = torch.autograd.grad(loss, x)
    return dict(head=o["head"].detach(), flow=o["flow"].detach(),
                tank_head=o["tank_head"].detach(), t_sec=o["t_sec"], status=o["status"],
                grads=grad)


def _plain(out):
    return [t.detach() for t in out]


# ---------------------------------------------------------------- work
def _state_work(n, links, iters):
    """Operations of one scenario: per iteration about 60 for a link's
    coefficients and update, and a sparse factor with its two substitutions,
    about 31 n log2 n for the nearly planar networks here."""
    return iters * (60.0 * links + 31.0 * n * log2(max(n, 2)))


def work(case):
    """Each input read once and each output written once, in float64, and the
    operations of the iterations (about 8, plus 3 polish steps and one
    adjoint where there is a gradient)."""
    kind, B, n = case["kind"], case["batch"], case["junctions"]
    links = 1.2 * n
    if kind == "steady":
        return dict(bytes=8.0 * B * (2 * n + 2 * n + links), flops=B * _state_work(n, links, 6))
    if kind == "multi":
        sizes = (100, 542, 782, n)
        return dict(bytes=sum(8.0 * B / 4 * (7 * m + 2 * 1.2 * m) for m in sizes),
                    flops=sum(B / 4 * _state_work(m, 1.2 * m, 12) for m in sizes))
    if kind == "unrolled":
        return dict(bytes=8.0 * B * (7 * n + 2 * links),
                    flops=B * _state_work(n, links, 2 * case["iterations"]))
    if kind == "sensitivity":
        m = min(N_SENSORS, n // 3)
        return dict(bytes=8.0 * B * (2 * n + m * links),
                    flops=B * (_state_work(n, links, 11) + m * 20.0 * n * log2(n)))
    if kind == "eps":
        F = case["periods"]
        return dict(bytes=8.0 * B * F * (4 * n + 2 * links),
                    flops=B * F * _state_work(n, links, 10))
    return dict(bytes=8.0 * B * (7 * n + 2 * links), flops=B * _state_work(n, links, 12))


# ---------------------------------------------------------------- plain 64-bit results
CSMALL, CBIG, RQTOL, HTOL, QTOL = 1e-6, 1e8, 1e-7, 0.0005, 0.0001
CLOSED, OPEN, ACTIVE = 2, 3, 4


class _Solve(torch.autograd.Function):
    """x = A^-1 b with A the junction matrix of conductances P and a diagonal."""

    @staticmethod
    def forward(ctx, m, P, diag, b):
        c = torch.linalg.cholesky(m.matrix(P, diag))
        x = m.refined(c, P, diag, b)
        ctx.m = m
        ctx.save_for_backward(c, P, diag, x)
        return x

    @staticmethod
    def backward(ctx, g):
        c, P, diag, x = ctx.saved_tensors
        w = ctx.m.refined(c, P, diag, g)
        return None, -ctx.m.along(w) * ctx.m.along(x), -w * x, w


class _Dense:
    """One network's equations in dense torch: head losses, the junction
    matrix and its solve.  Valve statuses are an argument."""

    def __init__(self, net):
        t = lambda a, dt=torch.float64: torch.as_tensor(np.asarray(a), dtype=dt, device=DEV)
        self.N, self.L = net.N, net.L
        nt = np.asarray(net.node_type)
        self.junc = t(np.flatnonzero(nt == 0), torch.int64)
        self.n = int(self.junc.numel())
        row = np.full(net.N, self.n, dtype=np.int64)   # fixed nodes share a scrap row
        row[nt == 0] = np.arange(self.n)
        n1, n2 = np.asarray(net.link_n1, np.int64), np.asarray(net.link_n2, np.int64)
        self.n1, self.n2 = t(n1, torch.int64), t(n2, torch.int64)
        self.r1, self.r2 = t(row[n1], torch.int64), t(row[n2], torch.int64)
        self.el = t(net.elev_ft)
        lt, st = np.asarray(net.link_type), np.asarray(net.init_status)
        setting = np.asarray(net.valve_setting_user, dtype=np.float64)
        diam = np.asarray(net.diam_ft, dtype=np.float64)
        self.pipe = t(lt <= synth.PIPE, torch.bool)
        self.pump = t(lt == synth.PUMP, torch.bool)
        km = np.zeros(net.L)
        tcv = lt == synth.TCV
        km[tcv] = 0.02517 * setting[tcv] / diam[tcv] ** 4
        self.km = t(km)
        self.closed = t(st == 0, torch.bool)
        pl = np.asarray(net.pump_link if net.pump_link is not None else [], dtype=np.int64)
        full = lambda v: np.bincount(pl, np.asarray(v, np.float64), net.L) if pl.size else np.zeros(net.L)
        self.h0, self.pr = t(full(net.pump_h0 if pl.size else [])), t(full(net.pump_r if pl.size else []))
        self.pn = t(full(net.pump_n) if pl.size else np.ones(net.L))
        self.hmax = t(full(net.pump_hmax if pl.size else []))
        self.speed = t(np.where(lt == synth.PUMP, setting, 1.0))
        q0 = 3.141592654 * diam ** 2 / 4.0
        if pl.size:
            q0[pl] = setting[pl] * np.asarray(net.pump_q0)
        self.q0 = t(np.where(st == 0, 1e-6, q0))
        v = np.flatnonzero(lt == synth.PRV)
        self.prv, self.jo, self.jc = t(v, torch.int64), t(row[n1[v]], torch.int64), t(row[n2[v]], torch.int64)
        self.hset = self.el[self.n2[self.prv]] + t(setting[v]) / synth.MperFT

    def loss(self, q, r, speed, h0, pr, status):
        """Head loss of every link at flow q."""
        sgn = torch.where(q < 0, -1.0, 1.0)
        qa = (q * sgn).clamp_min(1e-30)
        hg = 1.852 * r * qa ** 0.852
        hl = torch.where(hg < RQTOL, RQTOL * q, r * qa ** 1.852 * sgn)
        hv = torch.where(2 * self.km * qa < RQTOL, RQTOL * q, self.km * qa * q)
        hv = torch.where(self.km > 0, hv, CSMALL * q)
        hl = torch.where(self.pipe, hl, hv)
        re = pr * speed ** (2.0 - self.pn)
        slope = self.pn * re * qa ** (self.pn - 1.0)
        hp = speed * speed * h0 + torch.where(slope < RQTOL, RQTOL * q,
                                              re * qa ** (self.pn - 1.0) * q)
        hl = torch.where(self.pump, hp, hl)
        return torch.where(self.closed | (status <= CLOSED), CBIG * q, hl)

    def emitter(self, e, ke):
        ea = e.abs().clamp_min(1e-30)
        k = ke.clamp_min(CSMALL)
        return torch.where(2.0 * k * ea < RQTOL, RQTOL * e, k * ea * e)

    def slopes(self, q, e, r, ke, speed, h0, pr, status):
        with torch.enable_grad():
            q_, e_ = _leaf(q), _leaf(e)
            hl = self.loss(q_, r, speed, h0, pr, status)
            he = self.emitter(e_, ke)
            hg, = torch.autograd.grad(hl.sum(), q_)
            hge, = torch.autograd.grad(he.sum(), e_)
        return hl.detach(), hg, he.detach(), hge

    def scatter(self, v1, v2):
        """Junction sums of a value at each link's first and second end."""
        out = torch.zeros(v1.shape[0], self.n + 1, dtype=torch.float64, device=DEV)
        return out.index_add(1, self.r1, v1).index_add(1, self.r2, v2)[:, :self.n]

    def matrix(self, P, diag):
        B, m = P.shape[0], self.n + 1
        A = torch.zeros(B, m * m, dtype=torch.float64, device=DEV)
        for a, b, sg in ((self.r1, self.r1, 1), (self.r2, self.r2, 1), (self.r1, self.r2, -1),
                         (self.r2, self.r1, -1)):
            A = A.index_add(1, a * m + b, sg * P)
        A = A.view(B, m, m)[:, :self.n, :self.n]
        return A + torch.diag_embed(diag)

    def along(self, x):
        """Difference of a junction vector along each link (0 at fixed ends)."""
        x = torch.cat([x, x.new_zeros(x.shape[0], 1)], 1)
        return x[:, self.r1] - x[:, self.r2]

    def times(self, P, diag, x):
        """The junction matrix times x, link by link: the matrix itself holds
        the sum of conductances that differ by many orders."""
        t = P * self.along(x)
        return self.scatter(t, -t) + diag * x

    def refined(self, c, P, diag, b):
        x = torch.cholesky_solve(b.unsqueeze(-1), c).squeeze(-1)
        for _ in range(3):
            res = b - self.times(P, diag, x)
            x = x + torch.cholesky_solve(res.unsqueeze(-1), c).squeeze(-1)
        return x

    def solve(self, P, diag, rhs, act, con, transposed):
        """Junction unknowns and, per valve, its flow (or multiplier): rows of
        ACTIVE valves hold the head of jc (transposed: the constraint's)."""
        p = self.prv.numel()
        A = self.matrix(P, diag)
        if p == 0:
            x = self.refined(torch.linalg.cholesky(A), P, diag, rhs)
            return x, rhs.new_zeros(rhs.shape[0], 0)
        B, n = rhs.shape
        K = torch.zeros(B, n + p, n + p, dtype=torch.float64, device=DEV)
        K[:, :n, :n] = A
        i = torch.arange(p, device=DEV)
        a = act.to(torch.float64)
        col = torch.zeros(B, n, p, dtype=torch.float64, device=DEV)
        col[:, self.jc, i] = -a
        col[:, self.jo, i] = a
        row = torch.zeros(B, p, n, dtype=torch.float64, device=DEV)
        row[:, i, self.jc] = a
        if transposed:
            row, col = col.transpose(1, 2), row.transpose(1, 2)
        K[:, :n, n:], K[:, n:, :n] = col, row
        K[:, n + i, n + i] = 1.0 - a
        lu = torch.linalg.lu_factor(K)
        con = con * a
        back = lambda u, v: torch.linalg.lu_solve(*lu, torch.cat([u, v], 1).unsqueeze(-1))[..., 0]
        mul = lambda M, v: (M @ v.unsqueeze(-1))[..., 0]
        z = back(rhs, con)
        for _ in range(3):
            x, v = z[:, :n], z[:, n:]
            z = z + back(rhs - self.times(P, diag, x) - mul(col, v),
                         con - mul(row, x) - (1.0 - a) * v)
        return z[:, :n], z[:, n:]

    def heads(self, H, rh):
        out = rh.clone()
        out[:, self.junc] = H
        return out

    def steady(self, d, rh, ke, r, speed, h0, pr):
        """The state that satisfies every equation, with the statuses that its
        heads and flows confirm."""
        B = d.shape[0]
        em = (ke > 0)[:, self.junc].to(torch.float64)
        kej, dj, elj = ke[:, self.junc], d[:, self.junc], self.el[self.junc]
        S = torch.full((B, self.L), OPEN, device=DEV)
        S[:, self.prv] = ACTIVE
        q, e = self.q0.expand(B, -1).clone(), em.clone()
        H = torch.zeros(B, self.n, dtype=torch.float64, device=DEV)
        for _ in range(8):                      # statuses
            act = S[:, self.prv] == ACTIVE
            for it in range(60):                # Newton
                hl, hg, he, hge = self.slopes(q, e, r, kej, speed, h0, pr, S)
                P = 1.0 / hg
                P[:, self.prv] = torch.where(act, 0.0, P[:, self.prv])
                Hn = self.heads(H, rh)
                rl = hl - (Hn[:, self.n1] - Hn[:, self.n2])
                re = he - (H - elj)
                bal = self.scatter(-q, q) - em * e - dj
                rhs = bal - self.scatter(-P * rl, P * rl) + em * re / hge
                dH, dqv = self.solve(P, em / hge, rhs, act,
                                     self.hset - H[:, self.jc], False)
                dq = -P * (rl - self.along(dH))
                dq[:, self.prv] = torch.where(act, dqv, dq[:, self.prv])
                H, q, e = H + dH, q + dq, e + em * (dH - re) / hge
                if float((dq.abs().sum(1) / q.abs().sum(1)).max()) < 1e-13 and it > 1:
                    break
            old = S.clone()
            Hn = self.heads(H, rh)   # a pump pushed beyond its shut-off head closes
            beyond = Hn[:, self.n2] - Hn[:, self.n1] > speed * speed * self.hmax + HTOL
            S = torch.where(self.pump, torch.where(beyond, CLOSED, OPEN), S)
            qv, h1 = q[:, self.prv], self.heads(H, rh)[:, self.n1[self.prv]]
            h2, s, hs = self.heads(H, rh)[:, self.n2[self.prv]], S[:, self.prv], self.hset
            back = qv < -QTOL
            new = torch.where(s == ACTIVE,
                              torch.where(back, CLOSED, torch.where(h1 < hs - HTOL, OPEN, ACTIVE)),
                              torch.where(s == OPEN,
                                          torch.where(back, CLOSED,
                                                      torch.where(h2 >= hs + HTOL, ACTIVE, OPEN)),
                                          torch.where((h1 >= hs + HTOL) & (h2 < hs - HTOL), ACTIVE,
                                                      torch.where((h1 < hs - HTOL) & (h1 > h2 + HTOL),
                                                                  OPEN, CLOSED))))
            S[:, self.prv] = new
            if bool((S == old).all()):
                break
        return H, q, e * em, S

    def adjoint(self, state, rh, ke, r, speed, h0, pr, gH, gQ):
        """dL/d(demand, fixed head, Ke, r, speed, h0, pump r), each [B, .]."""
        H, q, e, S = state
        B = H.shape[0]
        em = (ke > 0)[:, self.junc].to(torch.float64)
        kej = ke[:, self.junc]
        act = S[:, self.prv] == ACTIVE
        e1 = torch.where(em > 0, e, torch.ones_like(e))
        _, hg, _, hge = self.slopes(q, e1, r, kej, speed, h0, pr, S)
        P = 1.0 / hg
        P[:, self.prv] = torch.where(act, 0.0, P[:, self.prv])
        rhs = self.scatter(-P * gQ, P * gQ) - gH[:, self.junc]
        lam, _ = self.solve(P, em / hge, rhs, act, -gQ[:, self.prv], True)
        ll = P * (gQ + self.along(lam))
        full = lambda v: torch.zeros(B, self.N, dtype=torch.float64, device=DEV).index_copy(1, self.junc, v)
        with torch.enable_grad():
            th = [_leaf(v.expand(B, self.L).clone()) for v in (r, speed, h0, pr)]
            k_ = _leaf(kej.expand(B, self.n).clone())
            hl = self.loss(q, *th, S)
            gth = torch.autograd.grad(hl, th, -ll)
            gke, = torch.autograd.grad(self.emitter(e1, k_), k_, -(em * lam / hge))
        grh = gH.clone()
        grh = grh.index_add(1, self.n1, ll).index_add(1, self.n2, -ll)
        grh[:, self.junc] = 0.0
        keep = lambda g, m: torch.where(m, g, 0.0)
        return (full(lam), grh, full(gke * em), keep(gth[0], self.pipe),
                *(keep(g, self.pump) for g in gth[1:]))

    def iterate(self, d, rh, ke, r, iterations, accuracy=None):
        """The solver's own iteration, differentiable: fixed statuses, K
        iterations, or until each scenario's relative change is within
        `accuracy`."""
        B = d.shape[0]
        kej, dj, elj = ke[:, self.junc], d[:, self.junc], self.el[self.junc]
        em = (kej > 0).to(torch.float64)
        q, e = self.q0.expand(B, -1), em.clone()
        S = torch.full((B, self.L), OPEN, device=DEV)
        live = torch.ones(B, 1, dtype=torch.bool, device=DEV)
        H = torch.zeros(B, self.n, dtype=torch.float64, device=DEV)
        iters = torch.zeros(B, dtype=torch.int64, device=DEV)
        for _ in range(iterations):
            sgn = torch.where(q < 0, -1.0, 1.0)
            qa = q * sgn
            hg0 = 1.852 * r * qa.clamp_min(1e-30) ** 0.852
            hg = torch.where(hg0 < RQTOL, RQTOL, hg0)
            hl = torch.where(hg0 < RQTOL, RQTOL * qa, hg * qa / 1.852) * sgn
            P, Y = 1.0 / hg, hl / hg
            ea = e.abs().clamp_min(1e-30)
            k = kej.clamp_min(CSMALL)
            he0 = 2.0 * k * ea
            hge = torch.where(he0 < RQTOL, RQTOL, he0)
            he = torch.where(he0 < RQTOL, RQTOL * e, hge * e / 2.0)
            fx = rh.clone()
            fx[:, self.junc] = 0.0
            F = self.scatter(Y - q + P * fx[:, self.n2], q - Y + P * fx[:, self.n1])
            F = F + em * (he + elj) / hge - em * e - dj
            Hn = _Solve.apply(self, P, em / hge, F)
            Hf = fx.index_copy(1, self.junc, Hn)
            dq = Y - P * (Hf[:, self.n1] - Hf[:, self.n2])
            de = em * (he - (Hn - elj)) / hge
            q2, e2 = q - dq, e - de
            if accuracy is None:
                H, q, e = Hn, q2, e2
                continue
            H, q, e = torch.where(live, Hn, H), torch.where(live, q2, q), torch.where(live, e2, e)
            iters = iters + live[:, 0].to(torch.int64)
            ds, qs = dq.abs().sum(1) + de.abs().sum(1), q2.abs().sum(1) + e2.abs().sum(1)
            live = live & (torch.where(qs > accuracy, ds / qs, ds) > accuracy)[:, None]
            if not bool(live.any()):
                break
        return H, q, e * em, iters


def _rows(x, B):
    return (x.unsqueeze(0) if x.dim() == 1 else x).expand(B, -1)


def _emit(m, e):
    return torch.zeros(e.shape[0], m.N, dtype=torch.float64, device=DEV).index_copy(1, m.junc, e)


def _chunks(m, B, copies=1):
    c = max(1, int(1.0e9 // (copies * (m.n + 1) ** 2)))
    return [slice(i, min(B, i + c)) for i in range(0, B, c)]


def _implicit_exact(net, s, B):
    m = _Dense(net)
    out, gr = [], []
    dim1 = lambda k, v: _rows(s.get(k, v), B)
    for c in _chunks(m, B, 2):
        d, rh = s["d"][c], s["rh"][c]
        b = d.shape[0]
        ke, r = dim1("ke", None)[c], dim1("r", None)[c]
        th = [dim1("speed", m.speed)[c], dim1("h0", m.h0)[c], dim1("pr", m.pr)[c]]
        st = m.steady(d, rh, ke, r, *th)
        head = m.heads(st[0], rh)
        gH = torch.zeros_like(head)
        gH[:, s["sens"]] = 2.0 * head[:, s["sens"]]
        gQ = torch.zeros(b, m.L, dtype=torch.float64, device=DEV)
        if s["meters"] is not None:
            gQ[:, s["meters"]] = 2.0 * st[1][:, s["meters"]]
        out.append((head, st[1], _emit(m, st[2])))
        gr.append(m.adjoint(st, rh, ke, r, *th, gH, gQ))
    cat = lambda v: [torch.cat(x) for x in zip(*v)]
    return m, cat(out), cat(gr)


def exact(case, seed):
    """`run`'s results in dense 64-bit torch.  None where that takes too long:
    ensembles whose dense factorisations are too many, and the extended-period
    runs (a dense matrix of 5000 to 20 000 rows per scenario, frame and
    iteration)."""
    kind, B, n = case["kind"], case["batch"], case["junctions"]
    if kind == "eps" or B * float(n) ** 3 > {"unrolled": 3e11, "multi": 8e12}.get(kind, 1.2e12):
        return None
    nets, s = _inputs(case, seed)
    if kind == "multi":
        res = [_implicit_exact(m, dict(d=d, rh=rh, ke=torch.as_tensor(m.node_ke, device=DEV),
                                       r=torch.as_tensor(m.r_hw, device=DEV), meters=None,
                                       sens=torch.as_tensor(_sensors(m), device=DEV)), d.shape[0])
               for m, d, rh in zip(nets, s["d"], s["rh"])]
        return dict(out=[r[1] for r in res],
                    grads=[r[2][0] for r in res] + [r[2][3].sum(0) for r in res])
    if kind in ("implicit", "pumps"):
        m, out, g = _implicit_exact(nets[0], s, B)
        if kind == "implicit":
            return dict(out=out, grads=[g[0], g[1], g[2].sum(0), g[3].sum(0)])
        return dict(out=out, grads=[g[0], g[1], g[3].sum(0), g[4], g[5].sum(0), g[6].sum(0)])
    m = _Dense(nets[0])
    if kind == "steady":
        parts = []
        for c in _chunks(m, B, 2):
            H, q, e, it = m.iterate(s["d"][c], s["rh"][c], _rows(s["ke"], B)[c],
                                    _rows(s["r"], B)[c], 200, case["accuracy"])
            parts.append((m.heads(H, s["rh"][c]), q, _emit(m, e), it))
        head, q, e, it = (torch.cat(x) for x in zip(*parts))
        return dict(head_ft=head, flow_cfs=q, emitter_cfs=e, iters=it)
    if kind == "unrolled":
        outs, gd, grh, gke, gr = [], [], [], 0.0, 0.0
        for c in _chunks(m, B, case["iterations"]):
            x = [_leaf(s["d"][c]), _leaf(s["rh"][c]), _leaf(s["ke"]), _leaf(s["r"])]
            b = x[0].shape[0]
            with torch.enable_grad():
                H, q, e, _ = m.iterate(x[0], x[1], _rows(x[2], b), _rows(x[3], b),
                                       case["iterations"])
                head = x[1].index_copy(1, m.junc, H)
                g = torch.autograd.grad(_loss(s, head, q), x)
            outs.append((head.detach(), q.detach(), _emit(m, e.detach())))
            gd.append(g[0])
            grh.append(g[1])
            gke, gr = gke + g[2], gr + g[3]
        return dict(out=[torch.cat(x) for x in zip(*outs)],
                    grads=[torch.cat(gd), torch.cat(grh), gke, gr])
    sens, rows = s["sens"], []
    ke, r = _rows(s["ke"], B), _rows(s["r"], B)
    th = [_rows(v, B) for v in (m.speed, m.h0, m.pr)]
    st = m.steady(s["d"], s["rh"], ke, r, *th)
    for j in sens.tolist():
        gH = torch.zeros(B, m.N, dtype=torch.float64, device=DEV)
        gH[:, j] = 1.0
        gQ = torch.zeros(B, m.L, dtype=torch.float64, device=DEV)
        rows.append(m.adjoint(st, s["rh"], ke, r, *th, gH, gQ)[3])
    return torch.stack(rows, 1).reshape(B * sens.numel(), m.L).cpu().numpy()
