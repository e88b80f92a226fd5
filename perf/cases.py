"""Performance cases of the batched power-flow engine: what its users run, from a small
interactive contingency list to the 9241-bus N-1 screening, through the public entry
points (PowerFlow, MultiGrid, the particle-swarm shim, the autograd function and the
C-ABI's device-buffer calls).

listed() are the fixed cases, draw() gives more of the same ranges, prepare() makes what
a program holds before the call (the grid's handle, the case definitions), run() is one
pass, work() the bytes and operations a pass cannot do without, and exact() the same
outputs in 64 bits from plain torch (dense Jacobians, branch-wise currents).

The grid of a case is fixed by its sizes and grid_seed, as a program's grid is; the seed
chooses outages, loads, particles and limits.
"""
import math

import numpy as np
import torch

import mapol_b200 as m
from mapol_b200 import pso
from mapol_b200._lib import lib
from mapol_b200.autograd import PowerFlowLoss

ALG = {"NR": m.NR, "FDXB": m.FDXB, "FDBX": m.FDBX}
PREC = {"fp64": m.FP64, "mixed": m.MIXED}


def _tol(case):
    """Convergence tolerance a program asks for: the default, 1e-10 where mixed-precision
    voltages feed later differences, 1e-12 where gradients are taken at the solution."""
    if case["prec"] == "fp64" or case.get("n_bus") == 9241:
        return m.runpf.EPS
    return 1e-12 if case["op"] in ("grad", "adjoint") else 1e-10

# branches, PV buses and tapped share of the repository's configurations
SHAPES = {30: (41, 5, 0.0), 118: (179, 53, 0.10), 300: (411, 69, 0.10), 1354: (1991, 259, 0.10),
          2869: (4582, 509, 0.10), 9241: (16049, 1445, 0.15)}

# outages of the 9241-bus grid after which Newton from the flat start finds no solution or
# wanders first (of 15,584): their voltages at the iteration limit are not a result
NO_SOLUTION = {9241: (5938, 7448, 9668, 15311)}


def listed():
    return [
        # a control-room query: the base case and ten outages of a small grid, host in and out
        dict(name="host_30_fp64", op="host", n_bus=30, n_cases=11, alg="NR", prec="fp64", outages=1, base=True),
        # one swarm evaluation of the optimiser loop (the reference's own use of the engine)
        dict(name="pso_300_mixed", op="pso", n_bus=300, n_cases=1024, alg="NR", prec="mixed"),
        # N-1 with generator reactive limits enforced
        dict(name="qlim_300_mixed", op="qlim", n_bus=300, n_cases=257, alg="NR", prec="mixed", outages=1, base=True),
        # one training step: overload loss of load scenarios and its gradients, through torch
        dict(name="grad_300_mixed", op="grad", n_bus=300, n_cases=500, alg="NR", prec="mixed"),
        # N-1 of three grids of uneven size in one batch
        dict(name="multi_mixed", op="multi", grids="118,1354,2869", cases="167,400,400", alg="NR", prec="mixed"),
        # the headline: N-1 screening of the 9241-bus grid
        dict(name="n1_9241_mixed", op="solve", n_bus=9241, n_cases=1000, alg="NR", prec="mixed", outages=1),
        # N-1 security screening in plain FP64: voltages, then branch flows against the ratings
        dict(name="screen_2869_fp64", op="screen", n_bus=2869, n_cases=600, alg="NR", prec="fp64", outages=1),
        # load scenarios from host memory, voltages back to host memory
        dict(name="scen_1354_mixed", op="host", n_bus=1354, n_cases=1000, alg="NR", prec="mixed", sigma=0.05),
        # solve and adjoint gradients of 4096 load scenarios, in device memory
        dict(name="adjoint_1354_mixed", op="adjoint", n_bus=1354, n_cases=4096, alg="NR", prec="mixed", sigma=0.05),
        # fast-decoupled N-1
        dict(name="fdxb_2869_fp64", op="solve", n_bus=2869, n_cases=400, alg="FDXB", prec="fp64", outages=1),
        # fast-decoupled N-2, a ragged batch
        dict(name="fdbx_1354_mixed", op="solve", n_bus=1354, n_cases=777, alg="FDBX", prec="mixed", outages=2),
        # a densely meshed grid (large fronts in the factorisation)
        dict(name="dense_1354_mixed", op="solve", n_bus=1354, n_cases=250, alg="NR", prec="mixed", outages=1,
             topology=1),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["host", "host", "pso", "qlim", "grad", "multi", "screen", "solve", "solve", "solve", "fd", "fd",
                     "dense", "adjoint"])
    prec = rng.choice(["fp64", "mixed"])
    seed = rng.randint(2, 1000)
    if op == "host":
        n = _log_int(rng, 30, 1500)
        if rng.random() < 0.5:
            c = _log_int(rng, 1, min(2000, 1_300_000 // n))
            return dict(op="host", n_bus=n, n_cases=c, alg="NR", prec=prec, sigma=0.05, grid_seed=seed)
        return dict(op="host", n_bus=n, n_cases=_log_int(rng, 1, min(400, n)), alg="NR", prec=prec, outages=1,
                    base=rng.random() < 0.5, grid_seed=seed)
    if op == "pso":
        return dict(op="pso", n_bus=_log_int(rng, 30, 500), n_cases=_log_int(rng, 16, 1024), alg="NR", prec=prec,
                    grid_seed=seed)
    if op == "qlim":
        n = _log_int(rng, 60, 500)
        return dict(op="qlim", n_bus=n, n_cases=_log_int(rng, 8, min(300, n)), alg="NR", prec=prec, outages=1,
                    base=True, grid_seed=seed)
    if op == "grad":
        return dict(op="grad", n_bus=_log_int(rng, 30, 500), n_cases=_log_int(rng, 8, 500), alg="NR", prec=prec,
                    grid_seed=seed)
    if op == "multi":
        sizes = [_log_int(rng, 60, 1500) for _ in range(rng.randint(2, 4))]
        return dict(op="multi", grids=",".join(map(str, sizes)),
                    cases=",".join(str(_log_int(rng, 5, min(400, s))) for s in sizes), alg="NR", prec=prec,
                    grid_seed=seed)
    if op == "screen":
        n = _log_int(rng, 118, 1500)
        return dict(op="screen", n_bus=n, n_cases=_log_int(rng, 4, min(900, n)), alg="NR", prec=prec, outages=1,
                    grid_seed=seed)
    if op == "fd":
        n = _log_int(rng, 30, 1500)
        return dict(op="solve", n_bus=n, n_cases=_log_int(rng, 1, min(800, n)), alg=rng.choice(["FDXB", "FDBX"]),
                    prec=prec, outages=rng.choice([1, 2]), grid_seed=seed)
    if op == "dense":
        n = _log_int(rng, 300, 1100)
        return dict(op="solve", n_bus=n, n_cases=_log_int(rng, 10, 200), alg="NR", prec="mixed", outages=1,
                    topology=1, grid_seed=seed)
    if op == "adjoint":
        n = _log_int(rng, 118, 1354)
        return dict(op="adjoint", n_bus=n, n_cases=_log_int(rng, 32, 2048), alg="NR", prec=prec, sigma=0.05,
                    grid_seed=seed)
    if rng.random() < 0.2:
        return dict(op="solve", n_bus=2869, n_cases=_log_int(rng, 1, 2000 if prec == "mixed" else 1000), alg="NR",
                    prec=prec, outages=1)
    if rng.random() < 0.3:  # the largest grid, any batch size
        return dict(op="solve", n_bus=9241, n_cases=_log_int(rng, 1, 900 if prec == "mixed" else 400), alg="NR",
                    prec=prec, outages=1)
    n = _log_int(rng, 118, 1500)
    return dict(op="solve", n_bus=n, n_cases=_log_int(rng, 1, n), alg="NR", prec=prec, outages=1, grid_seed=seed)


# ---------------------------------------------------------------- inputs
def _grid(n, seed, topology=0):
    if n in SHAPES:
        nbr, npv, tap = SHAPES[n]
    else:
        nbr, npv, tap = int((1.5 if n < 1000 and topology == 0 else 1.47 if topology else 1.6) * n), max(2, n // 6), 0.10
    return m.synth_grid(n, nbr, npv, tap, seed=seed, topology=topology)


def _outage_cases(branches, nb, n, k, seed, base=False):
    """n outage lists of k branches each (repeating when the grid has fewer non-bridge
    branches); the base case first when asked.  The second outage of a pair is not a
    bridge of what the first one leaves."""
    order = m.select_outages(branches, nb, int((~m.find_bridges(branches, nb)).sum()), seed)
    order = order[~np.isin(order, NO_SOLUTION.get(nb, ()))]
    cases = [[]] if base else []
    for i in range(n - len(cases)):
        a = int(order[i % len(order)])
        if k == 1:
            cases.append([a])
            continue
        rest = branches.copy()
        rest["status"][a] = 0
        bridge = m.find_bridges(rest, nb)
        j = next((int(order[(i + 1 + q) % len(order)]) for q in range(len(order))
                  if int(order[(i + 1 + q) % len(order)]) != a and not bridge[order[(i + 1 + q) % len(order)]]), None)
        cases.append([a] if j is None else [a, j])
    return cases


def _pso_grid(case):
    """The grid with switchable shunts at a tenth of its PQ buses, and its structures."""
    buses, branches = _grid(case["n_bus"], case.get("grid_seed", 1))
    pq = np.where(buses["type"] == 1)[0]
    buses["bsh"][pq[::10]] = 0.05
    return (buses, branches) + pso.estruturas(buses, branches)


def _particles(est, n, seed):
    """A swarm some iterations into a run: positions within 2 % (set-points, taps) and
    0.05 p.u. (shunts) of the defaults, inside the structures' bounds."""
    rng = np.random.default_rng(seed)
    d = np.array([e.default for e in est])
    width = np.array([0.05 if e.tipo == pso.SHC else 0.02 for e in est])
    x = d + width * rng.uniform(-1.0, 1.0, (n, len(est)))
    return np.clip(x, [e.min for e in est], [e.max for e in est])


def _inputs(case, seed):
    """(buses, branches, outage lists, injections or None) of a one-grid case."""
    nb, n = case["n_bus"], case["n_cases"]
    buses, branches = _grid(nb, case.get("grid_seed", 1), case.get("topology", 0))
    if case.get("outages"):
        cases = _outage_cases(branches, nb, n, case["outages"], seed, case.get("base", False))
    else:
        cases = [[] for _ in range(n)]
    sbus = m.load_scenarios(buses, n, case["sigma"], seed) if case.get("sigma") else None
    return buses, branches, cases, sbus


def _limits(case, buses, seed):
    """Reactive limits of every PV bus in p.u.: ranges of a size that some outages exceed."""
    rng = np.random.default_rng(seed)
    hi = np.where(buses["type"] == 2, rng.uniform(0.2, 0.8, len(buses)), np.inf)
    lo = np.where(buses["type"] == 2, -rng.uniform(0.2, 0.8, len(buses)), -np.inf)
    return lo, hi


def _multi_inputs(case, seed):
    sizes = [int(s) for s in case["grids"].split(",")]
    counts = [int(s) for s in case["cases"].split(",")]
    grids, cases = [], []
    for n, c in zip(sizes, counts):
        b, br = _grid(n, case.get("grid_seed", 1))
        grids.append((b, br))
        cases.append(_outage_cases(br, n, c, 1, seed))
    return grids, cases


# ---------------------------------------------------------------- the cases
def _check(pf, rc):
    if rc != 0:
        raise RuntimeError(lib().mpf_last_error(pf._h).decode())


def _result_buffers(n, nb):
    return dict(v=torch.empty((n, nb, 2), dtype=torch.float64, device="cuda"),
                iterations=torch.empty(n, dtype=torch.int32, device="cuda"),
                status=torch.empty(n, dtype=torch.uint8, device="cuda"))


def prepare(case, seed):
    op, alg, prec = case["op"], ALG[case["alg"]], PREC[case["prec"]]
    s = dict(op=op, alg=alg, prec=prec)
    if op == "multi":
        grids, cases = _multi_inputs(case, seed)
        s["mg"] = m.MultiGrid(grids, tol=_tol(case))
        s["mg"].set_cases(cases)
        s["pf"] = s["mg"].pf
        s["out"] = _result_buffers(sum(map(len, cases)), len(s["pf"].buses))
        return s
    if op == "pso":
        buses, branches, est, bie, rie = _pso_grid(case)
        s["est"] = est
        s["swarm"] = [pso.Particula(x) for x in _particles(est, case["n_cases"], seed)]
        s["engine"] = pso.hybrid_init(buses, branches, case["n_cases"], 1, est, alg, bie, rie, precision=prec,
                                      tol=_tol(case))
        return s
    if op == "grad":
        buses, branches = _grid(case["n_bus"], case.get("grid_seed", 1))
        s["pf"] = pf = m.PowerFlow(buses, branches, tol=_tol(case))
        _rate(pf)
        s["cases"] = [[] for _ in range(case["n_cases"])]
        sbus = torch.as_tensor(m.load_scenarios(buses, case["n_cases"], 0.05, seed)).cuda()
        s["p"] = sbus[..., 0].contiguous().requires_grad_()
        s["q"] = sbus[..., 1].contiguous().requires_grad_()
        return s
    buses, branches, cases, sbus = _inputs(case, seed)
    n, nb, nbr = len(cases), len(buses), len(branches)
    s["pf"] = pf = m.PowerFlow(buses, branches, tol=_tol(case))
    if op == "host":
        s["cases"], s["sbus"] = cases, sbus
        return s
    if op in ("screen", "adjoint"):
        _rate(pf)
    if op == "qlim":
        pf.set_q_limits(*_limits(case, buses, seed))
    pf.set_cases(cases, sbus=sbus)
    s["out"] = _result_buffers(n, nb)
    extra = {"screen": dict(ploss=(n,), overload=(n,), sf=(n, nbr, 2), st=(n, nbr, 2)),
             "adjoint": dict(grad_p=(n, nb), grad_q=(n, nb), grad_g=(n, nbr), grad_b=(n, nbr))}.get(op, {})
    s["extra"] = {k: torch.empty(shape, dtype=torch.float64, device="cuda") for k, shape in extra.items()}
    return s


def _rate(pf):
    """Ratings of 1.2 times the base case's flows (the overload loss starts at 0.9 of it)."""
    pf.set_cases([[]])
    pf.solve(m.NR, m.FP64)
    pf.set_ratings(1.2 * np.abs(pf.branch_flows(flows=True)["sf"][0]))


def _results(s, v, iterations, status):
    """A pass's outputs.  Not max_mis, whose value below the tolerance is rounding; and
    the iteration count in FP64 only: a mixed solve may take one more than another
    rounding of the same FP32 factors (tests/parity.py)."""
    out = dict(v=v, status=status)
    if s["prec"] == m.FP64:
        out["iterations"] = iterations
    return out


def run(s):
    op = s["op"]
    if op == "host":
        r = s["pf"].runpf(s["cases"], s["alg"], s["prec"], sbus=s["sbus"])
        return _results(s, r.v, r.iterations, r.status)
    if op == "pso":
        return dict(fitness=pso.hybrid_runpf(s["engine"], s["est"], s["swarm"]))
    if op == "grad":
        s["p"].grad = s["q"].grad = None
        loss = PowerFlowLoss.apply(s["p"], s["q"], s["pf"], s["cases"], s["prec"])
        loss.sum().backward()
        return dict(loss=loss.detach(), grad_p=s["p"].grad, grad_q=s["q"].grad)
    pf, o = s["pf"], s["out"]
    pf.solve(s["alg"], s["prec"])
    _check(pf, lib().mpf_get_results_device(pf._h, o["v"].data_ptr(), o["iterations"].data_ptr(),
                                            o["status"].data_ptr(), None, None))
    e = s.get("extra", {})
    if op == "screen":
        _check(pf, lib().mpf_branch_flows(pf._h, *(e[k].data_ptr() for k in ("ploss", "overload", "sf", "st")), None))
    if op == "adjoint":
        _check(pf, lib().mpf_adjoint(pf._h, s["prec"], *(e[k].data_ptr() for k in ("grad_p", "grad_q", "grad_g",
                                                                                  "grad_b")), None))
    return dict(_results(s, **o), **e)


def work(case):
    """Per Newton iteration a case's LU factors (about 30 values per bus, 400 operations)
    are written and read once: they do not fit on the chip beside the other cases'.  A
    fast-decoupled solve factors two systems a fifth that size once and substitutes in
    each half iteration.  Inputs and outputs once."""
    w = 8 if case["prec"] == "fp64" else 4
    if case["op"] == "multi":
        size = [(int(a), int(b)) for a, b in zip(case["grids"].split(","), case["cases"].split(","))]
    else:
        size = [(case["n_bus"], case["n_cases"])]
    nbytes = flops = 0.0
    for nb, n in size:
        lu, ops = 30.0 * nb * w, 400.0 * nb
        if case.get("topology"):
            lu, ops = lu * 9, ops * 60
        if case["alg"] == "NR":
            its = 5.0
            per, fl = its * (2 * lu + 40 * nb * w), its * (ops + 4 * 30 * nb + 300 * nb)
        else:
            its = 9.0
            per, fl = 2 * lu / 5 + its * 2 * lu / 5, 2 * ops / 5 + its * (4 * 12 * nb + 400 * nb)
        per += 16 * nb + 13 + (16 * nb if case.get("sigma") or case["op"] == "grad" else 0)
        nbr = 1.5 * nb
        if case["op"] == "screen":
            per, fl = per + 32 * nbr, fl + 60 * nbr
        if case["op"] in ("adjoint", "grad"):
            per, fl = per + 2 * lu + 16 * nb + (16 * nbr if case["op"] == "adjoint" else 0), fl + ops + 4 * 30 * nb
        if case["op"] == "qlim":
            per, fl = 2 * per, 2 * fl
        nbytes, flops = nbytes + n * per, flops + n * fl
    return dict(bytes=nbytes, flops=flops)


# ---------------------------------------------------------------- the same in 64 bits, plain torch
class _Net:
    """Branch admittances and bus data as torch float64 / complex128; columns are cases
    ([nb, 1] and [nbr, 1] where all cases share a value)."""

    def __init__(self, buses, branches, cases, sbus=None, dev=None):
        self.dev = dev = dev or ("cuda" if torch.cuda.is_available() else "cpu")
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)  # noqa: E731
        self.nb, self.nbr, self.n = len(buses), len(branches), len(cases)
        self.f = torch.as_tensor(branches["from"].astype(np.int64), device=dev)
        self.t = torch.as_tensor(branches["to"].astype(np.int64), device=dev)
        z = branches["r"] + 1j * branches["x"]
        self.g, self.b = t((1 / z).real)[:, None], t((1 / z).imag)[:, None]
        self.bc = t(branches["b"])[:, None] / 2
        self.tap = t(np.where(branches["tap"] != 0, branches["tap"], 1.0))[:, None]
        self.shift = t(np.deg2rad(branches["shift"]))[:, None]
        self.bsh, self.gsh = t(buses["bsh"])[:, None], t(buses["gsh"])[:, None]
        self.on = torch.ones((self.nbr, self.n), dtype=torch.float64, device=dev)
        self.on *= t(branches["status"].astype(float))[:, None]
        for c, out in enumerate(cases):
            for k in out:
                self.on[k, c] = 0.0
        s = np.stack([buses["p"], buses["q"]], -1)[None] if sbus is None else sbus
        self.p, self.q = t(s[..., 0]).T, t(s[..., 1]).T
        self.vm0, self.va0 = t(buses["vm"])[:, None], t(buses["va"])[:, None]
        typ = torch.as_tensor(buses["type"].astype(np.int64), device=dev)[:, None]
        self.th = (typ == 1) | (typ == 2)  # angle unknown, P equation
        self.mg = typ == 1                 # magnitude unknown, Q equation

    def pick(self, idx):
        """The same net for some of its cases."""
        o = object.__new__(_Net)
        o.__dict__.update(self.__dict__)
        o.n = len(idx)
        for k in ("g", "b", "bc", "tap", "shift", "bsh", "gsh", "on", "p", "q", "vm0", "va0", "th", "mg"):
            a = getattr(self, k)
            setattr(o, k, a[:, idx] if a.shape[1] > 1 else a)
        if self.n == 1:
            o.on = self.on[:, :1]
        return o

    def start(self):
        one = torch.ones((self.nb, self.n), dtype=torch.float64, device=self.dev)
        return self.va0 * one, self.vm0 * one

    def admittances(self, g=None, b=None):
        y = torch.complex(self.g if g is None else g, self.b if b is None else b)
        tap = torch.polar(self.tap * torch.ones_like(self.shift), self.shift * torch.ones_like(self.tap))
        ytt = y + 1j * self.bc
        return ytt / (tap * tap.conj()), -y / tap.conj(), -y / tap, ytt

    def flows(self, V, adm):
        yff, yft, ytf, ytt = adm
        vf, vt = V[self.f], V[self.t]
        sf = vf * (self.on * (yff * vf + yft * vt)).conj()
        st = vt * (self.on * (ytf * vf + ytt * vt)).conj()
        return sf, st

    def power(self, V, adm):
        """Complex power the network takes at every bus."""
        sf, st = self.flows(V, adm)
        s = V * ((self.gsh + 1j * self.bsh) * V).conj()
        return s.index_add(0, self.f, sf).index_add(0, self.t, st)

    def mismatch(self, V, adm):
        s = self.power(V, adm)
        zero = torch.zeros((), dtype=torch.float64, device=self.dev)
        return torch.where(self.th, s.real - self.p, zero), torch.where(self.mg, s.imag - self.q, zero)

    def dense_y(self, adm, c):
        """Dense Ybus [c, nb, nb]."""
        y = torch.zeros((c, self.nb, self.nb), dtype=torch.complex128, device=self.dev)
        yff, yft, ytf, ytt = ((self.on * a).T.expand(c, -1) for a in adm)
        flat = y.view(c, -1)
        for row, col, val in ((self.f, self.f, yff), (self.f, self.t, yft), (self.t, self.f, ytf), (self.t, self.t, ytt)):
            flat.index_add_(1, row * self.nb + col, val)
        torch.diagonal(y, dim1=1, dim2=2).add_(((self.gsh + 1j * self.bsh).T).expand(c, -1))
        return y

    def jacobian(self, va, vm, adm):
        """[c, 2 nb, 2 nb] over (Va, Vm), identity rows and columns where a bus has no unknown."""
        c = va.shape[1]
        y = self.dense_y(adm, c)
        V = torch.polar(vm, va).T
        I = (y @ V[..., None])[..., 0]
        e = V / V.abs()
        dva = -(y * V[:, None, :]).conj_physical_()
        torch.diagonal(dva, dim1=1, dim2=2).add_(I.conj())
        dva = 1j * V[:, :, None] * dva
        dvm = V[:, :, None] * (y * e[:, None, :]).conj_physical_()
        torch.diagonal(dvm, dim1=1, dim2=2).add_(I.conj() * e)
        del y
        J = torch.empty((c, 2 * self.nb, 2 * self.nb), dtype=torch.float64, device=self.dev)
        nb = self.nb
        J[:, :nb, :nb], J[:, :nb, nb:], J[:, nb:, :nb], J[:, nb:, nb:] = dva.real, dvm.real, dva.imag, dvm.imag
        live = torch.cat([self.th.expand(-1, c), self.mg.expand(-1, c)]).T
        J *= live[:, :, None]
        J *= live[:, None, :]
        torch.diagonal(J, dim1=1, dim2=2).add_((~live).double())
        return J

    def newton(self, va, vm, steps=25):
        adm = self.admittances()
        for _ in range(steps):
            P, Q = self.mismatch(torch.polar(vm, va), adm)
            F = torch.cat([P, Q])
            if float(F.abs().max()) < 3e-13:
                break
            d = torch.linalg.solve(self.jacobian(va, vm, adm), F.T[..., None])[..., 0].T
            va, vm = va - d[:self.nb], vm - d[self.nb:]
        return va, vm

    def solve(self, ref):
        """All cases: Newton with the fixed Jacobian of the reference solution ref = (va, vm,
        inverse of its Jacobian), then full Newton for the cases that this leaves unsolved."""
        adm = self.admittances()
        va, vm = self.start()
        va, vm = torch.where(self.th, ref[0], va), torch.where(self.mg, ref[1], vm)
        floor = None
        for k in range(200):
            P, Q = self.mismatch(torch.polar(vm, va), adm)
            F = torch.cat([P, Q])
            worst = F.abs().amax(0)
            if k % 10 == 0:
                now = float(worst.median())
                if float(worst.max()) < 1e-13 or (floor is not None and now > 0.5 * floor and now < 1e-11):
                    break
                floor = now
            d = ref[2] @ F
            va, vm = va - d[:self.nb], vm - d[self.nb:]
        P, Q = self.mismatch(torch.polar(vm, va), adm)
        bad = torch.nonzero(~(torch.cat([P, Q]).abs().amax(0) < 1e-11)).flatten().tolist()
        if len(bad) * self.nb ** 2 > 2e9:
            return None
        for c in bad:
            one = self.pick([c])
            a, b = one.newton(*(x[:, :1] for x in one.start()))
            va[:, c:c + 1], vm[:, c:c + 1] = a, b
        return va, vm


def _reference(buses, branches):
    """Base solution and the inverse of its Jacobian."""
    net = _Net(buses, branches, [[]])
    va, vm = net.newton(*net.start())
    return va, vm, torch.linalg.inv(net.jacobian(va, vm, net.admittances())[0])


def _rows(a):
    return torch.view_as_real(a.T.contiguous().resolve_conj()) if a.is_complex() else a.T.contiguous()


def _out(va, vm):
    return dict(v=_rows(torch.polar(vm, va)))


def _adjoint_exact(net, ref, va, vm, rating):
    """Gradients of the overload loss: J^T lambda = dL/dx by refinement with the base
    Jacobian's inverse, J^T lambda and the explicit parts by automatic differentiation."""
    xa, xm = va.detach().requires_grad_(), vm.detach().requires_grad_()
    g = (net.g * torch.ones_like(net.on)).requires_grad_()
    b = (net.b * torch.ones_like(net.on)).requires_grad_()
    adm = net.admittances(g, b)
    V = torch.polar(xm, xa)
    loss = ((net.flows(V, adm)[0].abs() - 0.9 * rating).clamp_min(0.0) ** 2).sum(0)
    P, Q = net.mismatch(V, adm)
    F = torch.cat([P, Q])
    live = torch.cat([net.th.expand(-1, net.n), net.mg.expand(-1, net.n)])
    ga, gm, gg, gb = torch.autograd.grad(loss.sum(), (xa, xm, g, b), retain_graph=True)
    dx = torch.cat([ga, gm]) * live
    lam = torch.zeros_like(dx)
    for _ in range(40):
        ja, jm = torch.autograd.grad(F, (xa, xm), lam, retain_graph=True)
        r = dx - torch.cat([ja, jm]) * live
        if float(r.abs().max()) <= 1e-15 * float(dx.abs().max()):
            break
        lam = lam + ref[2].T @ r
    lam = lam * live
    lg, lb = torch.autograd.grad(F, (g, b), lam)
    return dict(loss=loss.detach(), grad_p=_rows(lam[:net.nb]), grad_q=_rows(lam[net.nb:]), grad_g=_rows(gg - lg),
                grad_b=_rows(gb - lb))


def exact(case, seed):
    big = case["n_bus"] if case["op"] != "multi" else max(int(s) for s in case["grids"].split(","))
    if not torch.cuda.is_available() and big > 400:
        return None  # dense 64-bit factors of the larger grids take minutes on a host
    op = case["op"]
    if op == "multi":
        grids, cases = _multi_inputs(case, seed)
        off = np.cumsum([0] + [len(b) for b, _ in grids])
        v0 = torch.cat([torch.polar(*_Net(b, br, [[]]).start()[::-1]) for b, br in grids])
        v = torch.view_as_real(v0.T.contiguous()).repeat(sum(map(len, cases)), 1, 1)
        row = 0
        for k, (b, br) in enumerate(grids):
            got = _Net(b, br, cases[k]).solve(_reference(b, br))
            if got is None:
                return None
            v[row:row + len(cases[k]), off[k]:off[k + 1]] = _out(*got)["v"]
            row += len(cases[k])
        return dict(v=v)
    if op == "pso":
        buses, branches, est, bie, rie = _pso_grid(case)
        x = torch.as_tensor(_particles(est, case["n_cases"], seed))
        net = _Net(buses, branches, [[]] * case["n_cases"])
        x = x.to(net.dev)
        one = torch.ones((1, case["n_cases"]), dtype=torch.float64, device=net.dev)
        net.tap, net.bsh, net.vm0 = net.tap * one, net.bsh * one, net.vm0 * one
        for i in np.where(bie >= 0)[0]:
            (net.vm0 if est[bie[i]].tipo == pso.AVR else net.bsh)[i] = x[:, bie[i]]
        for k in np.where(rie >= 0)[0]:
            net.tap[k] = x[:, rie[k]]
        loss = []
        for c in range(0, net.n, 128):
            part = net.pick(list(range(c, min(net.n, c + 128))))
            va, vm = part.newton(*part.start())
            sf, st = part.flows(torch.polar(vm, va), part.admittances())
            loss.append((sf + st).real.sum(0))
        return dict(fitness=torch.cat(loss))
    if op == "grad":
        buses, branches = _grid(case["n_bus"], case.get("grid_seed", 1))
        cases, sbus = [[]] * case["n_cases"], m.load_scenarios(buses, case["n_cases"], 0.05, seed)
    else:
        buses, branches, cases, sbus = _inputs(case, seed)
    net = _Net(buses, branches, cases, sbus)
    if op == "qlim":
        lo, hi = (torch.as_tensor(a, device=net.dev)[:, None] for a in _limits(case, buses, seed))
        one = torch.ones((1, net.n), dtype=torch.float64, device=net.dev)
        net.q, net.mg = net.q * one, net.mg & (one > 0)
        va, vm = net.start()
        pv = net.th & ~net.mg
        for _ in range(20):
            parts = [net.pick(list(range(c, min(net.n, c + 64)))) for c in range(0, net.n, 64)]
            done = [p.newton(va[:, 64 * i:64 * i + p.n], vm[:, 64 * i:64 * i + p.n]) for i, p in enumerate(parts)]
            va, vm = torch.cat([d[0] for d in done], 1), torch.cat([d[1] for d in done], 1)
            q = net.power(torch.polar(vm, va), net.admittances()).imag
            over, under = pv & (q > hi), pv & (q < lo)
            if not bool((over | under).any()):
                break
            net.q = torch.where(over, hi, torch.where(under, lo, net.q))
            net.mg, pv = net.mg | over | under, pv & ~(over | under)
        return _out(va, vm)
    ref = _reference(buses, branches)
    got = net.solve(ref)
    if got is None:
        return None
    out = _out(*got)
    if op in ("screen", "adjoint", "grad"):
        base = _Net(buses, branches, [[]])
        rating = 1.2 * base.flows(torch.polar(ref[1], ref[0]), base.admittances())[0].abs()
    if op == "screen":
        sf, st = net.flows(torch.polar(got[1], got[0]), net.admittances())
        over = ((sf.abs() - 0.9 * rating).clamp_min(0.0) ** 2).sum(0)
        out.update(ploss=(sf + st).real.sum(0), overload=over, sf=_rows(sf), st=_rows(st))
    if op in ("adjoint", "grad"):
        a = _adjoint_exact(net, ref, *got, rating)
        if op == "grad":
            return dict(loss=a["loss"], grad_p=a["grad_p"], grad_q=a["grad_q"])
        a.pop("loss")
        out.update(a)
    if op == "host":
        v = out["v"].cpu().numpy()
        out["v"] = v[..., 0] + 1j * v[..., 1]
    return out
