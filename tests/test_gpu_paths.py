"""The two forms of a solve, level launches and one block per chunk of lanes: each against the
oracle where the other one is the rule's choice, and the rule at sizes where the choice was
measured to matter.  mpf_timing.launches tells them apart: a chunk solve is a few launches."""
import numpy as np
import pytest

import mapol_b200 as m
from oracle import oracle

pytestmark = pytest.mark.gpu


def grid(n_bus, topology=0):
    return m.synth_grid(n_bus, int(1.4 * n_bus), max(2, n_bus // 6), 0.1, seed=4, topology=topology)


def outages(branches, n_bus, n_cases):
    n1 = np.flatnonzero(~m.find_bridges(branches, n_bus))
    return ([[]] + [[int(b)] for b in np.resize(n1, n_cases)])[:n_cases]


@pytest.mark.parametrize("prec", [m.FP64, m.MIXED])
@pytest.mark.parametrize("alg", [m.FDXB, m.FDBX])
@pytest.mark.parametrize("n_bus,n_cases,topology", [(30, 1, 0), (118, 33, 0), (300, 70, 0), (300, 20, 1)])
def test_fast_decoupled_level_launches_match_oracle(gpu, monkeypatch, prec, alg, n_bus, n_cases, topology):
    """Tolerance: both sides stop at max |F| < 1e-10, so |dV| stays below the parity tests' 1e-8."""
    buses, branches = grid(n_bus, topology)
    cases = outages(branches, n_bus, n_cases)
    ref = oracle.runpf(buses, branches, cases, alg=alg, tol=1e-10)
    launches = []
    for chunk in ("0", "1"):
        monkeypatch.setenv("MPF_FD_CHUNK", chunk)
        with m.PowerFlow(buses, branches, tol=1e-10) as pf:
            res = pf.runpf(cases, alg=alg, precision=prec)
            launches.append(pf.timing()["launches"])
        assert np.array_equal(res.converged, ref["converged"]) and res.converged.all()
        assert np.abs(res.v - ref["v"]).max() < 1e-8
        if prec == m.FP64:
            assert np.array_equal(res.iterations, ref["iterations"])
    assert launches[0] > launches[1] + 50


def test_fast_decoupled_level_launches_on_several_grids_with_controls(gpu, monkeypatch):
    """Islands and per-case controls through the level launches and through the chunks: the same
    iterations, and voltages as close as two runs to max |F| < 1e-10 are (1e-8 as above)."""
    grids = [grid(30), grid(118)]
    out = []
    for chunk in ("0", "1"):
        monkeypatch.setenv("MPF_FD_CHUNK", chunk)
        with m.MultiGrid(grids, tol=1e-10) as mg:
            mg.set_cases([outages(grids[0][1], 30, 40), outages(grids[1][1], 118, 5)])
            pv = int(np.flatnonzero(mg.pf.buses["type"] == 2)[0])
            pq = int(np.flatnonzero(mg.pf.buses["type"] == 1)[-1])
            vals = np.stack([np.linspace(1.0, 1.03, 45), np.linspace(0.0, 0.1, 45)], -1)
            mg.pf.set_controls([(m.CTRL_AVR, pv), (m.CTRL_SHC, pq)], vals)
            mg.solve(m.FDXB, m.FP64)
            out.append(mg.results())
    for a, b in zip(*out):
        assert a.converged.all() and np.array_equal(a.iterations, b.iterations)
        assert np.abs(a.v - b.v).max() < 1e-8


@pytest.mark.parametrize("prec,n_bus,n_cases,chunks", [(m.FP64, 30, 2500, True), (m.FP64, 30, 20000, False),
                                                       (m.MIXED, 30, 40000, False), (m.FP64, 300, 2000, True),
                                                       (m.FP64, 300, 16000, False), (m.FP64, 11, 2000, True),
                                                       (m.FP64, 11, 16000, False)])
def test_fast_decoupled_form_by_batch(gpu, prec, n_bus, n_cases, chunks):
    """A factor of two or more from the line on either side."""
    buses, branches = grid(n_bus)
    with m.PowerFlow(buses, branches) as pf:
        res = pf.runpf(outages(branches, n_bus, n_cases), alg=m.FDXB, precision=prec)
        assert res.converged.all()
        assert (pf.timing()["launches"] < 50) == chunks


def lanes_that_run(n_bus, prec, lanes):
    """Lanes per block a forced count gives: 0 (level launches) beyond 32 bytes of lanes, and where
    the vectors, contribution blocks and fronts of that many lanes do not fit shared memory."""
    if prec == m.FP64 and lanes == 8:
        return 0
    if n_bus == 700 and lanes == (4 if prec == m.FP64 else 8):
        return 0
    return lanes


@pytest.mark.parametrize("lanes", [1, 2, 4, 8])
@pytest.mark.parametrize("prec", [m.FP64, m.MIXED])
@pytest.mark.parametrize("n_bus,n_cases", [(30, 1), (118, 33), (300, 70), (700, 9)])
def test_forced_newton_lanes_are_the_ones_that_run(gpu, monkeypatch, lanes, prec, n_bus, n_cases):
    """Tolerance: both sides stop at max |F| < 1e-11, so |dV| stays below the parity tests' 1e-8."""
    monkeypatch.setenv("MPF_NR_CHUNK", str(lanes))
    buses, branches = m.synth_grid(n_bus, int(1.5 * n_bus), max(2, n_bus // 6), 0.1, seed=4)
    cases = outages(branches, n_bus, n_cases)
    ref = oracle.runpf(buses, branches, cases, alg=m.NR, tol=1e-11)
    with m.PowerFlow(buses, branches, tol=1e-11) as pf:
        res = pf.runpf(cases, alg=m.NR, precision=prec)
        st = pf.stats()
    assert st["solve_lanes"] == lanes_that_run(n_bus, prec, lanes)
    assert st["solve_in_shared"] == (st["solve_lanes"] > 0)
    assert res.converged.all() and np.abs(res.v - ref["v"]).max() < 1e-8


@pytest.mark.parametrize("in_shared", [True, False])
@pytest.mark.parametrize("prec,lanes", [(m.FP64, 1), (m.FP64, 2), (m.FP64, 4), (m.MIXED, 1), (m.MIXED, 2),
                                        (m.MIXED, 4), (m.MIXED, 8)])
def test_forced_fast_decoupled_lanes_are_the_ones_that_run(gpu, monkeypatch, in_shared, prec, lanes):
    monkeypatch.setenv("MPF_CHUNK_LANES", str(lanes))
    if not in_shared:
        monkeypatch.setenv("MPF_CHUNK_GLOBAL", "1")
    for n_bus, n_cases in ((30, 1), (118, 33), (300, 70)):
        buses, branches = grid(n_bus)
        with m.PowerFlow(buses, branches) as pf:
            assert pf.runpf(outages(branches, n_bus, n_cases), alg=m.FDXB, precision=prec).converged.all()
            st = pf.stats()
        assert (st["solve_lanes"], st["solve_in_shared"]) == (lanes, in_shared)


# 160 cases of 8 lanes are 20 blocks, of 1 lane 160: one block per SM, or two with half of its
# shared memory each.  The 900-bus uniform grid has supernodes larger than a ring slot, which are
# read in place.
@pytest.mark.parametrize("in_shared", [True, False])
@pytest.mark.parametrize("prec,lanes", [(m.FP64, 1), (m.FP64, 2), (m.FP64, 4), (m.MIXED, 1), (m.MIXED, 2),
                                        (m.MIXED, 4), (m.MIXED, 8)])
@pytest.mark.parametrize("n_bus,n_cases,topology", [(30, 5, 0), (300, 160, 0), (900, 6, 1)])
def test_adjoint_chunks_match_level_launches(gpu, monkeypatch, n_bus, n_cases, topology, prec, lanes, in_shared):
    """Same factors, other order of the substitutions' sums: a backward error of about n 2^-53,
    times a condition number of up to 1e5 here 1e-8 of the largest gradient.  (Mixed: both forms
    are refined twice against the FP64 Jacobian, which leaves 1e-12.)"""
    buses, branches = m.synth_grid(n_bus, int(1.45 * n_bus), n_bus // 5, 0.1, seed=5, topology=topology)
    cases = outages(branches, n_bus, n_cases)
    with m.PowerFlow(buses, branches, tol=1e-11) as pf:
        pf.set_cases(cases)
        pf.solve(m.NR, prec)
        assert (pf.status() == m.runpf.CONVERGED).all()
        pf.set_ratings(0.8 * np.abs(pf.branch_flows(flows=True)["sf"][0]))
        monkeypatch.setenv("MPF_SUBST_CHUNK", "0")
        ref = pf.adjoint(prec)
        assert pf.stats()["adjoint_lanes"] == 0
        monkeypatch.delenv("MPF_SUBST_CHUNK")
        monkeypatch.setenv("MPF_CHUNK_LANES", str(lanes))
        if not in_shared:
            monkeypatch.setenv("MPF_CHUNK_GLOBAL", "1")
        got = pf.adjoint(prec)
        st = pf.stats()
    assert (st["adjoint_lanes"], st["adjoint_in_shared"]) == (lanes, in_shared)
    for k in ref:
        assert np.abs(ref[k]).max() > 0.0
        assert np.abs(got[k] - ref[k]).max() < 1e-8 * np.abs(ref[k]).max(), k


@pytest.mark.parametrize("prec,n_bus,n_cases,chunks", [(m.FP64, 30, 1000, True), (m.FP64, 30, 20000, False),
                                                       (m.MIXED, 30, 2500, True), (m.MIXED, 30, 60000, False),
                                                       (m.FP64, 300, 500, True), (m.FP64, 300, 12000, False)])
def test_adjoint_form_by_batch(gpu, prec, n_bus, n_cases, chunks):
    """A factor of two or more from the line on either side."""
    buses, branches = grid(n_bus)
    with m.PowerFlow(buses, branches) as pf:
        pf.set_cases(outages(branches, n_bus, n_cases))
        pf.solve(m.NR, prec)
        pf.set_ratings(np.full(len(branches), 0.2))
        pf.adjoint(prec)
        assert (pf.stats()["adjoint_lanes"] > 0) == chunks


def test_device_bytes_count_the_plans(gpu, monkeypatch):
    """The same batch on level launches and on chunks: the chunks' plans and row lists are device
    memory of the handle, at least one index per entry of the grid's Ybus diagonal."""
    buses, branches = grid(300)
    cases = outages(branches, 300, 64)
    held = {}
    for alg, env in ((m.NR, "MPF_NR_CHUNK"), (m.FDXB, "MPF_FD_CHUNK")):
        for on in ("0", "1"):
            monkeypatch.setenv(env, on)
            with m.PowerFlow(buses, branches) as pf:
                assert pf.runpf(cases, alg=alg).converged.all()
                assert (pf.stats()["solve_lanes"] > 0) == (on == "1")
                held[alg, on] = pf.stats()["device_bytes"]
        monkeypatch.delenv(env)
        assert held[alg, "1"] > held[alg, "0"] + 4 * 300


@pytest.mark.parametrize("use_graph", [2, 1, 0])
@pytest.mark.parametrize("chunk", ["0", "1"])
def test_fast_decoupled_times_by_family(gpu, monkeypatch, chunk, use_graph):
    """Either form reports what mismatches, substitutions and updates took, and no more than the
    solve."""
    monkeypatch.setenv("MPF_FD_CHUNK", chunk)
    buses, branches = grid(300)
    with m.PowerFlow(buses, branches, use_graph=use_graph) as pf:
        for _ in range(2):
            assert pf.runpf(outages(branches, 300, 64), alg=m.FDXB).converged.all()
        t = pf.timing()
        assert (pf.stats()["solve_lanes"] > 0) == (chunk == "1")
    parts = [t[k] for k in ("mismatch_ms", "solve_ms", "update_ms", "jacobian_ms", "factor_ms")]
    assert min(parts) > 0.0 and sum(parts) + t["other_ms"] <= 1.001 * t["total_ms"]
    assert t["solve_ms"] > t["update_ms"]


@pytest.mark.parametrize("prec,n_bus,n_cases,chunks", [(m.FP64, 1600, 5, False), (m.MIXED, 1600, 5, True),
                                                       (m.FP64, 300, 64, True), (m.FP64, 300, 8000, False)])
def test_newton_form_with_reactive_limits(gpu, prec, n_bus, n_cases, chunks):
    """A block's LU above 300,000 bytes, or a batch of many waves, keeps the level launches."""
    buses, branches = m.synth_grid(n_bus, int(1.5 * n_bus), n_bus // 5, 0.1, seed=3)
    with m.PowerFlow(buses, branches) as pf:
        pf.set_q_limits(np.full(n_bus, -0.3), np.full(n_bus, 0.3))
        pf.set_cases(outages(branches, n_bus, n_cases))
        pf.solve(m.NR, prec)
        st = pf.stats()
        assert (st["solve_lanes"] > 0) == chunks
        if n_bus == 1600:
            assert 8 * st["nnz_lu"] > 300000 > 4 * st["nnz_lu"]
