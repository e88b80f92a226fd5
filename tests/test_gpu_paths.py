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
                                                       (m.FP64, 300, 16000, False)])
def test_fast_decoupled_form_by_batch(gpu, prec, n_bus, n_cases, chunks):
    """A factor of two or more from the line on either side."""
    buses, branches = grid(n_bus)
    with m.PowerFlow(buses, branches) as pf:
        res = pf.runpf(outages(branches, n_bus, n_cases), alg=m.FDXB, precision=prec)
        assert res.converged.all()
        assert (pf.timing()["launches"] < 50) == chunks
