"""Kernels that keep a chunk of lanes on one block for a whole solve (kernels_chunk.cuh):
their plan on the CPU, and on the GPU every lane count against the oracle at the sizes
where a team, a chunk or a segment ends; the two large-front kernels against each other;
and the mismatch pass where its staged rows run out of room."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import mapol_b200 as m
from oracle import oracle

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_plans_cover_every_supernode_once(built, tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    exe = str(tmp_path / "chunk_plan_check")
    csrc = os.path.join(ROOT, "mapol_b200", "csrc")
    subprocess.run([cxx, "-O2", "-std=c++17", "-I" + os.path.join(ROOT, "include"), "-I" + csrc, "-o", exe,
                    os.path.join(ROOT, "tests", "native", "chunk_plan_check.cpp"), os.path.join(csrc, "symbolic.cpp"),
                    os.path.join(csrc, "synth.cpp")], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    assert int(out.stdout.split()[1]) > 400


@pytest.mark.gpu
@pytest.mark.parametrize("in_shared", [True, False])
@pytest.mark.parametrize("lanes", [1, 2, 4, 8])
@pytest.mark.parametrize("prec", [m.FP64, m.MIXED])
@pytest.mark.parametrize("n_bus,n_cases,topology", [(30, 1, 0), (118, 33, 0), (300, 70, 0), (300, 20, 1)])
def test_fast_decoupled_chunks_match_oracle(gpu, monkeypatch, in_shared, lanes, prec, n_bus, n_cases, topology):
    """Tolerance: both sides stop at max |F| < 1e-10; |dV| <= |J^-1| 1e-10 stays below the
    1e-8 bar of the parity tests."""
    monkeypatch.setenv("MPF_CHUNK_LANES", str(lanes))
    if not in_shared:
        monkeypatch.setenv("MPF_CHUNK_GLOBAL", "1")
    buses, branches = m.synth_grid(n_bus, int(1.4 * n_bus), max(2, n_bus // 6), 0.1, seed=4, topology=topology)
    n1 = np.flatnonzero(~m.find_bridges(branches, n_bus))
    cases = ([[]] + [[int(b)] for b in np.resize(n1, n_cases)])[:n_cases]
    for alg in (m.FDXB, m.FDBX):
        ref = oracle.runpf(buses, branches, cases, alg=alg, tol=1e-10)
        with m.PowerFlow(buses, branches, tol=1e-10) as pf:
            res = pf.runpf(cases, alg=alg, precision=prec)
        assert np.array_equal(res.converged, ref["converged"]) and res.converged.all()
        assert np.abs(res.v - ref["v"]).max() < 1e-8
        if prec == m.FP64:
            assert np.array_equal(res.iterations, ref["iterations"])


@pytest.mark.gpu
@pytest.mark.parametrize("lanes", [1, 2, 4, 8])
@pytest.mark.parametrize("prec", [m.FP64, m.MIXED])
@pytest.mark.parametrize("n_bus,n_cases", [(30, 1), (118, 33), (300, 70), (700, 9)])
def test_newton_chunks_match_oracle(gpu, monkeypatch, lanes, prec, n_bus, n_cases):
    """Newton on one block per chunk against the oracle (both to max |F| < 1e-11, so |dV|
    stays below the parity tests' 1e-8), and in parts (use_graph 1 and 0) bit for bit."""
    monkeypatch.setenv("MPF_NR_CHUNK", str(lanes))
    buses, branches = m.synth_grid(n_bus, int(1.5 * n_bus), max(2, n_bus // 6), 0.1, seed=4)
    n1 = np.flatnonzero(~m.find_bridges(branches, n_bus))
    cases = ([[]] + [[int(b)] for b in np.resize(n1, n_cases)])[:n_cases]
    ref = oracle.runpf(buses, branches, cases, alg=m.NR, tol=1e-11)
    out = []
    for use_graph in (2, 1, 0):
        with m.PowerFlow(buses, branches, tol=1e-11, use_graph=use_graph) as pf:
            out.append(pf.runpf(cases, alg=m.NR, precision=prec))
    assert out[0].converged.all() and ref["converged"].all()
    assert np.abs(out[0].v - ref["v"]).max() < 1e-8
    if prec == m.FP64:
        assert np.array_equal(out[0].iterations, ref["iterations"])
    for r in out[1:]:
        assert np.array_equal(r.v, out[0].v) and np.array_equal(r.iterations, out[0].iterations)
        assert np.array_equal(r.status, out[0].status) and np.array_equal(r.max_mis, out[0].max_mis)


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [m.FP64, m.MIXED])
@pytest.mark.parametrize("n_bus,n_cases", [(900, 3), (1354, 35)])
def test_large_front_kernels_agree(gpu, monkeypatch, prec, n_bus, n_cases):
    """Trailing block in shared-memory slabs (kind 6) or in global memory (7): the same
    panels, contribution blocks stored by lane pairs in either, bit for bit; against the
    oracle at the parity tests' bar (both to max |F| < 1e-11)."""
    buses, branches = m.synth_grid(n_bus, int(1.47 * n_bus), n_bus // 5, 0.1, seed=5, topology=1)
    n1 = np.flatnonzero(~m.find_bridges(branches, n_bus))
    cases = [[]] + [[int(b)] for b in n1[:n_cases - 1]]
    ref = oracle.runpf(buses, branches, cases[:4], alg=m.NR, tol=1e-11)
    out = []
    for kind in ("6", "7"):
        monkeypatch.setenv("MPF_FACTOR_KIND", kind)
        with m.PowerFlow(buses, branches, tol=1e-11) as pf:
            out.append(pf.runpf(cases, alg=m.NR, precision=prec))
    assert out[0].converged.all()
    assert np.array_equal(out[0].v, out[1].v) and np.array_equal(out[0].iterations, out[1].iterations)
    assert np.abs(out[0].v[:len(ref["v"])] - ref["v"]).max() < 1e-8


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [m.FP64, m.MIXED])
@pytest.mark.parametrize("n_bus,per_bus", [(64, 1.5), (65, 3.2), (130, 6.0)])
def test_mismatch_rows_beyond_the_staged(gpu, prec, n_bus, per_bus):
    """64 rows of fewer than 7 Ybus entries are staged, denser blocks only in part; one row
    more than a block.  autotune=0: the row kernel runs, not the whole-solve one.  Same bar
    as the parity tests (both to max |F| < 1e-11)."""
    buses, branches = m.synth_grid(n_bus, int(per_bus * n_bus), n_bus // 5, 0.1, seed=7, topology=1)
    n1 = np.flatnonzero(~m.find_bridges(branches, n_bus))
    cases = [[]] + [[int(b)] for b in n1[:5]] + [[int(n1[5]), int(n1[7])]]
    ref = oracle.runpf(buses, branches, cases, alg=m.NR, tol=1e-11)
    with m.PowerFlow(buses, branches, tol=1e-11, autotune=0) as pf:
        res = pf.runpf(cases, alg=m.NR, precision=prec)
    assert res.converged.all() and ref["converged"].all()
    assert np.abs(res.v - ref["v"]).max() < 1e-8
