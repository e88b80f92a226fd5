"""Batches at the edges of what the entry points accept."""
import numpy as np
import pytest

import mapol_b200 as m
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [m.FP64, m.MIXED])
@pytest.mark.parametrize("alg", [m.FDXB, m.FDBX, m.NR])
@pytest.mark.parametrize("order", [(0, 1, 2), (1, 2, 0), (1, 2)])
def test_multigrid_with_grids_of_pv_buses_only(gpu, order, alg, prec):
    """A grid whose buses are all PV (but the slack) has no variable in B''.  Tolerance: both
    sides stop at max |F| < 1e-10, so |dV| stays below the parity tests' 1e-8."""
    grids = [m.synth_grid(30, 41, 5, seed=2), m.synth_grid(9, 11, 8, seed=3), m.synth_grid(2, 1, 1, seed=3)]
    grids = [grids[k] for k in order]
    cases = [[[]] * (3 + 33 * k) for k in range(len(grids))]
    with m.MultiGrid(grids, tol=1e-10) as mg:
        mg.set_cases(cases)
        mg.solve(alg, prec)
        out = mg.results()
    for (buses, branches), c, res in zip(grids, cases, out):
        ref = oracle.runpf(buses, branches, c[:1], alg=alg, tol=1e-10)
        assert res.converged.all() and ref["converged"].all()
        assert np.abs(res.v - ref["v"][0]).max() < 1e-8
        if prec == m.FP64:
            assert (res.iterations == ref["iterations"][0]).all()


def test_multigrid_injections_follow_the_new_lane_map(gpu):
    """Batches of another split between the grids, one after the other on one handle: every
    batch's injections reach its own lanes.  Tolerance as above."""
    grids = [m.synth_grid(30, 41, 5, seed=2), m.synth_grid(118, 179, 53, 0.1, seed=3)]
    rng = np.random.default_rng(5)
    with m.MultiGrid(grids, tol=1e-10) as mg:
        for counts in ((70, 3), (3, 70), (1, 200), (200, 1), (33, 33)):
            sbus = [np.stack([b["p"], b["q"]], -1)[None] * rng.uniform(0.8, 1.1, (n, len(b), 1))
                    for (b, _), n in zip(grids, counts)]
            mg.set_cases([[[]] * n for n in counts], sbus)
            mg.solve(m.NR, m.FP64)
            for (buses, branches), s, res in zip(grids, sbus, mg.results()):
                with m.PowerFlow(buses, branches, tol=1e-10) as pf:
                    ref = pf.runpf([[]] * len(s), sbus=s)
                assert res.converged.all() and ref.converged.all()
                assert np.abs(res.v - ref.v).max() < 1e-8


def test_batches_of_more_groups_than_a_grid_has_rows(gpu):
    """65537 groups of 32 cases: too many to solve in one batch, but injections and controls are
    accepted and mpf_mismatch evaluates them.  A two-bus line against its formula; both are a
    handful of FP64 operations on values of order 10, so 1e-12 is 100 roundings."""
    import torch

    from mapol_b200._lib import lib

    n = 65536 * 32 + 1
    buses, branches = m.synth_grid(2, 1, 0, seed=3)
    slack = int(np.flatnonzero(buses["type"] == 3)[0])
    k = 1 - slack
    rng = np.random.default_rng(1)
    sbus = rng.uniform(-1.0, 1.0, (n, 2, 2))
    shunt = rng.uniform(0.0, 0.5, n)
    volts = rng.uniform(0.9, 1.1, (n, 2)) * np.exp(1j * rng.uniform(-0.3, 0.3, (n, 2)))
    b = branches[0]
    assert b["tap"] == 0.0 and b["shift"] == 0.0
    ys = 1.0 / (b["r"] + 1j * b["x"])
    vk, vs = volts[:, k], volts[:, slack]
    v = torch.from_numpy(np.ascontiguousarray(np.stack([volts.real, volts.imag], -1))).cuda()
    out = torch.zeros(n, dtype=torch.float64, device="cuda")
    with m.PowerFlow(buses, branches) as pf:
        pf.set_cases([[]] * n, sbus=sbus)
        for controls in (False, True):
            if controls:
                pf.set_controls([(m.CTRL_SHC, k)], shunt[:, None])
            yd = ys + 0.5j * b["b"] + buses["gsh"][k] + 1j * (shunt if controls else buses["bsh"][k])
            f = vk * np.conj(yd * vk - ys * vs) - (sbus[:, k, 0] + 1j * sbus[:, k, 1])
            ref = np.maximum(np.abs(f.real), np.abs(f.imag))
            assert lib().mpf_mismatch(pf._h, v.data_ptr(), out.data_ptr(), None) == 0
            torch.cuda.synchronize()
            assert np.abs(out.cpu().numpy() - ref).max() < 1e-12 * max(1.0, np.abs(ys) * 10)


def test_injections_laid_out_on_the_host_and_on_the_device(gpu):
    """Few injections are laid out on the host, more on the device: the same mismatches of the same
    cases, bit for bit, alone and as the first of a larger batch, and both refuse a value that is
    not finite and keep the batch they had."""
    import torch

    from mapol_b200._lib import lib

    buses, branches = m.synth_grid(300, 411, 69, 0.1, seed=2)
    rng = np.random.default_rng(3)
    n_small, n_large = 33, 400  # two groups: 19200 with padding lanes; the host takes 16384
    sbus = np.stack([buses["p"], buses["q"]], -1)[None] * rng.uniform(0.5, 1.5, (n_large, 300, 2))
    flat = np.stack([buses["vm"], np.zeros(300)], -1)
    with m.PowerFlow(buses, branches) as pf:

        def mismatch(n):
            v = torch.from_numpy(np.repeat(flat[None], n, 0)).cuda()
            out = torch.zeros(n, dtype=torch.float64, device="cuda")
            assert lib().mpf_mismatch(pf._h, v.data_ptr(), out.data_ptr(), None) == 0
            torch.cuda.synchronize()
            return out.cpu().numpy()

        pf.set_cases([[]] * n_large, sbus=sbus)
        large = mismatch(n_large)
        for n in (1, 27, 32, n_small, n_large):
            pf.set_cases([[]] * n, sbus=sbus[:n])
            assert np.array_equal(mismatch(n), large[:n])
            bad = sbus[:n].copy()
            bad[n - 1, 299, 1] = np.inf
            with pytest.raises(m.MpfError, match="non-finite"):
                pf.set_cases([[]] * n, sbus=bad)
            assert np.array_equal(mismatch(n), large[:n])


def test_evaluation_captured_right_after_new_cases(gpu):
    """mpf_mismatch_noalloc in a stream capture, called while the uploads of mpf_set_cases may still
    run: the replay gives what the plain call gives."""
    import torch

    from mapol_b200._lib import lib

    buses, branches, cases = m.workload("cfg1_300bus")
    flat = np.repeat(np.stack([buses["vm"] * np.cos(buses["va"]), buses["vm"] * np.sin(buses["va"])], -1)[None], 64, 0)
    v = torch.from_numpy(flat).cuda()
    ref = torch.zeros(64, dtype=torch.float64, device="cuda")
    got = torch.zeros(64, dtype=torch.float64, device="cuda")
    with m.PowerFlow(buses, branches) as pf:
        pf.set_cases(cases[:64])
        assert lib().mpf_mismatch_noalloc(pf._h, v.data_ptr(), ref.data_ptr(), None) == 0
        torch.cuda.synchronize()
        side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        pf.set_cases(cases[:64])
        with torch.cuda.graph(graph, stream=side):
            rc = lib().mpf_mismatch_noalloc(pf._h, v.data_ptr(), got.data_ptr(), side.cuda_stream)
        assert rc == 0, lib().mpf_last_error(pf._h)
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(got.cpu().numpy(), ref.cpu().numpy()) and (ref > 0).all()
        del graph


@pytest.mark.parametrize("prec", [m.FP64, m.MIXED])
@pytest.mark.parametrize("alg", [m.NR, m.FDXB])
@pytest.mark.parametrize("n_cases", [40, 9000])
def test_first_solves_on_other_streams(gpu, alg, prec, n_cases):
    """A new handle's first solve and adjoint on streams of the caller, which have to wait for the
    tables and plans that the calls themselves upload: bit for bit what its own stream gives.
    (40 cases run on chunks, 9000 on level launches.)"""
    import torch

    from mapol_b200._lib import lib

    buses, branches = m.synth_grid(118, 179, 53, 0.1, seed=3)
    n1 = np.flatnonzero(~m.find_bridges(branches, 118))
    cases = [[int(b)] for b in np.resize(n1, n_cases)]
    sbus = np.repeat(np.stack([buses["p"], buses["q"]], -1)[None], n_cases, 0) * np.linspace(0.9, 1.0, n_cases)[:, None, None]
    out = []
    for streams in ((None, None), (torch.cuda.Stream(), torch.cuda.Stream())):
        ptrs = [s.cuda_stream if s else None for s in streams]
        grads = [torch.zeros((n_cases, n), dtype=torch.float64, device="cuda") for n in (118, 118, 179, 179)]
        torch.cuda.synchronize()
        with m.PowerFlow(buses, branches) as pf:
            pf.set_cases(cases, sbus=sbus)
            pf.solve(alg, prec, stream=ptrs[0])
            pf.set_ratings(np.full(179, 0.3))
            assert lib().mpf_adjoint(pf._h, prec, *[g.data_ptr() for g in grads], ptrs[1]) == 0
            torch.cuda.synchronize()
            res = pf.results()
            assert res.converged.all()
            out.append([res.v, res.iterations] + [g.cpu().numpy() for g in grads])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
