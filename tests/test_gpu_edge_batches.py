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
