"""Runs on the kernel that keeps the gain units in shared memory (the library's choice for small
grids and runs of a graph's length and more) against the same steps taken one by one: states and
step records bit for bit, launch counts (a launch and a diagnostics reduction per 64 steps), and
the FP64 oracle (relative L-inf 1e-12, FP32 2e-5). Species of odd sizes, several cells (more than
one pass over the units), the symplectic method, a sparse M_Bin, b-rows of more than 256 16-byte
columns, more units than blocks and fewer, every Verbose level."""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sp

import oracle
from dtb import synth
from dtb.stepping import ForwardEulerStruct, ForwardSymplecticEulerStruct, Solve
from dtb.structs import BinaryMatrices, FluxMatrices, blocked_to_ref

pytestmark = pytest.mark.gpu

TOL = {"f64": 1e-12, "f32": 2e-5}
FIELDS = ("cr", "cr_bin", "cr_emi", "cr_flux", "sum_df", "sum_f", "finite")


def _workload(grid, cells, seed):
    w = synth.uneven_two_species(*grid, seed=seed)
    w.ps.x_num = cells
    n, rng = w.ps.n_state, np.random.default_rng(seed + 1)
    X = synth.space_flux(w.ps, rng, 1.0) if cells > 1 else sp.csc_matrix((n, n))
    w.fluxm = FluxMatrices(Ap_Flux=rng.uniform(0.8, 1.25, n), Am_Flux=np.ones(n), X_Flux=X,
                           P_Flux=synth.upwind_flux(w.ps, rng, 1.0).P_Flux * 0.5, Vol=rng.uniform(0.5, 1.5, cells))
    w.f0 = synth.lognormal_f0(w.ps, [0.0, 0.3], 1.0) * rng.uniform(0.5, 1.5, n)
    w.inj = rng.uniform(0.0, 1e-4, n)
    return w


def _launches(m):
    n = ctypes.c_int64()
    m.L.dtb_launch_count(m.ctx, ctypes.byref(n))
    return n.value


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("grid,cells,sympl,steps,verbose", [
    ((16, 8, 16, 8), 1, False, 70, 1), ((10, 8, 12, 4), 1, False, 130, 3), ((5, 3, 7, 2), 1, False, 64, 2),
    ((5, 3, 9, 3), 3, False, 67, 3), ((8, 4, 6, 4), 9, False, 64, 1), ((3, 1, 66, 8), 1, False, 64, 1),
    ((3, 1, 67, 8), 2, False, 65, 1), ((10, 8, 9, 7), 4, True, 66, 3), ((7, 5, 9, 3), 5, True, 129, 1),
    ((4, 2, 3, 3), 1, True, 64, 0)])
def test_resident_run_equals_single_steps(cuda, prec, grid, cells, sympl, steps, verbose):
    w = _workload(grid, cells, 80 + cells)
    cls = ForwardSymplecticEulerStruct if sympl else ForwardEulerStruct
    a, b = (cls(w.ps, w.f0, w.inj, w.binm, w.emim, w.fluxm, Precision=np.float64 if prec == "f64" else np.float32)
            for _ in range(2))
    dt = np.random.default_rng(3).uniform(0.5, 1.0, steps)
    before = _launches(a)
    hist = a.run(dt, Verbose=verbose, diag=True)
    assert _launches(a) - before == 2 * ((steps + 63) // 64)
    for k in range(steps):
        b(0.0, 1e9, float(dt[k]), verbose)
        if verbose:
            assert [getattr(hist[k], x) for x in FIELDS] == [getattr(b.last_diag, x) for x in FIELDS], k
    np.testing.assert_array_equal(a.f, b.f)
    a.run(dt[:64])  # a second run from the new state, beside one more step each way
    for k in range(64):
        b(0.0, 1e9, float(dt[k]), 0)
    np.testing.assert_array_equal(a.f, b.f)
    if not sympl:
        a.f = w.f0
        a.run(dt)
        ops, f = oracle.blocked_from_workload(w), w.f0.copy()
        for k in range(steps):
            f, _, _ = ops.step(f, float(dt[k]), 0)
        assert np.max(np.abs(a.f - f)) / np.max(np.abs(f)) <= TOL[prec]
    a.close()
    b.close()


def test_resident_sparse_and_solve_intervals(cuda):
    """A sparse M_Bin, and a Solve whose save intervals are shorter and longer than a launch's
    steps: equal, bit for bit, to the stepwise loop."""
    w = _workload((6, 4, 5, 4), 2, 90)
    for g in w.binm.gains:
        g.G = np.where(np.random.default_rng(5).random(g.G.shape) < 0.3, g.G, 0.0)
    M = sp.csc_matrix(blocked_to_ref(w.ps, w.binm))
    m = ForwardEulerStruct(w.ps, w.f0, w.inj, BinaryMatrices(M_Bin=M), w.emim, w.fluxm)
    t_save = [0.0, 3.0, 14.0, 110.0, 111.0, 180.0]
    fast, slow = Solve(m, 1.0, t_save, Verbose=0), Solve(m, 1.0, t_save, Verbose=0, stepwise=True)
    for x, y in zip(fast.f, slow.f):
        np.testing.assert_array_equal(x, y)
    ops, f = oracle.blocked_from_workload(w), w.f0.copy()
    for _ in range(180):
        f, _, _ = ops.step(f, 1.0, 0)
    assert np.max(np.abs(fast.f[-1] - f)) / np.max(np.abs(f)) <= TOL["f64"]
    m.close()
