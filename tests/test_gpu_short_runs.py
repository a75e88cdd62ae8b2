"""Which route the steps of a small grid take: runs of 64 steps and a Solve's save intervals of eight and
more keep the gain in shared memory (a launch and a diagnostics reduction per 64 steps), shorter ones
and contexts that kernel declines take the two kernels of a step, in work units chosen for them. The
symplectic method on either route against the FP64 oracle (relative L-inf 1e-12, FP32 2e-5)."""
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


def _workload(grid, cells, seed, x_slots=0):
    """uneven_two_species on `cells` cells; x_slots > 0: an X flux of about that many slots a row."""
    w = synth.uneven_two_species(*grid, seed=seed)
    w.ps.x_num = cells
    n, rng = w.ps.n_state, np.random.default_rng(seed + 1)
    X = synth.space_flux(w.ps, rng, 1.0) if cells > 1 else sp.csc_matrix((n, n))
    if x_slots:
        X = sp.random(n, n, density=x_slots / n, random_state=seed, format="csc") * (0.1 / x_slots)
    w.fluxm = FluxMatrices(Ap_Flux=rng.uniform(0.8, 1.25, n), Am_Flux=np.ones(n), X_Flux=X,
                           P_Flux=synth.upwind_flux(w.ps, rng, 1.0).P_Flux * 0.5, Vol=rng.uniform(0.5, 1.5, cells))
    w.f0 = synth.lognormal_f0(w.ps, [0.0, 0.3], 1.0) * rng.uniform(0.5, 1.5, n)
    w.inj = rng.uniform(0.0, 1e-4, n)
    return w


def _method(w, prec="f64", sympl=False, binm=None, **kw):
    return (ForwardSymplecticEulerStruct if sympl else ForwardEulerStruct)(
        w.ps, w.f0, w.inj, binm or w.binm, w.emim, w.fluxm, Precision=np.float64 if prec == "f64" else np.float32, **kw)


def _launches(m):
    n = ctypes.c_int64()
    m.L.dtb_launch_count(m.ctx, ctypes.byref(n))
    return n.value


def _oracle_symplectic(w, dts):
    r, L = oracle.ref_from_workload(w), oracle.lib()
    X, P = (oracle._csc_arrays(M) for M in (w.fluxm.X_Flux, w.fluxm.P_Flux))
    f, d = w.f0.copy(), np.zeros(8)
    for dt in dts:
        assert L.orc_step_symplectic_ref(
            r.n_mom, r.n_space, oracle._d(r.M_Bin), oracle._d(r.M_Emi), oracle._i(X[0]), oracle._i(X[1]),
            oracle._d(X[2]), oracle._i(P[0]), oracle._i(P[1]), oracle._d(P[2]), 0, oracle._d(r.invAp), oracle._d(r.Vol),
            oracle._d(r.inj), float(dt), float(np.float32(1e-10)), float(np.float32(1e-20)), 1, oracle._d(f),
            oracle._d(d), oracle._b(r.dom)) == 0
    return f


@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_route_of_a_run_and_its_bits(cuda, prec):
    w = _workload((10, 8, 12, 4), 1, 91)
    a, b = _method(w, prec), _method(w, prec)
    for n in (1, 2, 3, 4, 5, 8, 10, 37, 63, 64):
        dt = np.random.default_rng(n).uniform(0.5, 1.0, n)
        before = _launches(a)
        a.run(dt)
        assert _launches(a) - before == (2 if n >= 64 else 2 * n + 1), n
        for x in dt:
            b(0.0, 1e9, float(x), 0)
        np.testing.assert_array_equal(a.f, b.f)
    a.close()
    b.close()


def test_solve_intervals_and_sparse_operators_take_it_too(cuda):
    w = _workload((6, 4, 5, 4), 2, 92)
    for g in w.binm.gains:
        g.G = np.where(np.random.default_rng(5).random(g.G.shape) < 0.3, g.G, 0.0)
    M = BinaryMatrices(M_Bin=sp.csc_matrix(blocked_to_ref(w.ps, w.binm)))
    m = _method(w, binm=M)
    Solve(m, 1.0, [0.0, 1.0], Verbose=0)
    before = _launches(m)
    fast = Solve(m, 1.0, [0.0, 3.0, 14.0, 110.0, 111.0, 180.0], Verbose=0)
    # intervals of 3 and 1 steps: two kernels a step and one reduction; of 11, 96 and 69: two launches per 64
    assert _launches(m) - before == (2 * 3 + 1) + 2 + 4 + (2 + 1) + 4
    slow = Solve(m, 1.0, [0.0, 3.0, 14.0, 110.0, 111.0, 180.0], Verbose=0, stepwise=True)
    for x, y in zip(fast.f, slow.f):
        np.testing.assert_array_equal(x, y)
    m.close()


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("grid,cells,x_slots,resident", [((10, 8, 9, 7), 4, 0, True), ((7, 5, 9, 3), 5, 0, True),
                                                         ((6, 4, 40, 8), 2, 0, True), ((6, 4, 40, 8), 2, 14, False)])
def test_symplectic_runs_match_the_oracle(cuda, prec, grid, cells, x_slots, resident):
    w = _workload(grid, cells, 93 + cells, x_slots)
    m = _method(w, prec, sympl=True)
    dt = np.random.default_rng(4).uniform(0.5, 1.0, 66)
    before = _launches(m)
    m.run(dt)
    assert _launches(m) - before == (4 if resident else 3 * 66 + 2)
    f = _oracle_symplectic(w, dt)
    assert np.max(np.abs(m.f - f)) / np.max(np.abs(f)) <= TOL[prec]
    if not resident:  # declined: the units of a context that never considers that kernel, hence its bits
        s = _method(w, prec, sympl=True, graph_steps=64)
        s.run(dt)
        np.testing.assert_array_equal(m.f, s.f)
        s.close()
    m.close()
