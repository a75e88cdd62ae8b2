"""The gain pass over several space cells: every number of cells that shares one read of G (one to
eight, and the remainders past them), binary domains, and b-rows of one, two and four 16-byte
columns per thread, FP64 and FP32, against the FP64 oracle (relative L-inf 1e-12 and 2e-5, the
tolerances of the plain path)."""
import numpy as np
import pytest
import scipy.sparse as sp

import oracle
from dtb import synth
from dtb.stepping import ForwardEulerStruct
from dtb.structs import BinaryMatrices, EmissionMatrices, FluxMatrices

pytestmark = pytest.mark.gpu

TOL = {"f64": 1e-12, "f32": 2e-5}


def _cells_workload(grid, cells, seed, flux=True):
    """uneven_two_species' operators on `cells` space cells with their own spectra and Vol."""
    w = synth.uneven_two_species(*grid, seed=seed) if flux else None
    if w is None:  # long b-rows: the flux of thousands of states adds nothing here
        p_e, u_e, p_g, u_g = grid
        small = synth.uneven_two_species(4, 2, 4, 2, seed=seed)
        ps = small.ps
        ps.px_num_list, ps.py_num_list = [p_e, p_g], [u_e, u_g]
        ps.pxr_list = [np.logspace(-2, 2, n + 1) for n in ps.px_num_list]
        rng = np.random.default_rng(seed)
        ne, ng = ps.species_sizes
        gains = [synth.GainBlock(o, 0, 1, 10.0 ** rng.uniform(-6, 0, (n, ne, ng)) * synth.gain_kappa(-6, 0, n, 1.0))
                 for o, n in ((0, ne), (1, ng))]
        losses = [synth.LossBlock(0, 1, 10.0 ** rng.uniform(-6, 0, (ne, ng)) * synth.loss_kappa(-6, 0, 1.0))]
        small.binm, small.emim = BinaryMatrices(gains=gains, losses=losses), EmissionMatrices()
        w = small
    w.ps.x_num = cells
    n, rng = w.ps.n_state, np.random.default_rng(seed + 1)
    P = synth.upwind_flux(w.ps, rng, 1.0).P_Flux if flux else sp.csc_matrix((n, n))
    w.fluxm = FluxMatrices(Ap_Flux=rng.uniform(0.8, 1.25, n), Am_Flux=np.ones(n), X_Flux=sp.csc_matrix((n, n)),
                           P_Flux=P, Vol=rng.uniform(0.5, 1.5, cells))
    w.f0 = synth.lognormal_f0(w.ps, [0.0, 0.3], 1.0) * rng.uniform(0.5, 1.5, n)
    w.inj = rng.uniform(0.0, 1e-4, n)
    return w


def _check(w, prec, steps=3):
    m = ForwardEulerStruct(w.ps, w.f0, w.inj, w.binm, w.emim, w.fluxm,
                           Precision=np.float64 if prec == "f64" else np.float32)
    ops, f = oracle.blocked_from_workload(w), w.f0.copy()
    for _ in range(steps):
        m(0.0, 1e9, 0.8 * m.dt0, 1)
        f, _, _ = ops.step(f, 0.8, 1)
    got = m.f
    m.close()
    assert np.max(np.abs(got - f)) / np.max(np.abs(f)) <= TOL[prec]


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("cells,domain", [(1, None), (2, None), (3, None), (4, None), (5, None), (6, None), (7, None),
                                          (8, None), (9, None), (17, None), (11, [0, 1, 4, 5, 6, 9, 10]), (6, [5])])
def test_cells_of_a_pass_match_oracle(cuda, prec, cells, domain):
    w = _cells_workload((5, 3, 9, 3), cells, 40 + cells)
    w.binm.Domain = domain
    _check(w, prec)


@pytest.mark.parametrize("prec,cells,p_g,u_g", [
    ("f64", 1, 64, 8), ("f64", 1, 65, 8), ("f64", 5, 65, 8), ("f64", 1, 103, 10), ("f64", 3, 128, 8), ("f64", 2, 128, 16),
    ("f32", 1, 130, 8), ("f32", 4, 130, 8), ("f32", 3, 128, 16), ("f32", 1, 150, 14)])
def test_long_b_rows_match_oracle(cuda, prec, cells, p_g, u_g):
    """256 16-byte columns per b-row and just past, up to 1024: one, two and four per thread."""
    _check(_cells_workload((3, 1, p_g, u_g), cells, 7, flux=False), prec, steps=2)
