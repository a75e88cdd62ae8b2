"""The batched epilogue's row tiles against the FP64 oracle (relative L-inf 1e-5, the batched
path's tolerance): species and cells that end inside a tile, group rows that are no multiples of
four, emission pieces that change inside a tile (after eight rows and more, and sooner), few and
many slots (16 x 16 and 32 x 32 tiles)."""
import numpy as np
import pytest
import scipy.sparse as sp

import oracle
from dtb import synth
from dtb.batch import BatchedEuler
from dtb.structs import EmiBlock, EmissionMatrices, FluxMatrices

pytestmark = pytest.mark.gpu

TOL_MIXED = 1e-5


def _workload(grid, cells, batch, cuts, seed):
    """uneven_two_species on `cells` cells; the photon emission of every cell cut into row pieces at `cuts`."""
    w = synth.uneven_two_species(*grid, seed=seed)
    E = w.emim.blocks[0].E
    w.ps.x_num = cells
    nm, off, n = w.ps.n_momentum, w.ps.momentum_species_offset[1], w.ps.n_state
    rng = np.random.default_rng(seed + 1)
    edges = [0] + [c for c in cuts if c < E.shape[0]] + [E.shape[0]]
    w.emim = EmissionMatrices(blocks=[EmiBlock(row0=k * nm + off + lo, col0=k * nm, E=E[lo:hi])
                                      for k in range(cells) for lo, hi in zip(edges, edges[1:])])
    w.fluxm = FluxMatrices(Ap_Flux=rng.uniform(0.8, 1.25, n), Am_Flux=np.ones(n), X_Flux=sp.csc_matrix((n, n)),
                           P_Flux=synth.upwind_flux(w.ps, rng, 1.0).P_Flux, Vol=rng.uniform(0.5, 1.5, cells))
    w.inj = rng.uniform(0.0, 1e-4, n)
    w.f0 = synth.lognormal_f0(w.ps, [0.0, 0.3], 1.0) * rng.uniform(0.5, 1.5, (batch, n))
    w.dt = rng.uniform(0.5, 1.0, batch)
    return w


@pytest.mark.parametrize("grid,cells,batch,cuts", [
    ((8, 4, 8, 4), 1, 5, ()), ((7, 5, 9, 3), 1, 1, ()), ((7, 5, 9, 3), 3, 17, ()), ((11, 3, 5, 5), 2, 33, (9,)),
    ((4, 4, 13, 4), 1, 6, (3, 20, 21)), ((16, 8, 5, 3), 1, 40, (2,)), ((8, 4, 7, 5), 1, 2400, ()),
    ((8, 4, 8, 8), 2, 1300, (8, 11))])
def test_row_tiles_match_oracle(cuda, grid, cells, batch, cuts):
    w = _workload(grid, cells, batch, cuts, seed=60 + batch)
    m = BatchedEuler(w.ps, w.inj, w.binm, w.emim, w.fluxm, batch)
    for i in range(batch):
        m.admit(i, w.f0[i], float(w.dt[i]), 12)
    m.run(12)
    got = m.get_f_all()
    m.close()
    ops = oracle.blocked_from_workload(w)
    for i in sorted({0, batch // 2, batch - 1}):
        f = w.f0[i].copy()
        for _ in range(12):
            f, _, _ = ops.step(f, float(w.dt[i]), 0)
        assert np.max(np.abs(got[i] - f)) / np.max(np.abs(f)) <= TOL_MIXED
