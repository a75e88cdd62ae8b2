"""The longest state vectors the plain gain stages in shared memory (20,800 FP64 or 41,600 FP32 states,
padded per species): accepted and right by a contraction and by a stepped context, against FP64
(relative L-inf 1e-12 and 2e-5, the tolerances of the plain path); a longer one is refused."""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sp

from dtb import _lib, synth
from dtb.stepping import ForwardEulerStruct
from dtb.structs import BinaryMatrices, EmissionMatrices, FluxMatrices, GainBlock

pytestmark = pytest.mark.gpu

LONGEST = {"f64": 20800, "f32": 41600}
TOL = {"f64": 1e-12, "f32": 2e-5}


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("n2", [8, 1024])
def test_longest_contraction(cuda, prec, n2):
    import torch
    L, dt = _lib.load(), torch.float64 if prec == "f64" else torch.float32
    code = _lib.DTB_DTYPE_F64 if prec == "f64" else _lib.DTB_DTYPE_F32
    g = torch.Generator(device="cuda")
    g.manual_seed(n2)

    def contract(n1):
        G = torch.rand((2, n1, n2), generator=g, device="cuda", dtype=dt)
        f1, f2 = (torch.rand(n, generator=g, device="cuda", dtype=dt) for n in (n1, n2))
        out = torch.zeros(2, device="cuda", dtype=torch.float64)
        s = torch.cuda.current_stream().cuda_stream
        rc = L.dtb_gain_contract(code, *(ctypes.c_void_p(x) for x in (G.data_ptr(),)), 2, n1, n2,
                                 *(ctypes.c_void_p(x) for x in (f1.data_ptr(), f2.data_ptr(), out.data_ptr(), s)))
        torch.cuda.synchronize()
        return rc, out, torch.einsum("abc,b,c->a", G.double(), f1.double(), f2.double())

    rc, out, ref = contract(LONGEST[prec] - n2)
    assert rc == _lib.DTB_OK
    assert float((out - ref).abs().max() / ref.abs().max()) <= TOL[prec]
    assert contract(LONGEST[prec] - n2 + 8)[0] == _lib.DTB_EINVAL


@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_longest_state_steps(cuda, prec):
    """8 photon states and an electron species that fills the rest: G[photon][electron][photon]."""
    n0, n1 = LONGEST[prec] - 8, 8
    ps = synth.uneven_two_species(4, 2, 4, 2, seed=1).ps
    ps.px_num_list, ps.py_num_list = [n0, 4], [1, 2]
    rng = np.random.default_rng(2)
    G, f0 = rng.uniform(0.0, 1.0 / n0, (n1, n0, n1)), rng.uniform(0.5, 1.5, n0 + n1)
    n = n0 + n1
    empty = sp.csc_matrix((n, n))
    m = ForwardEulerStruct(ps, f0, np.zeros(n), BinaryMatrices(gains=[GainBlock(1, 0, 1, G)]), EmissionMatrices(),
                           FluxMatrices(Ap_Flux=np.ones(n), Am_Flux=np.ones(n), X_Flux=empty, P_Flux=empty,
                                        Vol=np.ones(1)),
                           Precision=np.float64 if prec == "f64" else np.float32)
    m.run([0.5])
    exp = f0.copy()
    exp[n0:] += 0.5 * np.einsum("abc,b,c->a", G, f0[:n0], f0[n0:])
    assert np.max(np.abs(m.f - exp)) / np.max(np.abs(exp)) <= TOL[prec]
    m.close()
