"""The plain gain's variants by G's size: contractions large enough for three and four 16-byte columns per
thread (one FP32 cell), at the edges of their row lengths, against FP64 sums of the same values
(relative L-inf 2e-5 FP32, 1e-12 FP64), and steps of several cells on rows of more than 512 columns,
which take one FP32 cell and three or four FP64 cells per pass, against the FP64 oracle."""
import ctypes

import pytest

from dtb import _lib

from test_gpu_gain_pass import _cells_workload, _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,n2", [("f32", n) for n in (32, 40, 48, 72, 264, 384, 392, 1032, 2048, 2056, 2600, 3072,
                                                          3080, 4096)] + [("f64", n) for n in (40, 520, 1032, 2048)])
@pytest.mark.parametrize("n1", [37, 256])
def test_large_contraction(cuda, prec, n2, n1):
    import torch
    dt = torch.float64 if prec == "f64" else torch.float32
    esz = 8 if prec == "f64" else 4
    n_out = 82_000_000 // (n1 * n2 * esz) + 1  # just above the size from which more columns are taken
    g = torch.Generator(device="cuda")
    g.manual_seed(n2 + n1)
    G = torch.rand((n_out, n1, n2), generator=g, device="cuda", dtype=dt)
    f1, f2 = (torch.rand(n, generator=g, device="cuda", dtype=dt) for n in (n1, n2))
    out = torch.zeros(n_out, device="cuda", dtype=torch.float64)
    s = torch.cuda.current_stream().cuda_stream
    _lib.check(_lib.load().dtb_gain_contract(
        _lib.DTB_DTYPE_F64 if prec == "f64" else _lib.DTB_DTYPE_F32, ctypes.c_void_p(G.data_ptr()), n_out, n1, n2,
        *(ctypes.c_void_p(x) for x in (f1.data_ptr(), f2.data_ptr(), out.data_ptr(), s))))
    torch.cuda.synchronize()
    ref = torch.stack([f1.double() @ (G[a].double() @ f2.double()) for a in range(n_out)])
    assert float((out - ref).abs().max() / ref.abs().max()) <= (1e-12 if prec == "f64" else 2e-5)


@pytest.mark.parametrize("prec,cells,p_g,u_g", [("f32", 2, 257, 8), ("f32", 3, 384, 8), ("f32", 5, 512, 8),
                                                ("f64", 4, 129, 8), ("f64", 4, 215, 8), ("f64", 4, 216, 8),
                                                ("f64", 4, 256, 8), ("f64", 8, 129, 8), ("f64", 7, 250, 8)])
def test_cells_on_long_rows(cuda, prec, cells, p_g, u_g):
    _check(_cells_workload((2, 1, p_g, u_g), cells, 8, flux=False), prec, steps=2)


@pytest.mark.parametrize("prec,cells,p_e,p_g", [("f32", 1, 4, 129), ("f32", 1, 2, 239), ("f32", 7, 4, 20), ("f64", 1, 3, 129),
                                                ("f64", 1, 4, 70), ("f64", 1, 9, 79), ("f64", 2, 3, 66), ("f64", 2, 3, 60),
                                                ("f64", 2, 3, 119), ("f64", 3, 5, 30), ("f64", 3, 2, 79), ("f64", 7, 6, 10)])
def test_runs_on_long_rows_equal_steps(cuda, prec, cells, p_e, p_g):
    """Runs of 66 steps with the gain in shared memory, every columns-per-thread variant and both state
    lengths per thread, bit for bit against single steps."""
    import numpy as np
    from dtb.stepping import ForwardEulerStruct
    w = _cells_workload((p_e, 1, p_g, 8), cells, 9, flux=False)
    a, b = (ForwardEulerStruct(w.ps, w.f0, w.inj, w.binm, w.emim, w.fluxm,
                               Precision=np.float64 if prec == "f64" else np.float32) for _ in range(2))
    dt = np.random.default_rng(5).uniform(0.5, 1.0, 66)
    n0, n1 = ctypes.c_int64(), ctypes.c_int64()
    a.L.dtb_launch_count(a.ctx, ctypes.byref(n0))
    a.run(dt)
    a.L.dtb_launch_count(a.ctx, ctypes.byref(n1))
    assert n1.value - n0.value == 4
    for x in dt:
        b(0.0, 1e9, float(x), 0)
    np.testing.assert_array_equal(a.f, b.f)
    a.close()
    b.close()
