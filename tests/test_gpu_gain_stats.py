"""dtb_gain_kernel_stats: the bytes of a gain launch count one read of the gain blocks per pass over the
cells of the binary domain (up to eight cells share a read), not one per cell."""
import ctypes

import numpy as np
import pytest

from dtb import _lib
from dtb.stepping import ForwardEulerStruct

from test_gpu_gain_pass import _cells_workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("cells,domain,reads", [(1, None, 1), (8, None, 1), (9, None, 2), (17, None, 3),
                                                (9, [0, 2, 5, 8], 1), (3, [], 0)])
def test_bytes_per_launch(cuda, prec, cells, domain, reads):
    w = _cells_workload((5, 3, 9, 3), cells, 7)
    w.binm.Domain = domain
    m = ForwardEulerStruct(w.ps, w.f0, w.inj, w.binm, w.emim, w.fluxm,
                           Precision=np.float64 if prec == "f64" else np.float32)
    L, ms, by = _lib.load(), ctypes.c_double(), ctypes.c_double()
    _lib.check(L.dtb_set_profiling(m.ctx, 1))
    m.run(np.full(4, 0.5))
    _lib.check(L.dtb_gain_kernel_stats(m.ctx, ctypes.byref(ms), ctypes.byref(by)))
    elems = (15 + 27) * 15 * 27
    assert by.value == reads * elems * (8 if prec == "f64" else 4)
    assert (ms.value > 0) == (reads > 0)
    m.close()
