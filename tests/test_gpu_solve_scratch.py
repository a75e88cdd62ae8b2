"""A Solve with moments allocates no device memory once its context has run one: the stream-ordered
pool's high-water mark stays at zero, and the device bytes of the context where the first call left
them. Moments of more save points than the context keeps room for agree with dtb_moments as well."""
import ctypes

import numpy as np
import pytest

from dtb import synth
from dtb.stepping import ForwardEulerStruct, Solve
from dtb.structs import energy_weights

pytestmark = pytest.mark.gpu

USED_HIGH = 8  # CU_MEMPOOL_ATTR_USED_MEM_HIGH


def _pool():
    import torch
    torch.zeros(1, device="cuda")
    cu, pool, dev = ctypes.CDLL("libcuda.so.1"), ctypes.c_void_p(), ctypes.c_int()
    assert cu.cuCtxGetDevice(ctypes.byref(dev)) == 0
    assert cu.cuDeviceGetDefaultMemPool(ctypes.byref(pool), dev) == 0
    return cu, pool


def _method():
    w = synth.uneven_two_species(5, 4, 6, 4, seed=3)
    return w, ForwardEulerStruct(w.ps, w.f0, w.inj, w.binm, w.emim, w.fluxm)


def test_solve_with_moments_keeps_its_scratch(cuda):
    w, m = _method()
    weights = energy_weights(w.ps)
    t = [0.0, 10.0, 25.0, 40.0]
    first = Solve(m, 1.0, t, Verbose=0, moment_weights=weights)
    held = m.device_bytes()
    cu, pool = _pool()
    high = ctypes.c_uint64(0)
    assert cu.cuMemPoolSetAttribute(pool, USED_HIGH, ctypes.byref(high)) == 0
    again = Solve(m, 1.0, t, Verbose=0, moment_weights=weights)
    assert cu.cuMemPoolGetAttribute(pool, USED_HIGH, ctypes.byref(high)) == 0
    assert high.value == 0 and m.device_bytes() == held
    np.testing.assert_array_equal(first.number, again.number)
    np.testing.assert_array_equal(first.energy, again.energy)
    m.close()


@pytest.mark.parametrize("saves", [2, 32768, 33000])  # 1 MB holds 32,768 saves of two species' moments
def test_moments_of_few_and_many_saves(cuda, saves):
    w, m = _method()
    weights = energy_weights(w.ps)
    o = Solve(m, 1.0, [float(k) for k in range(saves)], Verbose=0, moment_weights=weights)
    for k in (0, saves // 2, saves - 1):
        m.f = o.f[k]
        number, energy = m.moments(weights)
        np.testing.assert_array_equal(o.number[k], number)
        np.testing.assert_array_equal(o.energy[k], energy)
    m.close()
