"""Several live plain contexts (and the context-free contraction) that share kernel instances but need
different amounts of shared memory: whatever is committed or called in between, a context's steps,
runs and Solves go on, with the bits of a context that was alone."""
import ctypes

import numpy as np
import pytest

from dtb import _lib, synth
from dtb.stepping import ForwardEulerStruct, Solve

pytestmark = pytest.mark.gpu


def _method(grid, prec, graph_steps=0):
    w = synth.uneven_two_species(*grid, seed=sum(grid))
    return ForwardEulerStruct(w.ps, w.f0, w.inj, w.binm, w.emim, w.fluxm,
                              Precision=np.float64 if prec == "f64" else np.float32, graph_steps=graph_steps)


def _drive(m):
    """A long run, a step and a Solve from the initial state: every state they end in."""
    out = []
    m.reset()
    m.run(np.linspace(0.5, 1.0, 70))
    out.append(m.f)
    m(0.0, 1e9, 0.75, 1)
    out.append(m.f)
    return out + Solve(m, 1.0, [0.0, 9.0, 80.0], Verbose=0).f


def _contract(n1, n2, prec):
    import torch
    dt = torch.float64 if prec == "f64" else torch.float32
    G, f1, f2 = (torch.ones(s, device="cuda", dtype=dt) for s in ((4, n1, n2), (n1,), (n2,)))
    out = torch.zeros(4, device="cuda", dtype=torch.float64)
    s = torch.cuda.current_stream().cuda_stream
    _lib.check(_lib.load().dtb_gain_contract(_lib.DTB_DTYPE_F64 if prec == "f64" else _lib.DTB_DTYPE_F32,
                                             *(ctypes.c_void_p(x) for x in (G.data_ptr(),)), 4, n1, n2,
                                             *(ctypes.c_void_p(x) for x in (f1.data_ptr(), f2.data_ptr(), out.data_ptr(), s))))
    torch.cuda.synchronize()
    assert (out == n1 * n2).all()


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("graph_steps", [0, 16])  # the gain kept in shared memory, and streamed
@pytest.mark.parametrize("large,small", [((16, 8, 16, 8), (4, 2, 4, 2)), ((16, 8, 16, 8), (16, 8, 15, 8)),
                                         ((13, 8, 12, 8), (8, 8, 8, 8))])
def test_contexts_of_different_sizes_run_in_turn(cuda, prec, graph_steps, large, small):
    a = _method(large, prec, graph_steps)
    alone = _drive(a)
    b = _method(small, prec, graph_steps)  # the smaller need is stated last
    _contract(8, 8, prec)
    other = _drive(b)
    for _ in range(2):
        for m, ref in ((a, alone), (b, other)):
            for x, y in zip(_drive(m), ref):
                np.testing.assert_array_equal(x, y)
            _contract(24, 8, prec)
    a.close()
    b.close()


def test_contexts_run_at_once_on_their_own_threads(cuda):
    """Three contexts on their own streams and host threads, two that keep the gain in shared memory (every
    block of a launch waits for the others) and one that streams: each ends in the bits it has alone."""
    import threading
    cases = [((16, 8, 16, 8), "f64", 0), ((13, 8, 12, 8), "f32", 0), ((8, 8, 8, 8), "f64", 16)]
    ms = [_method(*c) for c in cases]
    dt = np.linspace(0.5, 1.0, 200)

    def drive(m):
        m.reset()
        for _ in range(5):
            m.run(dt)
            m(0.0, 1e9, 0.75, 1)
        return m.f

    alone, at_once = [drive(m) for m in ms], [None] * len(ms)
    threads = [threading.Thread(target=lambda k=k: at_once.__setitem__(k, drive(ms[k]))) for k in range(len(ms))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for x, y in zip(alone, at_once):
        np.testing.assert_array_equal(x, y)
    for m in ms:
        m.close()
