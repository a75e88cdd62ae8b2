"""Performance cases of the explicit Euler framework, each one pass through its public entry points.

The work a program has the framework do, over its range: host round trips of one step on a small
grid, whole Solves, long runs of one instance on grids from 2 x 16 to 2 x 1024 states in FP64 and
FP32, grids with several space cells (explicit and symplectic), a sparse M_Bin, batches of
instances on one grid (FP32 state, BF16 hi + lo operators) and a served stream of requests.

Operators and spectra follow the package's synthetic recipe (dtb.synth): upwind flux, log-uniform
gain, loss and emission entries scaled so that a step moves a small fraction of each species,
log-normal spectra. Everything a program keeps between calls (the method with its uploaded
operators, its page-locked host arrays) is made by prepare; run starts from the given spectra.

Batched and FP32 states are returned in FP32, the precision these methods keep f in."""
import math
import os
import sys

import numpy as np
import torch

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "diplodocustransport.jl_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

from dtb import synth  # noqa: E402
from dtb.batch import BatchedEuler  # noqa: E402
from dtb.serve import Server  # noqa: E402
from dtb.stepping import ForwardEulerStruct, ForwardSymplecticEulerStruct, Solve  # noqa: E402
from dtb.structs import (BinaryMatrices, EmiBlock, EmissionMatrices, FluxMatrices, GainBlock, LossBlock,  # noqa: E402
                         PhaseSpace, energy_weights)

THR = float(np.float32(1e-10))
THR_SPACE = float(np.float32(1e-20))


# ---------------------------------------------------------------- the cases
def _case(name, kind, grid, precision="f64", cells=1, steps=64, saves=0, batch=0, symplectic=False, sparse=False):
    """grid: "p x u" per species, two or three of them ("16x8,16x8")."""
    return dict(name=name, kind=kind, grid=grid, precision=precision, cells=cells, steps=steps, saves=saves,
                batch=batch, symplectic=symplectic, sparse=sparse)


def listed():
    return [
        # one step from host memory with its diagnostics, as a host program that owns f drives the
        # functor; the smallest call, on species of different, odd sizes
        _case("step_io_uneven_f64", "step_io", "10x8,12x4", steps=1),
        # Solve with save points and their moments on the smallest serving grid (1000 steps)
        _case("solve_p16u8_f64", "solve", "16x8,16x8", steps=1000, saves=10),
        # an ordinary FP64 run: 2 x 256 states, a gain operator of 268 MB
        _case("run_p32u8_f64", "run", "32x8,32x8"),
        # the largest single instance: 2 x 1024 states in FP32, 8.6 GB of gain operator
        _case("run_p64u16_f32", "run", "64x16,64x16", precision="f32"),
        # transport on eight space cells that share the collision operator
        _case("cells8_p32u8_f64", "run", "32x8,32x8", cells=8, steps=32),
        # the symplectic method on a few cells, FP32, sizes that are multiples of nothing
        _case("cells5_sympl_f32", "run", "20x7,18x7", precision="f32", cells=5, symplectic=True),
        # a sparse M_Bin in the reference layout (Bin_sparse), two cells
        _case("sparse_p12u7_f64", "run", "12x7,12x7", cells=2, sparse=True),
        # a full batch on the smallest serving grid: short GEMMs, many small steps
        _case("batch256_p16u8", "batch", "16x8,16x8", precision="mixed", batch=256),
        # the batched headline: 256 instances of 2 x 256 states
        _case("batch256_p32u8", "batch", "32x8,32x8", precision="mixed", batch=256),
        # three species with three interactions, 64 instances, 4.6 GB of operators per step
        _case("batch64_p48u12x3", "batch", "48x12,48x12,48x12", precision="mixed", batch=64, steps=16),
        # a ragged small batch: uneven species, three cells, 21 instances
        _case("batch21_cells3_uneven", "batch", "20x8,14x7", precision="mixed", batch=21, cells=3),
        # a served stream: requests of 40 to 300 steps on two grids, more requests than slots
        _case("serve_two_grids", "serve", "16x8,32x8", precision="mixed", batch=16, steps=300),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _two(rng, most, least=16):
    """Two species' grids, even odds of the same grid for both; at most `most` states each."""
    while True:
        g = [(_size(rng, 6, 64), _size(rng, 2, 16)) for _ in range(2)]
        if rng.random() < 0.5:
            g[1] = g[0]
        if all(least <= p * u <= most for p, u in g):
            return ",".join("%dx%d" % x for x in g)


def draw(rng):
    kind = rng.choice(["step_io", "solve", "run", "run", "cells", "cells", "sparse", "batch", "batch", "batch3", "serve"])
    prec = rng.choice(["f64", "f32"])
    if kind == "step_io":
        c = _case("", "step_io", _two(rng, 256), prec, steps=1)
    elif kind == "solve":
        c = _case("", "solve", _two(rng, 200), prec, steps=_size(rng, 100, 1000), saves=rng.randint(1, 20))
    elif kind == "run":
        c = _case("", "run", _two(rng, 640, least=48), prec, steps=rng.randint(10, 64))
    elif kind == "cells":
        c = _case("", "run", _two(rng, 256), prec, cells=rng.randint(2, 12), steps=rng.randint(10, 40),
                  symplectic=rng.random() < 0.4)
    elif kind == "sparse":
        c = _case("", "run", _two(rng, 90), prec, cells=rng.randint(1, 3), steps=rng.randint(20, 64), sparse=True)
    elif kind == "batch":
        cells = rng.choice([1, 1, 1, 2, 4])
        c = _case("", "batch", _two(rng, 512 if cells == 1 else 200), "mixed", cells=cells,
                  batch=_size(rng, 3, 256 if cells == 1 else 64), steps=rng.randint(10, 64))
    elif kind == "batch3":
        p, u = _size(rng, 8, 32), _size(rng, 3, 10)
        c = _case("", "batch", ",".join(["%dx%d" % (p, u)] * 3), "mixed", batch=_size(rng, 3, 128),
                  steps=rng.randint(8, 32))
    else:
        a, b = sorted(_two(rng, 256).split(","))
        c = _case("", "serve", "%s,%s" % (a, b), "mixed", batch=rng.randint(6, 48), steps=rng.randint(60, 300))
    del c["name"]
    return c


# ---------------------------------------------------------------- operators of a case
def _grids(case):
    return [tuple(int(x) for x in g.split("x")) for g in case["grid"].split(",")]


def _phase_space(grids, cells):
    pr = [np.logspace(-2.0, 2.0, p + 1) for p, _ in grids]
    k = len(grids)
    return PhaseSpace(name_list=["Ele", "Pho"] if k == 2 else ["Ele", "Pos", "Pho"],
                      px_num_list=[p for p, _ in grids], py_num_list=[u for _, u in grids], pz_num_list=[1] * k,
                      pxr_list=pr, pyr_list=[np.linspace(-1.0, 1.0, u + 1) for _, u in grids],
                      pzr_list=[np.array([0.0, 2.0])] * k, mass_list=[1.0] * (k - 1) + [0.0], x_num=cells, dt0=1.0)


def _upwind(n, lo, hi, rng, cfl):
    """Faces (lo[k], hi[k]) with velocity U[-1, 1]: the upwind side loses, the downwind side gains."""
    v = rng.uniform(-1.0, 1.0, lo.size)
    src, dst = np.where(v > 0, lo, hi), np.where(v > 0, hi, lo)
    w = np.abs(v)
    M = synth.sp.csc_matrix((np.concatenate([w, -w]), (np.concatenate([src, dst]), np.concatenate([src, src]))),
                            shape=(n, n))
    M.sum_duplicates()
    top = M.diagonal().max() if M.nnz else 0.0  # the spectral radius is at most twice the diagonal's maximum
    return M * (cfl / (2.0 * top)) if top > 0 else M


def _flux(ps, rng):
    n, nm = ps.n_state, ps.n_momentum
    lo, hi = [], []
    for off, p, u in zip(ps.momentum_species_offset, ps.px_num_list, ps.py_num_list):
        i = off + np.arange(p * u).reshape(u, p)
        lo += [i[:, :-1].ravel(), i[:-1].ravel()]
        hi += [i[:, 1:].ravel(), i[1:].ravel()]
    lo, hi = np.concatenate(lo), np.concatenate(hi)
    cell = nm * np.arange(ps.n_space)[:, None]
    P = _upwind(n, (lo + cell).ravel(), (hi + cell).ravel(), rng, 0.4)
    s = np.arange(n - nm)
    X = _upwind(n, s, s + nm, rng, 0.2) if ps.n_space > 1 else synth.sp.csc_matrix((n, n))
    return FluxMatrices(Ap_Flux=rng.uniform(0.8, 1.25, n), Am_Flux=np.ones(n), X_Flux=X, P_Flux=P,
                        Vol=rng.uniform(0.7, 1.3, ps.n_space))


def _energy_mask(ps, out):
    """Where a collision feeds output `out`: its momentum bin lies near the larger of the inputs'."""
    pa, pb, pc = (np.arange(ps.species_sizes[s]) % ps.px_num_list[s] for s in (out, 0, 1))
    return np.abs(pa[:, None, None] - np.maximum(pb[None, :, None], pc[None, None, :])) <= 2


def _csc_m_bin(ps, gains, losses):
    """The blocks scattered into the reference layout (half of each value to either input order)."""
    n, off = ps.n_momentum, ps.momentum_species_offset
    r, c, v = [], [], []
    for g in gains:
        a, b, k = (i.astype(np.int64) for i in np.nonzero(g.G))
        w = g.G[a, b, k] / 2
        a, b, k = a + off[g.out_sp], b + off[g.in1_sp], k + off[g.in2_sp]
        r, c, v = r + [b * n + a, k * n + a], c + [k, b], v + [w, w]
    for x in losses:
        a, k = (i.astype(np.int64) for i in np.nonzero(x.L))
        w = -x.L[a, k] / 2
        a, k = a + off[x.sp], k + off[x.other_sp]
        r, c, v = r + [a * n + a, k * n + a], c + [k, a], v + [w, w]
    return synth.sp.csc_matrix((np.concatenate(v), (np.concatenate(r), np.concatenate(c))), shape=(n * n, n))


def _workload(case, grids, cells, seed):
    """Operators, vectors and spectra of one grid, from the seed alone."""
    ps = _phase_space(grids, cells)
    rng = np.random.default_rng(seed)
    sizes, n = ps.species_sizes, ps.n_momentum
    flux = _flux(ps, rng)
    rng_g = (-8.0, 0.0) if len(grids) == 3 else (-6.0, 0.0)
    blocks = [(0, 0, 1), (1, 0, 1)] if len(grids) == 2 else [(0, 0, 2), (2, 0, 2), (1, 1, 2), (2, 1, 2), (0, 2, 2), (1, 2, 2)]
    dtype = torch.float64 if case["precision"] == "f64" else torch.float32
    gains = []
    for k, (o, b, c) in enumerate(blocks):
        shape, kappa = (sizes[o], sizes[b], sizes[c]), synth.gain_kappa(*rng_g, sizes[o], 1.0)
        if case["sparse"]:
            G = np.where(_energy_mask(ps, o), 10.0 ** rng.uniform(*rng_g, size=shape) * kappa * 3.0, 0.0)
        else:
            G = synth.device_log_uniform(shape, *rng_g, kappa, (seed * 1000 + 31 + k) % (1 << 60), dtype)
        gains.append(GainBlock(o, b, c, G))
    pairs = [(0, 1), (1, 0)] if len(grids) == 2 else [(0, 2), (2, 0), (1, 2), (2, 1), (2, 2)]
    losses = [LossBlock(a, b, 10.0 ** rng.uniform(*rng_g, size=(sizes[a], sizes[b])) * synth.loss_kappa(*rng_g, 1.0))
              for a, b in pairs]
    last, off = len(grids) - 1, ps.momentum_species_offset
    emi = EmissionMatrices()
    for s in range(last):  # the charged species radiate into the photons of their own cell
        E = 10.0 ** rng.uniform(*rng_g, size=(sizes[last], sizes[s])) * synth.emi_kappa(*rng_g, sizes[last], 1.0)
        emi.blocks += [EmiBlock(row0=k * n + off[last], col0=k * n + off[s], E=E) for k in range(cells)]
    torch.cuda.synchronize()  # the uploads read the gain blocks on the method's own stream
    inj = rng.uniform(0.0, 1e-6, ps.n_state)
    binm = BinaryMatrices(M_Bin=_csc_m_bin(ps, gains, losses)) if case["sparse"] else BinaryMatrices(gains=gains, losses=losses)
    return dict(ps=ps, flux=flux, gains=gains, losses=losses, emi=emi, inj=inj, binm=binm, rng=rng)


def _spectra(ps, rng, count):
    """Log-normal spectra, mean log p in U[-1, 1], with a little structure from cell to cell."""
    f = np.stack([synth.lognormal_f0(ps, [mu] * len(ps.name_list), 1.0) for mu in rng.uniform(-1.0, 1.0, count)])
    return f * rng.uniform(0.8, 1.2, f.shape)


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()


def _serve_requests(case, ps, rng):
    """Half again as many requests as slots, of 40 up to `steps` steps."""
    k = case["batch"] * 3 // 2
    return _spectra(ps, rng, k), rng.uniform(0.5, 1.0, k), rng.integers(min(40, case["steps"]), case["steps"] + 1, k)


# ---------------------------------------------------------------- prepare, run
def prepare(case, seed):
    kind = case["kind"]
    if kind == "serve":
        server, requests = Server(hbm_budget_bytes=150 << 30), []
        for g, grid in enumerate(_grids(case)):
            w = _workload(case, [grid, grid], 1, 2 * seed + g)
            requests.append(_serve_requests(case, w["ps"], w["rng"]))
            server.add_grid(BatchedEuler(w["ps"], w["inj"], w["binm"], w["emi"], w["flux"], case["batch"]))
        server.start()
        return dict(case=case, server=server, requests=requests)
    w = _workload(case, _grids(case), case["cells"], seed)
    ps = w["ps"]
    if kind == "batch":
        f0, dt = _spectra(ps, w["rng"], case["batch"]), w["rng"].uniform(0.5, 1.0, case["batch"])
        m = BatchedEuler(ps, w["inj"], w["binm"], w["emi"], w["flux"], case["batch"])
        for s in range(case["batch"]):
            m.admit(s, f0[s], float(dt[s]), 1 << 40)
        m.prepare()
        io = _pinned(f0.shape), _pinned(f0.shape)
        io[0][:] = f0
        return dict(case=case, m=m, f0=io[0], out=io[1])
    f0 = _spectra(ps, w["rng"], 1)[0]
    method = ForwardSymplecticEulerStruct if case["symplectic"] else ForwardEulerStruct
    m = method(ps, f0, w["inj"], w["binm"], w["emi"], w["flux"],
               Precision=np.float64 if case["precision"] == "f64" else np.float32)
    state = dict(case=case, m=m, f0=f0, scales=w["rng"].uniform(0.5, 1.0, case["steps"]))
    if kind == "run":
        m.prepare()
    if kind == "step_io":
        state["f0"], state["out"] = _pinned(f0.shape), _pinned(f0.shape)
        state["f0"][:] = f0
    if kind == "solve":
        state["t_save"] = _save_times(case)
        state["w"] = energy_weights(ps)
    return state


def _save_times(case):
    """`steps` steps of dt = 1 in whole intervals between the save points."""
    return [float(case["steps"] * k // case["saves"]) for k in range(case["saves"] + 1)]


def _kept(case, f):
    return f if case["precision"] == "f64" else f.astype(np.float32)


def run(state):
    case = state["case"]
    if case["kind"] == "serve":
        srv = state["server"]
        ids = [[srv.submit(g, f, float(dt), int(n)) for f, dt, n in zip(*r)] for g, r in enumerate(state["requests"])]
        return [_kept(case, np.stack([srv.wait(i)[0] for i in r])) for r in ids]
    m = state["m"]
    if case["kind"] == "batch":
        return _kept(case, m.run_io(state["f0"], case["steps"], state["out"]))
    if case["kind"] == "step_io":
        f, _, _ = m.step_io(state["f0"], 0.0, 1e9, float(state["scales"][0]), Verbose=1, out=state["out"])
        return {"f": _kept(case, f), "cr": m.last_diag.cr if case["precision"] == "f64" else np.float32(m.last_diag.cr)}
    if case["kind"] == "solve":
        o = Solve(m, 1.0, state["t_save"], Verbose=0, moment_weights=state["w"])
        f = np.stack(o.f)
        return {"f": _kept(case, f), "number": _kept(case, o.number), "energy": _kept(case, o.energy)}
    m.f = state["f0"]
    m.run(state["scales"])
    return _kept(case, m.f)


# ---------------------------------------------------------------- work, exact values
def work(case):
    grids = _grids(case)
    runs = [[g, g] for g in grids] if case["kind"] == "serve" else [grids]
    size = {"f64": 8, "f32": 4, "mixed": 4}[case["precision"]]
    by = fl = 0.0
    for gs in runs:
        ps = _phase_space(gs, case["cells"])
        n = ps.species_sizes
        blocks = [(0, 0, 1), (1, 0, 1)] if len(n) == 2 else [(0, 0, 2), (2, 0, 2), (1, 1, 2), (2, 1, 2), (0, 2, 2), (1, 2, 2)]
        elems = 0.0
        for o, b, c in blocks:
            elems += float(_energy_mask(ps, o).sum()) if case["sparse"] else float(n[o]) * n[b] * n[c]
        cols, steps = case["cells"] * max(1, case["batch"]), case["steps"]
        if case["kind"] == "serve":  # half again as many requests as slots, half the steps on average
            cols = cols * 1.5 * 0.5
        by += steps * elems * size + 16.0 * cols * sum(n) * (1 + case["saves"])
        fl += 2.0 * steps * elems * cols
    return {"bytes": by, "flops": fl}


class _Exact:
    """The step in 64 bits with torch, on the operators of a workload."""

    def __init__(self, w):
        d = dict(dtype=torch.float64, device="cuda")
        self.ps, self.w = w["ps"], w
        self.G = [(g.out_sp, g.in1_sp, g.in2_sp, torch.as_tensor(g.G).to("cuda")) for g in w["gains"]]
        if sum(x[3].numel() for x in self.G) <= 1 << 31:
            self.G = [(o, b, c, G.double()) for o, b, c, G in self.G]
        self.L = [(x.sp, x.other_sp, torch.tensor(x.L, **d)) for x in w["losses"]]
        self.E = [(x.row0, x.col0, torch.tensor(x.E, **d)) for x in w["emi"].blocks]
        self.P, self.X = (torch.tensor(M.toarray(), **d) for M in (w["flux"].P_Flux, w["flux"].X_Flux))
        self.inv, self.vol, self.inj = (torch.tensor(v, **d) for v in (1.0 / w["flux"].Ap_Flux, w["flux"].Vol, w["inj"]))

    def rates(self, f, with_x):
        """df of (instances, n_state) spectra before the scaling by invAp dt."""
        k, nm = f.shape[0], self.ps.n_momentum
        df = -(f @ (self.P + self.X if with_x else self.P).T)
        for r, c, E in self.E:
            df[:, r:r + E.shape[0]] += f[:, c:c + E.shape[1]] @ E.T
        cell = f.reshape(k * self.ps.n_space, nm)
        sl = [self.ps.species_slice(s) for s in range(len(self.ps.name_list))]
        bin_ = torch.zeros_like(cell)
        for o, b, c, G in self.G:
            x = (cell[:, sl[b], None] * cell[:, None, sl[c]]).reshape(cell.shape[0], -1)
            part = max(1, (1 << 28) // x.shape[1])
            for a in range(0, G.shape[0], part):
                g = G[a:a + part].reshape(-1, x.shape[1]).double()
                bin_[:, sl[o].start + a:sl[o].start + a + g.shape[0]] += x @ g.T
        for s, o, L in self.L:
            bin_[:, sl[s]] -= cell[:, sl[s]] * (cell[:, sl[o]] @ L.T)
        return df + (bin_.reshape(k, self.ps.n_space, nm) * self.vol[None, :, None]).reshape(k, -1)

    def step(self, f, dt, symplectic=False):
        """One step of every instance with its dt; returns f and Cr."""
        dt = torch.as_tensor(dt, dtype=torch.float64, device="cuda").reshape(-1, 1)
        df = self.rates(f, not symplectic) * (self.inv * dt)
        if symplectic:
            fm = f + df
            fm = torch.where(fm >= THR, fm, 0.0)
            fs = fm - (fm @ self.X.T) * (self.inv * dt)
            v = torch.where(fs >= THR_SPACE, fs, 0.0) + self.inj * dt
            return torch.where(v >= THR_SPACE, v, 0.0), None
        ratio = df / f
        cr = -torch.where(torch.isnan(ratio), math.inf, ratio).min()
        v = f + (df + self.inj * dt)
        return torch.where(v >= THR, v, 0.0), float(cr)


def _host(f):
    return f.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "serve":
        outs = []
        for g, grid in enumerate(_grids(case)):
            w = _workload(case, [grid, grid], 1, 2 * seed + g)
            f0, dt, n = _serve_requests(case, w["ps"], w["rng"])
            e, f = _Exact(w), torch.tensor(f0, device="cuda")
            dt, n = torch.tensor(dt, device="cuda"), torch.tensor(n, device="cuda")
            for k in range(int(n.max())):
                f = torch.where((n > k)[:, None], e.step(f, dt)[0], f)
            outs.append(_host(f))
        return outs
    w = _workload(case, _grids(case), case["cells"], seed)
    if kind == "batch":
        f, dt = _spectra(w["ps"], w["rng"], case["batch"]), w["rng"].uniform(0.5, 1.0, case["batch"])
        e, f = _Exact(w), torch.tensor(f, device="cuda")
        for _ in range(case["steps"]):
            f = e.step(f, dt)[0]
        return _host(f)
    f0 = _spectra(w["ps"], w["rng"], 1)
    scales = w["rng"].uniform(0.5, 1.0, case["steps"])
    e, f = _Exact(w), torch.tensor(f0, device="cuda")
    if kind == "step_io":
        f, cr = e.step(f, scales[0])
        return {"f": _host(f)[0], "cr": cr}
    if kind == "solve":
        ps, wt = w["ps"], torch.tensor(energy_weights(w["ps"]), device="cuda")
        saves, marks = [f], _save_times(case)[1:]
        for k in range(case["steps"]):
            f = e.step(f, 1.0)[0]
            saves += [f] * marks.count(float(k + 1))
        F = torch.cat(saves)
        sl = [ps.species_slice(s) for s in range(len(ps.name_list))]
        return {"f": _host(F), "number": _host(torch.stack([F[:, s].sum(1) for s in sl], 1))[:, None, :],
                "energy": _host(torch.stack([(F[:, s] * wt[s]).sum(1) for s in sl], 1))[:, None, :]}
    for dt in scales:
        f = e.step(f, dt, case["symplectic"])[0]
    return _host(f)[0]
