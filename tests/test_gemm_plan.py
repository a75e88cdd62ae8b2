"""The bound on what one FP32 accumulator of the batched gain GEMM sums (16 K tiles on one SM, 32 on SM
pairs), over the plans the autotuner may choose and those a cache file may bring. The rule is host
arithmetic (csrc/gemm_plan.h), compiled here into a small program."""
import os
import subprocess

import numpy as np
import pytest

import oracle
from dtb import synth
from dtb.batch import BatchedEuler, set_tune_cache

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "diplodocustransport.jl_b200", "csrc")
PROGRAM = r"""
#include <cstdio>
#include <cstring>
#include "gemm_plan.h"
using namespace dtb;
// per line "m_tiles n_cb N1 cols pair bn splits": the plan's tiles per accumulator, the fill's,
// whether it is valid, then every candidate of the shape as pair:bn:splits:tiles
int main() {
    GemmShape g{0, 0, 0, 0, 148, 72};
    GemmPlan p;
    while (std::scanf("%d %d %d %d %d %d %d", &g.m_tiles, &g.n_cb, &g.N1, &g.cols, &p.pair, &p.bn, &p.splits) == 7) {
        std::printf("%d %d", gemm_tiles_per_acc(g, p), (int)gemm_plan_valid(g, p));
        for (const GemmPlan& q : gemm_plan_candidates(g)) {
            GemmPlan f = q;
            f.splits = gemm_fill_splits(g, q.pair, q.bn);
            std::printf(" %d:%d:%d:%d:%d", q.pair, q.bn, q.splits, gemm_tiles_per_acc(g, q), gemm_tiles_per_acc(g, f));
        }
        std::printf("\n");
    }
}
"""


@pytest.fixture(scope="module")
def plans(tmp_path_factory):
    d = tmp_path_factory.mktemp("gemm_plan")
    (d / "p.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, str(d / "p.cpp"), "-o", str(d / "p")], check=True)

    def ask(lines):
        out = subprocess.run([str(d / "p")], input="\n".join(" ".join(map(str, x)) for x in lines) + "\n", text=True,
                             capture_output=True, check=True).stdout.splitlines()
        return [ln.split() for ln in out]
    return ask


def _shape(rows, n1, n2, cols):
    return (rows + 127) // 128, (n2 + 63) // 64, n1, cols


# two species of equal size, three interactions on three, uneven ones; few to many columns
SHAPES = [_shape(2 * n, n, n, c) for n in (32, 96, 128, 150, 180, 192, 200, 256, 320, 384, 512, 576, 1024)
          for c in (4, 24, 64, 72, 100, 128, 192, 256, 260, 512, 768)]
SHAPES += [_shape(3 * n, n, n, c) for n in (85, 128, 256, 576) for c in (8, 64, 128, 300)]
SHAPES += [_shape(258, 160, 98, 72), _shape(640, 128, 512, 256), _shape(520, 8, 512, 64), _shape(100, 90, 10, 32)]


def test_candidates_respect_the_accumulator_bound(plans):
    kinds = set()
    for shape, row in zip(SHAPES, plans([s + (0, 64, 1) for s in SHAPES])):
        assert len(row) > 2
        for c in row[2:]:
            pair, bn, splits, tiles, fill_tiles = map(int, c.split(":"))
            kinds.add((pair, bn, tiles <= fill_tiles))
            assert splits >= 1
            # past the bound only as the plan that fills the device, where its waves are capped
            assert tiles <= max(32 if pair else 16, fill_tiles), (shape, c)
    assert {k[:2] for k in kinds} == {(0, 64), (0, 128), (0, 256), (1, 256)}
    assert (0, 64, False) in kinds  # fewer splits than the fill are still tried within the bound


def test_plans_past_the_bound_are_refused(plans):
    wide = _shape(360, 180, 180, 256)  # 540 K tiles, three m tiles: one accumulator with 256-wide tiles
    got = plans([wide + (0, 256, 49), wide + (0, 256, 24), wide + (0, 128, 24), wide + (0, 256, 0), wide + (1, 256, 40),
                 _shape(256, 128, 128, 260) + (1, 256, 13), _shape(256, 128, 128, 260) + (1, 256, 5)])
    assert [(int(r[0]), r[1] == "1") for r in got] == [(12, True), (23, False), (8, True), (540, False), (14, False),
                                                       (20, True), (52, False)]


@pytest.mark.gpu
def test_cached_plan_past_the_bound_is_measured_afresh(cuda, tmp_path):
    """A cache line whose accumulators would sum 24 K tiles on one SM (2 x 192 states, 256 slots, three m
    tiles, 24 splits): the context times its own plan, within the bound, and steps to 1e-5 (relative
    L-inf, the batched path's tolerance) of the FP64 oracle."""
    import torch
    B = 256
    w = synth.batched_two_species(24, 1e-2, 1e2, 8, B, seed=31)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    cache = tmp_path / "plans.txt"
    cache.write_text(f"sm{sms}:M384:N1192:n2192:cols{B}:cells1 0 256 24 30.0\n")
    set_tune_cache(str(cache))
    try:
        m = BatchedEuler(w.ps, w.inj, w.binm, w.emim, w.fluxm, B)
    finally:
        set_tune_cache(None)
    p = m.gemm_plan(0)
    per_acc = 192 * 3 / p["n_splits"] / (1 if p["pair"] else 512 // p["bn"] - 1)
    assert p["tuned_us"] > 0 and per_acc <= (32 if p["pair"] else 16)
    assert len(cache.read_text().splitlines()) == 2
    for i in range(B):
        m.admit(i, w.f0[i], w.dt[i], 10)
    m.run(10)
    ops = oracle.blocked_from_workload(w)
    for i in (0, 100, B - 1):
        f = w.f0[i].copy()
        for _ in range(10):
            f, _, _ = ops.step(f, float(w.dt[i]), 0)
        assert np.max(np.abs(m.get_f(i) - f)) / np.max(np.abs(f)) <= 1e-5
    m.close()


@pytest.mark.gpu
def test_plans_belong_to_their_epilogue(cuda, tmp_path):
    """Two grids with equal gain blocks and different epilogues (one without emission) are timed each for
    itself: a cache line each, with its epilogue in the last field. A third context takes the plan of the
    first's line, a line without that field serves both."""
    B = 40
    w = synth.batched_two_species(16, 1e-2, 1e2, 8, B, seed=32)
    cache = tmp_path / "plans.txt"

    def commit(emission):
        from dtb.structs import EmissionMatrices
        m = BatchedEuler(w.ps, w.inj, w.binm, w.emim if emission else EmissionMatrices(), w.fluxm, B)
        p = m.gemm_plan(0)
        m.close()
        return p

    set_tune_cache(str(cache))
    try:
        plans = [commit(True), commit(False), commit(True)]
        lines = [ln.split() for ln in cache.read_text().splitlines()]
        assert len(lines) == 2 and all(len(ln) == 6 for ln in lines)
        assert lines[0][0] == lines[1][0] and lines[0][5] != lines[1][5]
        assert plans[2] == plans[0]
        # the recorded lines seed a new table; a line of the shape alone serves every epilogue
        key = lines[0][0]
        for text, plan in ((" ".join([key, "0", "64", "40", "7.0", lines[0][5]]), (False, 64, 40)),
                           (f"{key} 0 64 36 7.0", (False, 64, 36))):
            cache.write_text(text + "\n")
            set_tune_cache(str(cache))
            got = commit(True)
            assert (got["pair"], got["bn"], got["n_splits"]) == plan
        assert commit(False)["n_splits"] == 36
    finally:
        set_tune_cache(None)
