"""Stepping calls captured into a graph of the caller's, in turn with direct calls: whatever the order of
captures, replays, runs and rewritten boundary values, every call gives the words of the same steps taken
one by one by a solver that is never captured."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from mojo_lbm_gb300 import Flags, LBM_Config, LBM_method
from mojo_lbm_gb300.batch import BatchSolver
from mojo_lbm_gb300.solver import Solver
from tests.lbm_cases import initial_f, make_grid, mixed_flags
from tests.test_gpu_step import to_dev
from tests.test_gpu_walls import _bc, _one_by_one

pytestmark = pytest.mark.gpu

# r: a direct run of that many steps, c: the same captured (not replayed), p: a replay of the last capture.
# 40 steps is long enough for masks without the walls at rest.  The boundary values are rewritten before
# every r and p.
ORDERS = ["r40 c10 p r2 r40 p r2", "c10 r2 p r40 p r2 p", "r64 c16 r16 r2 p", "r2 c40 r10 p r10 p", "c40 p r40 c2 p p r2",
          "r40 c40 r40 p r2 p r64"]
REST = [0.7, 1.0, 0.0, 0.5, 0.2]  # the share of the walls at rest, cycled through


def _play(order, run, new_bc, check):
    side, graph = torch.cuda.Stream(), None
    for k, op in enumerate(order.split()):
        n = int(op[1:] or 0)
        if op[0] == "c":
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=side):
                run(n, torch.cuda.current_stream())
            captured = n
            continue
        new_bc(REST[k % len(REST)])
        if op[0] == "p":
            graph.replay()
            n = captured
        else:
            run(n, None)
        torch.cuda.synchronize()
        check(n, f"{op} at {k}")


@pytest.mark.parametrize("order", ORDERS)
@pytest.mark.parametrize("meth,f16", [("db", False), ("eso", True)])
@pytest.mark.parametrize("lat,shape,tile", [("D2Q9", (32, 48, 1), (16, 16, 1)), ("D3Q19", (16, 16, 12), (8, 8, 4)),
                                            ("D3Q19", (11, 9, 7), "untiled")])
def test_captured_runs_equal_single_steps(lat, shape, tile, meth, f16, order):
    grid = make_grid(lat, shape, tile)
    m = LBM_method.DOUBLE_BUFFER if meth == "db" else LBM_method.ESOTERIC_PULL
    cfg = LBM_Config(m, BCs={Flags.EQUILIBRIUM}, DDF_shift=f16, use_float16c=f16)
    rng = np.random.default_rng(grid.num_points)
    flags, _ = mixed_flags(grid, rng)
    f0 = initial_f(grid, cfg, rng)
    fl, bc = to_dev(flags), to_dev(_bc(grid, rng, 0.7))
    a1, b1, a2, b2 = (to_dev(f0) for _ in range(4))
    s, ref = Solver(grid, cfg), Solver(grid, cfg)
    word = torch.int16 if f16 else torch.int32

    def check(n, what):
        _one_by_one(ref, cfg, a2, b2, bc, fl, 0.8, n)
        assert torch.equal(a1.view(word), a2.view(word)) and torch.equal(b1.view(word), b2.view(word)), what

    _play(order, lambda n, stream: s.run(a1, b1, bc, fl, 0.8, n, 0, stream),
          lambda rest: bc.copy_(torch.from_numpy(_bc(grid, rng, rest))), check)


@pytest.mark.parametrize("order", [o for o in ORDERS if o[0] == "r"])
def test_captured_batch_runs_equal_single_steps(order):
    """(The first run of a batch uploads its descriptors and cannot be captured.)"""
    grids = [make_grid("D2Q9", (32, 16 * k, 1), (16, 16, 1)) for k in (1, 3, 2)]
    cfg = LBM_Config(LBM_method.DOUBLE_BUFFER, BCs={Flags.EQUILIBRIUM})
    rng = np.random.default_rng(7)
    batch = BatchSolver(grids, cfg)
    doms = []
    for i, g in enumerate(grids):
        flags, _ = mixed_flags(g, rng)
        f0 = initial_f(g, cfg, rng)
        d = dict(grid=g, solver=Solver(g, cfg), fl=to_dev(flags), bc=to_dev(_bc(g, rng, 0.6)),
                 f=[to_dev(f0) for _ in range(4)])
        batch.set_domain(i, d["f"][0], d["f"][1], d["bc"], d["fl"], 0.8)
        doms.append(d)

    def new_bc(rest):
        for d in doms:
            d["bc"].copy_(torch.from_numpy(_bc(d["grid"], rng, rest)))

    def check(n, what):
        for d in doms:
            _one_by_one(d["solver"], cfg, d["f"][2], d["f"][3], d["bc"], d["fl"], 0.8, n)
            for k in (0, 1):
                assert torch.equal(d["f"][k].view(torch.int32), d["f"][2 + k].view(torch.int32)), what

    _play(order, lambda n, stream: batch.run(n, 0, stream), new_bc, check)
