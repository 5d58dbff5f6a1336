"""Walls at rest in multi-step runs: a run of many steps builds its masks without the walls whose
moving-wall term is exactly zero (lbm_run, lbm_batch_run) and must give the words of the same steps taken
one by one, whose masks come from the flags alone: with walls at rest and moving, components that cancel,
bc values rewritten between runs, runs and single steps in turn, and another stream."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from mojo_lbm_gb300 import Flags, LBM_Config, LBM_method
from mojo_lbm_gb300.batch import BatchSolver
from mojo_lbm_gb300.solver import Solver
from tests.lbm_cases import initial_f, make_grid, mixed_flags
from tests.test_gpu_step import to_dev

pytestmark = pytest.mark.gpu

GRIDS = [("D2Q9", (32, 48, 1), (16, 16, 1)), ("D3Q19", (16, 16, 12), (8, 8, 4)), ("D3Q27", (8, 16, 8), (8, 8, 4)),
         ("D3Q19", (11, 9, 7), "untiled")]
RUN = 40  # steps of a run long enough for such masks


def _bc(grid, rng, rest):
    """Boundary values [components, cells] in the tiled layout: a share of the walls at rest, some whose
    components cancel along a diagonal, the others moving."""
    lay, N, D = grid.layouts, grid.num_points, grid.D
    v = rng.uniform(-0.05, 0.05, (D + 1, N)).astype(np.float32)
    v[D] = rng.uniform(0.97, 1.03, N)
    v[:D, rng.random(N) < rest] = 0.0
    v[:D, rng.random(N) < 0.1] = np.float32(0.03)
    n = np.arange(N)
    out = np.empty(N * (D + 1), np.float32)
    for k in range(D + 1):
        out[n % lay.T + lay.T * (k + (D + 1) * (n // lay.T))] = v[k]
    return out


def _one_by_one(s, cfg, a, b, bc, fl, tau, n):
    for k in range(n):
        if cfg.lbm_method == LBM_method.ESOTERIC_PULL:
            s.esoteric_pull_step(a, bc, fl, tau, k % 2 == 0)
        elif k % 2 == 0:
            s.double_buffer_step(b, a, bc, fl, tau)
        else:
            s.double_buffer_step(a, b, bc, fl, tau)


@pytest.mark.parametrize("path", [0, 1, 3])
@pytest.mark.parametrize("meth,f16,coll", [("db", False, "SRT"), ("db", True, "TRT"), ("eso", True, "SRT"),
                                           ("eso", False, "RLBM")])
@pytest.mark.parametrize("lat,shape,tile", GRIDS)
def test_runs_equal_single_steps(lat, shape, tile, meth, f16, coll, path):
    if path == 3 and (meth == "eso" or tile == "untiled"):
        pytest.skip("the cell-pair kernel is double-buffer, 256-cell tiles")
    grid = make_grid(lat, shape, tile)
    m = LBM_method.DOUBLE_BUFFER if meth == "db" else LBM_method.ESOTERIC_PULL
    cfg = LBM_Config(m, collision_op=coll, BCs={Flags.EQUILIBRIUM}, DDF_shift=f16, use_float16c=f16)
    rng = np.random.default_rng(grid.num_points + path)
    flags, _ = mixed_flags(grid, rng)
    f0 = initial_f(grid, cfg, rng)
    f0[rng.random(f0.size) < 0.02] = 0x8000 if f16 else -0.0
    fl = to_dev(flags)
    run, ref = Solver(grid, cfg), Solver(grid, cfg)
    for s in (run, ref):
        s.set_kernel_path(path)
    a1, b1, a2, b2 = (to_dev(f0) for _ in range(4))
    bc = to_dev(_bc(grid, rng, 0.7))
    side = torch.cuda.Stream()
    for k, (n, rest, stream) in enumerate([(RUN, 0.7, None), (RUN, 1.0, None), (2, 0.0, None), (RUN, 0.0, None),
                                           (RUN, 0.7, side), (4, 0.2, None), (RUN, 0.5, None)]):
        bc.copy_(torch.from_numpy(_bc(grid, rng, rest)))
        if stream is not None:
            torch.cuda.synchronize()
        run.run(a1, b1, bc, fl, 0.8, n, 0, stream)
        _one_by_one(ref, cfg, a2, b2, bc, fl, 0.8, n)
        torch.cuda.synchronize()
        word = torch.int16 if f16 else torch.int32
        assert torch.equal(a1.view(word), a2.view(word)) and torch.equal(b1.view(word), b2.view(word)), f"part {k}"


def test_batch_runs_equal_single_steps():
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
    for n, rest in ((RUN, 0.6), (RUN, 1.0), (2, 0.1), (RUN, 0.3)):
        for d in doms:
            d["bc"].copy_(torch.from_numpy(_bc(d["grid"], rng, rest)))
        batch.run(n, 0)
        for d in doms:
            _one_by_one(d["solver"], cfg, d["f"][2], d["f"][3], d["bc"], d["fl"], 0.8, n)
            assert torch.equal(d["f"][0].view(torch.int32), d["f"][2].view(torch.int32))
            assert torch.equal(d["f"][1].view(torch.int32), d["f"][3].view(torch.int32))
