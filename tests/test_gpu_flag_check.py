"""Flags that change between calls on the tiled layouts: the one-launch check that follows the first build
of the masks rebuilds a changed tile and those around it.  A handle that has seen every change must step
as one that is created for the new flags: isolated flags that come and go at the faces, edges and
corners of tiles and of the grid, one tile and several tiles per block, one or two tiles along an axis,
and a flag buffer that is not 16-byte aligned."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from mojo_lbm_gb300 import Flags, LBM_Config, LBM_method
from mojo_lbm_gb300.solver import Solver
from tests.lbm_cases import initial_f, make_grid

pytestmark = pytest.mark.gpu

GRIDS = [("D2Q9", (48, 32, 1), (16, 16, 1)), ("D2Q9", (16, 32, 1), (16, 16, 1)), ("D2Q9", (800, 800, 1), (16, 16, 1)),
         ("D3Q19", (24, 16, 12), (8, 8, 4)), ("D3Q19", (96, 96, 80), (8, 8, 4)), ("D3Q27", (32, 8, 16), (16, 4, 4))]


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("meth", ["db", "eso"])
@pytest.mark.parametrize("lat,shape,tile", GRIDS)
def test_masks_follow_isolated_changes(lat, shape, tile, meth, shift):
    grid = make_grid(lat, shape, tile)
    N = grid.num_points
    m = LBM_method.DOUBLE_BUFFER if meth == "db" else LBM_method.ESOTERIC_PULL
    cfg = LBM_Config(m, BCs={Flags.EQUILIBRIUM})
    rng = np.random.default_rng(N)
    lay = grid.layouts
    f0 = torch.from_numpy(initial_f(grid, cfg, rng)).cuda()
    bc = torch.zeros(N * (grid.D + 1), device="cuda")
    bcv = np.zeros(N * (grid.D + 1), np.float32)
    bcv[(np.arange(bcv.size) // lay.T) % (grid.D + 1) == grid.D] = 1.0
    bcv[(np.arange(bcv.size) // lay.T) % (grid.D + 1) == 0] = 0.02
    bc.copy_(torch.from_numpy(bcv))
    buf = torch.zeros(N + 1, dtype=torch.uint8, device="cuda")
    fl = buf[shift:shift + N]
    kept = Solver(grid, cfg)
    kept.set_kernel_path(2)
    edge = [np.array(sorted({0, n - 1, t - 1, t % n, n // t // 2 * t % n})) for n, t in zip(shape, tile)]
    host = np.zeros(N, np.uint8)
    for k in range(8):
        if k == 4:
            host[:] = 0
        for _ in range(4):
            x, y, z = (int(rng.choice(e)) for e in edge)
            at = int(lay.flag_offset(x, y, z))
            host[at] = 0 if host[at] else int(rng.choice([Flags.SOLID, Flags.EQUILIBRIUM, Flags.EXCLUDE]))
        fl.copy_(torch.from_numpy(host))
        fresh = Solver(grid, cfg)
        fresh.set_kernel_path(2)
        out = []
        for s in (kept, fresh):
            a, b = f0.clone(), f0.clone()
            if meth == "eso":
                s.esoteric_pull_step(a, bc, fl, 0.8, True)
            else:
                s.double_buffer_step(b, a, bc, fl, 0.8)
            out.append(a if meth == "eso" else b)
        assert torch.equal(out[0].view(torch.int32), out[1].view(torch.int32)), f"change {k}"
        fresh.close()
