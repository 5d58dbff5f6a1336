"""The block-per-tile kernels whose thread blocks own half a tile, against the generic kernel."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from mojo_lbm_gb300 import Flags, LBM_Config, LBM_method
from mojo_lbm_gb300.solver import Solver
from tests.lbm_cases import initial_f, make_grid, mixed_flags
from tests.test_gpu_step import to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lat,shape,tile", [("D2Q9", (32, 8, 1), (32, 8, 1)), ("D2Q9", (16, 48, 1), (16, 16, 1)),
                                            ("D3Q19", (8, 8, 4), (8, 8, 4)), ("D3Q19", (2, 48, 16), (1, 16, 16)),
                                            ("D3Q27", (64, 4, 2), (64, 2, 2)), ("D3Q27", (16, 8, 12), (16, 4, 4))])
@pytest.mark.parametrize("method", [LBM_method.DOUBLE_BUFFER, LBM_method.ESOTERIC_PULL])
@pytest.mark.parametrize("store,coll,les", [("fp32", "SRT", False), ("f16c", "TRT", True), ("fp32", "RLBM", True),
                                            ("f16c", "KBC", False)])
def test_half_tile_blocks_equal_generic(lat, shape, tile, method, store, coll, les):
    """Grids of one to six tiles with flags of every kind: populations and captures equal the generic
    kernel's bit for bit, in single steps of both parities and replayed ones."""
    grid = make_grid(lat, shape, tile)
    rng = np.random.default_rng(7)
    f16 = store == "f16c"
    cfg = LBM_Config(method, collision_op=coll, LES=les, BCs={Flags.EQUILIBRIUM}, DDF_shift=f16, use_float16c=f16,
                     capture_density=True, capture_velocity=True)
    flags, bc = mixed_flags(grid, rng)
    f0, bc, fl = initial_f(grid, cfg, rng), np.nan_to_num(bc, nan=0.01), to_dev(flags)
    out = []
    for path in (1, 2):
        s = Solver(grid, cfg)
        s.set_kernel_path(path)
        a, bcd = to_dev(f0), to_dev(bc)
        eso = method == LBM_method.ESOTERIC_PULL
        b = None if eso else a.clone()
        for k in range(2):
            if eso:
                s.esoteric_pull_step(a, bcd, fl, 0.6, k % 2 == 0)
            else:
                s.double_buffer_step(*((b, a) if k % 2 == 0 else (a, b)), bcd, fl, 0.6)
        s.run(a, b, bcd, fl, 0.6, 5, 2)
        out.append((a, bcd) if eso else (a, bcd, b))
    for x, y in zip(*out):
        w = torch.int16 if x.dtype == torch.int16 else torch.int32
        assert torch.equal(x.view(w), y.view(w))
