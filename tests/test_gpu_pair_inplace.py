"""The cell-pair kernel of the in-place method (fast arithmetic, large grids), against the per-cell kernel."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from mojo_lbm_gb300 import Flags, LBM_Config, LBM_method
from mojo_lbm_gb300.solver import Solver
from tests.lbm_cases import initial_f, make_grid, mixed_flags
from tests.test_gpu_step import to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lat,shape,tile", [("D2Q9", (784, 800, 1), (16, 16, 1)), ("D3Q19", (96, 88, 80), (8, 8, 4)),
                                            ("D3Q27", (96, 88, 80), (8, 8, 4)), ("D3Q19", (64, 96, 112), (2, 16, 8))])
@pytest.mark.parametrize("store", ["fp32", "f16c"])
@pytest.mark.parametrize("coll,les", [("SRT", False), ("SRT", True), ("TRT", True), ("KBC", False), ("KBC", True),
                                      ("RLBM", True)])
def test_in_place_pair_equals_tile(lat, shape, tile, store, coll, les):
    """The in-place method in the fast arithmetic, which the automatic choice steps two cells per thread
    on grids of at least 2432 tiles: populations and captures equal the per-cell kernel's word for
    word, in single steps of both parities and graph-replayed ones, next to flags of every kind; buffers
    that are not 8-byte aligned run the per-cell kernel."""
    grid = make_grid(lat, shape, tile)
    assert grid.num_points // 256 >= 2432
    rng = np.random.default_rng(5)
    f16 = store == "f16c"
    cfg = LBM_Config(LBM_method.ESOTERIC_PULL, collision_op=coll, LES=les, BCs={Flags.EQUILIBRIUM}, DDF_shift=f16,
                     use_float16c=f16, capture_density=True, capture_velocity=True, arithmetic="fast")
    flags, bc = mixed_flags(grid, rng)
    flags[rng.random(flags.size) < 0.97] = 0
    f0 = initial_f(grid, cfg, rng)
    bc = np.nan_to_num(bc, nan=0.01)
    fl = to_dev(flags)
    out = []
    for path, shift in ((0, 0), (2, 0), (0, 1)):
        s = Solver(grid, cfg)
        s.set_kernel_path(path)
        src = to_dev(f0)
        buf = torch.zeros(src.numel() + 1, dtype=src.dtype, device="cuda")
        a, bcd = buf[shift:shift + src.numel()], to_dev(bc)
        a.copy_(src)
        for k in range(3):
            s.esoteric_pull_step(a, bcd, fl, 0.6, k % 2 == 0)
        s.run(a, None, bcd, fl, 0.6, 65, 3)
        out.append((a.clone(), bcd, s.kernel_path))
    word = torch.int16 if f16 else torch.int32
    for o in out[1:]:
        assert torch.equal(out[0][0].view(word), o[0].view(word))
        assert torch.equal(out[0][1].view(torch.int32), o[1].view(torch.int32))
    assert out[1][2] == 2
