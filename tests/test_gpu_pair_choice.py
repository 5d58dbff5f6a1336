"""Which kernel the automatic choice takes for the in-place method in the fast arithmetic on grids of at
least 2432 tiles: the cell-pair kernel where it is built to be, the per-cell one elsewhere (so that the
comparison of the two in test_gpu_pair_inplace.py has two kernels to compare)."""
from __future__ import annotations

import pytest

from mojo_lbm_gb300 import LBM_Config, LBM_method
from mojo_lbm_gb300.solver import Solver
from tests.lbm_cases import make_grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lat,shape,tile", [("D2Q9", (784, 800, 1), (16, 16, 1)), ("D3Q19", (96, 88, 80), (8, 8, 4)),
                                            ("D3Q27", (96, 88, 80), (8, 8, 4)), ("D3Q19", (64, 96, 112), (2, 16, 8))])
@pytest.mark.parametrize("f16", [False, True])
@pytest.mark.parametrize("coll", ["SRT", "TRT", "KBC", "RLBM"])
@pytest.mark.parametrize("les", [False, True])
def test_in_place_choice(lat, shape, tile, f16, coll, les):
    def path(arith, sh=shape):
        cfg = LBM_Config(LBM_method.ESOTERIC_PULL, collision_op=coll, LES=les, DDF_shift=f16, use_float16c=f16,
                         arithmetic=arith)
        return Solver(make_grid(lat, sh, tile), cfg).kernel_path

    pairs = {"D2Q9": coll != "KBC" or f16, "D3Q19": True, "D3Q27": f16 and coll != "KBC"}[lat]
    assert path("fast") == (3 if pairs else 2)
    assert path("exact") == 2
    assert path("fast", tuple(t * (1 if t == 1 else 4) for t in tile)) == 2  # few tiles
