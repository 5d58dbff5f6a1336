"""The split sums of the mass and momentum reductions on cells that leave no room for rounding: many
populations whose part between 2^-22 and 2^-42 is as large as it can be, the others near 1e-6.  Every
population is a multiple of 2^-43 and every sum below 2^10, so float64 holds each sum exactly, and the
reductions have to return it exactly."""
from __future__ import annotations

import ctypes as C
from fractions import Fraction

import numpy as np
import pytest
import torch

from mojo_lbm_gb300 import LBM_Config, LBM_method, _capi
from mojo_lbm_gb300.solver import Solver
from tests.lbm_cases import make_grid
from tests.test_gpu_step import to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sign", [1, -1])
@pytest.mark.parametrize("lat,shape", [("D2Q9", (31, 17, 1)), ("D3Q19", (9, 8, 7)), ("D3Q27", (9, 8, 7))])
def test_sums_are_exact(lat, shape, sign):
    grid = make_grid(lat, shape, "untiled")
    cfg = LBM_Config(LBM_method.DOUBLE_BUFFER)
    rng = np.random.default_rng(grid.Q)
    N, Q = grid.num_points, grid.Q
    # below 2^-6, where float32 steps by 2^-30: the low part just under 2^-22 is kept
    f = rng.integers(64, 20000, (Q, N)) * 2.0 ** -21 + sign * (2.0 ** -22 - 2.0 ** -30)
    tiny = rng.random((Q, N)) < rng.random(N) * 0.3
    f[tiny] = rng.integers(2 ** 23, 2 ** 24, int(tiny.sum())) * 2.0 ** -43
    f = f.astype(np.float32)
    assert np.all(f.astype(np.float64) * 2.0 ** 43 == np.rint(f.astype(np.float64) * 2.0 ** 43))
    c = np.concatenate([np.ones((1, Q), np.int64), grid.lattice.directions[:, :grid.D].T.astype(np.int64)])
    units = (f.astype(np.float64) * 2.0 ** 43).astype(np.int64)
    want = [float(Fraction(int((c[k][:, None] * units).sum()), 2 ** 43)) for k in range(grid.D + 1)]
    flags = torch.zeros(N, dtype=torch.uint8, device="cuda")
    fd = to_dev(np.ascontiguousarray(f).reshape(-1))  # untiled: [Q][cells]
    got = Solver(grid, cfg).mass_momentum(fd, flags)
    out, cc, g = (C.c_double * 4)(), cfg.to_c(), grid.to_c()
    _capi.check(_capi.lib().lbm_reduce_mass_momentum_noalloc(C.byref(cc), C.byref(g), fd.data_ptr(), flags.data_ptr(), 0,
                                                             out, None))
    assert list(got[:grid.D + 1]) == want and list(out[:grid.D + 1]) == want
