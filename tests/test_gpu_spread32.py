"""The FP32 spread in each of its splits of a tile over CTAs: grids on both sides of the lines
between them, a few beads and many, and clusters that fill several lists and stages. Against
the FP64 spread (itself against the oracle in test_gpu_fcm.py) with that file's bar for the
two precisions; the sums do not depend on how many beads are staged at a time."""
import ctypes

import numpy as np
import pytest

from filsim_b200 import abi
from filsim_b200.configs import params_for
from filsim_b200.fcm import Context, Fcm
from test_gpu_fcm import FP32_SPREAD_REL, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,nb,ngd,clump", [
    ((64, 64, 144), 700, 12, 1.0),       # 144 tiles: quarter tiles
    ((64, 64, 144), 700, 20, 0.2),
    ((64, 64, 160), 1, 12, 1.0),         # 160: half tiles
    ((64, 64, 160), 1500, 13, 0.2),
    ((192, 192, 144), 3000, 12, 1.0),    # 1,296 and 1,584 tiles: half, whole
    ((192, 192, 176), 3000, 12, 1.0),
    ((192, 192, 176), 3000, 14, 0.1),    # whole tiles with several lists
    ((192, 192, 176), 17000, 12, 1.0),   # too dense for whole tiles
    ((320, 320, 320), 2000, 12, 1.0),    # 8,000 and 8,400 tiles: whole, by four warps
    ((320, 320, 336), 2000, 12, 1.0),
    ((320, 320, 336), 2000, 17, 0.05),   # the same with several lists
])
def test_matches_fp64_in_every_split(gpu_lib, dims, nb, ngd, clump):
    p = params_for(dims, ngd=ngd)
    rng = np.random.default_rng(nb + ngd)
    L = np.array(dims) * p.dx
    Y = np.fmod(rng.uniform(-1.0, 1.0, (nb, 3)) * L * clump, L)
    F, T = rng.standard_normal((nb, 3)), rng.standard_normal((nb, 3))
    ctx = Context(p, max_beads=nb, max_filaments=nb)
    fcm = Fcm(ctx, nb)
    fcm.set(Y, F, T)
    want = fcm.spread().cpu().numpy()
    ctx.set_precision(abi.FS_PREC_FP32)
    for cols in (2, 4, 8):
        got = []
        for chunk in (32, 64):
            tune = np.array([chunk, 8, 0, cols], np.int32)
            abi.check(abi.lib().fs_set_tuning(ctx.h, tune.ctypes.data_as(ctypes.c_void_p)), "fs_set_tuning")
            got.append(fcm.spread().cpu().numpy())
        assert rel_err(got[0], want) < FP32_SPREAD_REL, cols
        assert np.array_equal(got[0], got[1]), cols
    ctx.close()
