"""The FP32 spread on both sides of the lines between its splits of a tile over CTAs: 2, 10 and 40
tiles per SM, and 12, 20, 28 and 48 beads reaching a tile, also with clusters that fill several lists.
Against the FP64 spread, with the bar of test_gpu_spread32.py."""
import numpy as np
import pytest
import torch

from filsim_b200 import abi
from filsim_b200.configs import params_for
from filsim_b200.fcm import Context, Fcm
from test_gpu_fcm import FP32_SPREAD_REL, rel_err

pytestmark = pytest.mark.gpu


# grids of n x 4 x 4 tiles; 12-point stencils reach (27 / 16)^3 = 4.8 tiles
@pytest.mark.parametrize("per_sm,reach", [(2, 20), (10, 12), (10, 48), (40, 28)])
@pytest.mark.parametrize("more_tiles", [False, True])
@pytest.mark.parametrize("more_beads", [False, True])
@pytest.mark.parametrize("clump", [1.0, 0.08])
def test_matches_fp64_at_the_lines(gpu_lib, per_sm, reach, more_tiles, more_beads, clump):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = -(-per_sm * sms // 16) - (0 if more_tiles else 1)
    dims = (16 * n, 64, 64)
    nb = int(16 * n * reach / (27 / 16) ** 3) + (1 if more_beads else -1)
    p = params_for(dims)
    rng = np.random.default_rng(n + reach)
    Y = rng.uniform(0.0, 1.0, (nb, 3)) * np.array(dims) * p.dx * [clump, 1.0, 1.0]
    ctx = Context(p, max_beads=nb, max_filaments=nb)
    fcm = Fcm(ctx, nb)
    fcm.set(Y, rng.standard_normal((nb, 3)), rng.standard_normal((nb, 3)))
    want = fcm.spread().cpu().numpy()
    ctx.set_precision(abi.FS_PREC_FP32)
    assert rel_err(fcm.spread().cpu().numpy(), want) < FP32_SPREAD_REL
    ctx.close()
