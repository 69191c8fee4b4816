"""The scale of the line transforms' projection, 1 / (q^2 Nx Ny Nz), with one mode alone: a force that
alternates along x and is the same along y and z, on lengths of the factors 2 and 3, where every sum of
the transforms is exact. u is then the force over q^2, q = pi / dx, up to the roundings of q, of 1 / q^2
and of the scale, which differ from one dx to the next. A factor that is rounded the same way for all
of them, as 1 / (Nx Ny Nz) stored in working precision, would show in their mean."""
import math

import numpy as np
import pytest
import torch

from filsim_b200 import abi
from filsim_b200.configs import params_for
from filsim_b200.fcm import Context, Fcm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,unit", [(abi.FS_PREC_FP32, 2.0 ** -24), (abi.FS_PREC_FP64, 2.0 ** -53)])
def test_no_common_error(gpu_lib, prec, unit):
    dims = (48, 144, 144)  # 1 / (Nx Ny Nz) is off by 0.51 units in FP32, by 0.77 in FP64
    f = torch.zeros((3,) + dims, dtype=torch.float64, device="cuda")
    f[1] = (1.0 - 2.0 * (torch.arange(dims[0], device="cuda") % 2).double())[:, None, None]
    err = []
    for dx in np.random.default_rng(1).uniform(0.3, 1.1, 100):
        ctx = Context(params_for(dims, dx=dx), max_beads=1)
        ctx.set_precision(prec)
        u = Fcm(ctx, 1).flow_solve(f)
        ctx.close()
        v = u[1, 0, 0, 0]
        assert not bool(u[0].any()) and not bool(u[2].any()) and bool((u[1] == v * f[1]).all())
        err.append(float(np.longdouble(float(v)) * (np.longdouble(math.pi) / np.longdouble(dx)) ** 2 - 1) / unit)
    err = np.array(err)
    # q: up to three roundings, twice in q^2; the square, the reciprocal, the scale, the product: at
    # most 10 units, and of their standard deviation a tenth in the mean of 100
    assert np.abs(err).max() <= 10
    assert abs(err.mean()) < 3 * err.std() / 10, (err.mean(), err.std())
