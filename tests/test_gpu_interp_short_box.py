"""FP32 interpolation in boxes whose z axis is hardly longer than the stencil (Nz < ngd + 6): each
product of velocity and weight is added in FP64, so velocities that cancel between neighbouring z
points leave the small rest whole; and points off the stencil count for nothing."""
import ctypes
import math

import numpy as np
import pytest
import torch

from filsim_b200 import abi
from filsim_b200.configs import params_for
from filsim_b200.fcm import Context

pytestmark = pytest.mark.gpu


def vp(t):
    return ctypes.c_void_p(t.data_ptr())


# one to four warps per bead (up to 740, to 1,480, and more beads)
@pytest.mark.parametrize("nb", [1, 900, 1600])
@pytest.mark.parametrize("ngd", [12, 16])
@pytest.mark.parametrize("iz", range(16))
def test_cancelling_velocities(gpu_lib, ngd, iz, nb):
    dx = 0.5  # a power of two: the weights of the two points beside the bead are the same numbers
    p = params_for((32, 32, 16), ngd=ngd, dx=dx)
    Y = np.array([[8.3, 9.1, (iz + 0.5) * dx]])
    ix, iy = int(Y[0, 0] / dx), int(Y[0, 1] / dx) + 2
    u = np.full((3, 32, 32, 16), np.nan)
    stencil = [np.array([int(Y[0, a] / dx) - ngd // 2 + 1 + i for i in range(ngd)]) % u.shape[1 + a] for a in range(3)]
    u[:, stencil[0][:, None, None], stencil[1][:, None], stencil[2]] = 0.0
    small, large = 0.75, 3.0e7
    u[0, ix, iy, iz] = large
    u[0, ix, iy, (iz + 1) % 16] = -large
    u[0, ix, iy, (iz - 1) % 16] = small
    ctx = Context(p, max_beads=nb)
    ctx.set_precision(abi.FS_PREC_FP32)
    Yd = torch.as_tensor(np.repeat(Y, nb, 0), device="cuda")
    ud, V, W = torch.as_tensor(u, device="cuda"), torch.empty_like(Yd), torch.empty_like(Yd)
    ctx.call("fs_fcm_interpolate", vp(ud), vp(Yd), nb, vp(V), vp(W))
    V, W = V.cpu().numpy(), W.cpu().numpy()
    ctx.close()
    d = np.array([ix, iy, iz - 1]) * dx - Y[0]
    g = math.exp(-(d @ d) / (2 * p.sigma ** 2)) / (2 * math.pi * p.sigma ** 2) ** 1.5
    gd = math.exp(-(d @ d) / (2 * p.sigma_dip ** 2)) / (2 * math.pi * p.sigma_dip ** 2) ** 1.5
    want_v = small * g * dx ** 3
    # W_z = -1/2 (u_y r_x - u_x r_y) gd, r = -d / sigma_dip^2
    want_w = -0.5 * (-small * (-d[1] / p.sigma_dip ** 2)) * gd * dx ** 3
    # FP32 weights: three Gaussians of 4 eps each (the exponent's rounding, expf, the product), a
    # ratio, four products: 20 eps; and what is left of exactly equal products of +-large is 0
    eps = 20 * 2.0 ** -24
    assert np.abs(V[:, 0] - want_v).max() <= eps * abs(want_v)
    assert np.abs(W[:, 2] - want_w).max() <= eps * abs(want_w)
    assert not V[:, 1:].any() and not W[:, 0].any()
