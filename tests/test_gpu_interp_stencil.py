"""The interpolation reads a bead's own stencil and nothing else: velocities elsewhere on the grid,
however large or not a number, leave U and Omega bit for bit as zeros there do."""
import ctypes

import numpy as np
import pytest
import torch

from filsim_b200 import abi
from filsim_b200.configs import params_for
from filsim_b200.fcm import Context

pytestmark = pytest.mark.gpu


def vp(t):
    return ctypes.c_void_p(t.data_ptr())


def interpolate(ctx, u, Y):
    V, W = torch.empty_like(Y), torch.empty_like(Y)
    ctx.call("fs_fcm_interpolate", vp(u), vp(Y), Y.shape[0], vp(V), vp(W))
    return V.cpu().numpy(), W.cpu().numpy()


def on_stencil(p, Y, dims):
    """Mask of the grid points in some bead's stencil (gaussian_setup's index rule)."""
    mask = np.zeros(dims, bool)
    for y in Y:
        i = [(np.trunc(y[a] / p.dx).astype(int) - p.ngd // 2 + 1 + np.arange(p.ngd)) % dims[a] for a in range(3)]
        mask[np.ix_(*i)] = True
    return mask


@pytest.mark.parametrize("fill", [np.nan, np.inf, -1e300])
@pytest.mark.parametrize("dims,ngd,nb", [((64, 48, 32), 12, 5), ((32, 32, 32), 11, 3), ((32, 16, 16), 12, 2),
                                         ((48, 48, 48), 20, 1), ((16, 64, 64), 12, 4), ((256, 256, 32), 5, 6400)])
def test_nothing_beside_the_stencil_counts(gpu_lib, dims, ngd, nb, fill):
    p = params_for(dims, ngd=ngd)
    rng = np.random.default_rng(ngd + nb)
    Y = rng.uniform(0, 1, (nb, 3)) * np.array(dims) * p.dx
    if nb > 1000:  # one warp per bead: stencils that leave columns free
        Y = np.stack([p.dx * (3.2 + 3 * (np.arange(nb) % 80)), p.dx * (2.7 + 3 * (np.arange(nb) // 80)),
                      p.dx * rng.uniform(6, 26, nb)], 1)
    mask = on_stencil(p, Y, dims)
    u = rng.standard_normal((3,) + dims)
    ctx = Context(p, max_beads=nb)
    Yd = torch.as_tensor(Y, device="cuda")
    V0, W0 = interpolate(ctx, torch.as_tensor(np.where(mask, u, 0.0), device="cuda"), Yd)
    V, W = interpolate(ctx, torch.as_tensor(np.where(mask, u, fill), device="cuda"), Yd)
    ctx.close()
    assert np.isfinite(V0).all() and np.isfinite(W0).all()
    assert np.array_equal(V, V0) and np.array_equal(W, W0)
