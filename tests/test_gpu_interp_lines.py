"""The interpolation on both sides of the bead counts where a bead goes from four warps to two and to
one, for short and long stencils, against the stencil sums in PyTorch FP64. The bars are those of
test_gpu_fcm_edges.py (1e-10 and 1e-5 of the largest component)."""
import ctypes
import math

import pytest
import torch

from filsim_b200 import abi
from filsim_b200.configs import params_for
from filsim_b200.fcm import Context

pytestmark = pytest.mark.gpu


def vp(t):
    return ctypes.c_void_p(t.data_ptr())


def reference(p, u, Y):
    """particle_velocities and particle_rotations (FCMfunctions.cpp:740-808)."""
    n = u.shape[1:]
    k = torch.arange(p.ngd, device="cuda")
    V, W = torch.empty_like(Y), torch.empty_like(Y)
    for b in range(0, Y.shape[0], 512):
        y = Y[b:b + 512]
        ax = []
        for a in range(3):
            xg = torch.trunc(y[:, a] / p.dx).long()[:, None] - p.ngd // 2 + 1 + k
            xx = xg.double() * p.dx - y[:, a:a + 1]
            gauss = [torch.exp(-xx * xx / (2 * s * s)) / math.sqrt(2 * math.pi * s * s) for s in (p.sigma, p.sigma_dip)]
            shape = [-1] + [p.ngd if d == a else 1 for d in range(3)]
            ax.append([t.reshape(shape) for t in (xg % n[a], gauss[0], gauss[1], -xx / p.sigma_dip ** 2)])
        (ix, gx, dx, rx), (iy, gy, dy, ry), (iz, gz, dz, rz) = ax
        v = [u[a][ix, iy, iz] for a in range(3)]
        g, d, r = gx * gy * gz, dx * dy * dz, (rx, ry, rz)
        for a in range(3):
            i, j = (a + 1) % 3, (a + 2) % 3
            V[b:b + 512, a] = (v[a] * g).sum((1, 2, 3)) * p.dx ** 3
            W[b:b + 512, a] = -0.5 * ((v[j] * r[i] - v[i] * r[j]) * d).sum((1, 2, 3)) * p.dx ** 3
    return V, W


@pytest.mark.parametrize("ngd,lines", [(12, (4, 8, 6.75, 13.5)), (14, (6.75, 13.5)), (15, (4, 40)), (20, (40,))])
def test_at_the_lines(gpu_lib, ngd, lines):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    p = params_for((64, 48, 80), ngd=ngd)
    gen = torch.Generator(device="cuda").manual_seed(ngd)
    u = torch.randn((3, 64, 48, 80), generator=gen, dtype=torch.float64, device="cuda")
    L = torch.tensor([64, 48, 80], device="cuda").double() * p.dx
    for line in lines:
        for nb in (int(line * sms), int(line * sms) + 1):
            Y = torch.rand((nb, 3), generator=gen, dtype=torch.float64, device="cuda") * L
            want = reference(p, u, Y)
            ctx = Context(p, max_beads=nb)
            for prec, tol in ((abi.FS_PREC_FP64, 1e-10), (abi.FS_PREC_FP32, 1e-5)):
                ctx.set_precision(prec)
                got = torch.empty_like(Y), torch.empty_like(Y)
                ctx.call("fs_fcm_interpolate", vp(u), vp(Y), nb, vp(got[0]), vp(got[1]))
                for a, b in zip(got, want):
                    assert float((a - b).abs().max() / b.abs().max()) < tol, (line, nb, prec)
            ctx.close()
