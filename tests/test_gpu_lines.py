"""The line transforms of the Stokes solve (fs_lines.cuh) at every length they take, on
every axis, in both precisions, against a PyTorch FP64 flow solve. Tolerances: the
transforms err by a few units of rounding times log2 N per axis, about 1e-15 (FP64) and
5e-7 (FP32) of the largest component; the bars are the flow solve's of test_gpu_fcm.py,
1e-12 and 1e-5."""
import math

import pytest
import torch

from filsim_b200 import abi
from filsim_b200.configs import params_for
from filsim_b200.fcm import Context, Fcm

pytestmark = pytest.mark.gpu

LENGTHS = (32, 48, 64, 80, 96, 112, 128, 144, 160, 192, 224, 256, 320, 384, 448, 512)
# each length once per axis
DIMS = [(LENGTHS[i], LENGTHS[(5 * i + 3) % 16], LENGTHS[(11 * i + 7) % 16]) for i in range(16)]


def flow_solve(p, f):
    """flow_solve (FCMfunctions.cpp:648-736) in FP64, the k = 0 mode zeroed, the inverse along z
    taking the real part of the kz = 0 and kz = Nz/2 coefficients."""
    dims = f.shape[1:]
    s = torch.fft.rfftn(f, dim=(1, 2, 3))
    q = []
    for a, n in enumerate(dims):
        i = torch.arange(n if a < 2 else n // 2 + 1, device=f.device)
        i = torch.where(i <= n // 2, i, i - n).double() * (2 * math.pi / (n * p.dx))
        q.append(i.reshape([-1 if a == b else 1 for b in range(3)]))
    norm = 1.0 / (q[0] ** 2 + q[1] ** 2 + 1e-18 + q[2] ** 2)
    along = (q[0] * s[0] + q[1] * s[1] + q[2] * s[2]) * norm
    for a in range(3):
        s[a] = norm * (s[a] - q[a] * along) / float(dims[0] * dims[1] * dims[2])
    s[:, 0, 0, 0] = 0
    s = torch.fft.ifftn(s, dim=(1, 2), norm="forward")
    s[..., 0].imag.zero_()
    s[..., -1].imag.zero_()
    return torch.fft.irfft(s, n=dims[2], dim=3, norm="forward")


@pytest.mark.parametrize("dims", DIMS)
def test_flow_solve_at_every_length(gpu_lib, dims):
    p = params_for(dims)
    ctx = Context(p, max_beads=1)
    fcm = Fcm(ctx, 1)
    g = torch.Generator(device="cuda").manual_seed(dims[0] + 7 * dims[1])
    noise = torch.randn((3,) + dims, generator=g, dtype=torch.float64, device="cuda")
    checker = noise[..., :1] * torch.cos(math.pi * torch.arange(dims[2], device="cuda", dtype=torch.float64))  # kz = Nz/2
    for f in (noise, checker):
        ref = flow_solve(p, f)
        for prec, tol in ((abi.FS_PREC_FP64, 1e-12), (abi.FS_PREC_FP32, 1e-5)):
            ctx.set_precision(prec)
            u = fcm.flow_solve(f)
            assert float((u - ref).abs().max() / ref.abs().max()) < tol, prec
    ctx.close()
