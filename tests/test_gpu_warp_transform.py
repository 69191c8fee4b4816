"""The warp transform of the largest FP32 grids (fs_fft.cu): every grid that runs it, shown by the
kernels that ran, against FP64 flow solves: noise, the kz = 0 and kz = Nz/2 planes, kx = Nx/2, and a
uniform force, whose velocity is zero. The FP64 solve itself against PyTorch's, with test_gpu_lines.py's
bar; the FP32 bar is that file's too."""
import math

import pytest
import torch

from filsim_b200 import abi
from filsim_b200.configs import params_for
from filsim_b200.fcm import Context, Fcm
from test_gpu_lines import flow_solve
from test_gpu_lines_rule import kernels, route

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(512, 384, 384), (512, 384, 512), (512, 512, 384), (512, 512, 512)])
def test_matches_fp64(gpu_lib, dims):
    ctx = Context(params_for(dims), max_beads=1)
    fcm = Fcm(ctx, 1)
    g = torch.Generator(device="cuda").manual_seed(dims[1] + 2 * dims[2])
    noise = torch.randn((3,) + dims, generator=g, dtype=torch.float64, device="cuda")
    sign = [(1.0 - 2.0 * (torch.arange(n, device="cuda") % 2)).double() for n in dims]
    inputs = {"noise": lambda: noise, "kz0": lambda: noise[..., :1].expand_as(noise).contiguous(),
              "kzN": lambda: noise[..., :1] * sign[2], "kxN": lambda: noise[:, :1] * sign[0][:, None, None]}
    for kind, make in inputs.items():
        f = make()
        ctx.set_precision(abi.FS_PREC_FP64)
        ref = fcm.flow_solve(f)
        if kind == "noise":
            exact = flow_solve(ctx.params, f)
            assert float((ref - exact).abs().max() / exact.abs().max()) < 1e-12
            del exact
        ctx.set_precision(abi.FS_PREC_FP32)
        if kind == "noise":
            assert route(kernels(lambda: fcm.flow_solve(f))) == "warp"
        u = fcm.flow_solve(f)
        assert float((u - ref).abs().max() / ref.abs().max()) < 1e-5, kind
        del f, u, ref
    ones = torch.full_like(noise, 3.0)
    # the zero mode is dropped; what the transforms leave of it is rounding of the force over the
    # smallest q^2
    q = 2 * math.pi / (max(dims) * ctx.params.dx)
    assert float(fcm.flow_solve(ones).abs().max()) < 1e-5 * 3.0 / q ** 2
    ctx.close()
    del noise, ones
    torch.cuda.empty_cache()
