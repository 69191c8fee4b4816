"""The lengths of the line transforms are a rule, multiples of 16 from 32 to 512 of the factors 2, 3, 5
and 7 (line_length, fs_internal.cuh). Every such length on every axis runs the line transforms and
none runs cuFFT, shown by the kernels that ran, and solves as a PyTorch FP64 flow solve does, with the
bars of test_gpu_lines.py; a length off the rule on one axis leaves the grid to cuFFT."""
import time

import pytest
import torch
from torch.profiler import ProfilerActivity, profile

from filsim_b200 import abi
from filsim_b200.configs import params_for
from filsim_b200.fcm import Context, Fcm
from test_gpu_lines import LENGTHS as TESTED, flow_solve

pytestmark = pytest.mark.gpu


def smooth(n):
    for f in (2, 3, 5, 7):
        while n % f == 0:
            n //= f
    return n == 1


RULE = [n for n in range(32, 513, 16) if smooth(n)]
NEW = [n for n in RULE if n not in TESTED]  # the others are solved in test_gpu_lines.py


def kernels(call):
    """Names of the kernels that call() launches, run twice with pauses around it: the tracer may drop
    what runs close to the ends of its window."""
    with profile(activities=[ProfilerActivity.CUDA], acc_events=True) as p:
        for _ in range(2):
            time.sleep(0.02)
            call()
            torch.cuda.synchronize()
        time.sleep(0.02)
    names = [e.key for e in p.key_averages()]
    if not any("k_" in k or "fft" in k for k in names):
        pytest.skip("no kernel is traced on this machine")
    return names


def route(names):
    """The transform that ran."""
    found = {r for r, mark in (("lines", "k_lines_"), ("warp", "k_fft_"), ("cufft", "k_project")) if any(mark in k for k in names)}
    assert len(found) == 1, names
    return found.pop()


@pytest.mark.parametrize("n", RULE)
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_every_length_runs_the_lines(gpu_lib, n, axis):
    dims = [32, 32, 32]
    dims[axis] = n
    ctx = Context(params_for(dims), max_beads=1)
    fcm = Fcm(ctx, 1)
    f = torch.zeros([3] + dims, dtype=torch.float64, device="cuda")
    for prec in (abi.FS_PREC_FP64, abi.FS_PREC_FP32):
        ctx.set_precision(prec)
        assert route(kernels(lambda: fcm.flow_solve(f))) == "lines"
    ctx.close()


@pytest.mark.parametrize("dims", [(16, 32, 32), (32, 176, 32), (32, 32, 272)])
def test_other_lengths_do_not(gpu_lib, dims):
    ctx = Context(params_for(dims), max_beads=1)
    f = torch.zeros((3,) + dims, dtype=torch.float64, device="cuda")
    assert route(kernels(lambda: Fcm(ctx, 1).flow_solve(f))) == "cufft"
    ctx.close()


# each new length once per axis
@pytest.mark.parametrize("dims", [(n, NEW[(i + 2) % len(NEW)], NEW[(5 * i + 1) % len(NEW)]) for i, n in enumerate(NEW)])
def test_flow_solve_at_the_new_lengths(gpu_lib, dims):
    ctx = Context(params_for(dims), max_beads=1)
    fcm = Fcm(ctx, 1)
    g = torch.Generator(device="cuda").manual_seed(sum(dims))
    f = torch.randn((3,) + dims, generator=g, dtype=torch.float64, device="cuda")
    ref = flow_solve(ctx.params, f)
    for prec, tol in ((abi.FS_PREC_FP64, 1e-12), (abi.FS_PREC_FP32, 1e-5)):
        ctx.set_precision(prec)
        assert float((fcm.flow_solve(f) - ref).abs().max() / ref.abs().max()) < tol, prec
    ctx.close()
    torch.cuda.empty_cache()
