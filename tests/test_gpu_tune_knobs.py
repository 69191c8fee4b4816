"""fs_autotune times what a suspension's solves read and leaves the rest: a knob without effect keeps its
value, and is not swept. The solves are counted by the profile's interpolation stage."""
import ctypes

import numpy as np
import pytest

from filsim_b200 import abi
from filsim_b200.configs import params_for
from filsim_b200.fcm import Context, Simulation
from filsim_b200.suspension import Suspension

pytestmark = pytest.mark.gpu


def vp(a):
    return a.ctypes.data_as(ctypes.c_void_p)


@pytest.mark.parametrize("prec,npts,nfil,first,solves", [
    (abi.FS_PREC_FP64, 64, 40, (64, 16, 0, 8), 1),  # beads split over warps: nothing to choose
    (abi.FS_PREC_FP64, 64, 40, (32, 4, 1, 2), 1),
    (abi.FS_PREC_FP64, 96, 400, (64, 16, 1, 4), 3),  # the beads per CTA
    (abi.FS_PREC_FP32, 64, 40, (64, 8, 0, 2), 2 * 2 * 3),  # stages, transforms, column shapes
    (abi.FS_PREC_FP32, 160, 400, (32, 8, 0, 2), 2 * 3 * 2 * 3),  # and the beads per CTA
    (abi.FS_PREC_FP32, 176, 40, (32, 8, 1, 2), 2 * 3),  # cuFFT alone
])
def test_sweeps_what_is_read(gpu_lib, prec, npts, nfil, first, solves):
    nw, reps = 5, 2
    rng = np.random.default_rng(npts)
    X = np.repeat(rng.uniform(0, 20, (nfil, 1, 3)), nw, 1) + np.arange(nw)[None, :, None] * [2.2, 0, 0]
    s = Suspension(np.arange(nfil + 1) * nw, X.reshape(-1, 3), np.tile([1.0, 0, 0, 0], (nfil * nw, 1)), kap=1.0, c=1.0)
    ctx = Context(params_for(npts, precision=prec), max_beads=s.np, max_filaments=nfil)
    Simulation(ctx, s)
    abi.check(abi.lib().fs_set_tuning(ctx.h, vp(np.array(first, np.int32))), "fs_set_tuning")
    choice, ms = np.zeros(4, np.int32), ctypes.c_float()
    ctx.profile_enable()
    abi.check(abi.lib().fs_autotune(ctx.h, reps, vp(choice), ctypes.byref(ms)), "fs_autotune")
    ran = ctx.profile()["k_interp"][1]
    ctx.close()
    kept = {0, 2, 3} if prec == abi.FS_PREC_FP64 else {2} if npts == 176 else set()
    if nfil == 40:
        kept.add(1)
    assert all(choice[k] == first[k] for k in kept), choice
    assert ran == solves * (1 + reps)
