"""The spread, interpolation and bead sort where their branches change: half and quarter
spread tiles, several batches of candidates per tile, one to four interpolation warps per
bead, axes as short as the stencil; the one-CTA sort and the launched one. V and W against
the oracle: 1e-10 (FP64) and 1e-5 (FP32) of the largest component, the bars of
test_gpu_fcm.py. The sort exactly, through the cell lists, against numpy."""
import numpy as np
import pytest

from filsim_b200 import abi
from filsim_b200.configs import params_for
from filsim_b200.fcm import Context, Fcm, LinkedList
from test_gpu_fcm import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,nb,ngd,clump", [
    ((128, 128, 128), 2001, 12, 1.0),   # half tiles; one warp per bead; a partial last CTA
    ((128, 112, 96), 1480, 11, 1.0),    # two warps per bead
    ((48, 48, 48), 1481, 20, 1.0),      # quarter tiles, 27 candidate bins, one warp per bead
    ((32, 32, 64), 740, 12, 0.2),       # four warps per bead; hundreds of candidates per tile
    ((128, 128, 64), 1500, 12, 0.1),    # the same on half tiles
    ((16, 32, 16), 33, 16, 1.0),        # stencils as long as the axes
    ((32, 16, 16), 5, 12, 1.0),
    ((64, 64, 64), 4097, 12, 1.0),
])
def test_mobility_at_the_branches(oracle, gpu_lib, dims, nb, ngd, clump):
    p = params_for(dims, ngd=ngd)
    rng = np.random.default_rng(nb)
    L = np.array(dims) * p.dx
    Y = np.fmod(rng.uniform(-1.0, 1.0, (nb, 3)) * L * clump, L)
    F, T = rng.standard_normal((nb, 3)), rng.standard_normal((nb, 3))
    V0, W0 = oracle.fcm_mobility(p, Y, F, T)
    ctx = Context(p, max_beads=nb, max_filaments=nb)
    fcm = Fcm(ctx, nb)
    fcm.set(Y, F, T)
    for prec, tol in ((abi.FS_PREC_FP64, 1e-10), (abi.FS_PREC_FP32, 1e-5)):
        ctx.set_precision(prec)
        fcm.mobility_solve()
        V, W = fcm.V.cpu().numpy(), fcm.W.cpu().numpy()
        assert rel_err(V, V0) < tol and rel_err(W, W0) < tol, prec
        fcm.mobility_solve()
        assert np.array_equal(fcm.V.cpu().numpy(), V) and np.array_equal(fcm.W.cpu().numpy(), W)
    ctx.close()


@pytest.mark.parametrize("npts,nb", [(32, 0), (32, 1), (32, 33), (64, 1024), (64, 1025), (160, 4096), (160, 4097),
                                     (176, 4096)])  # 4,096 items and 40,960 cells end the one-CTA sort
def test_cell_lists_at_the_sort_limits(gpu_lib, npts, nb):
    p = params_for(npts)
    ctx = Context(p, max_beads=max(nb, 1), max_filaments=max(nb, 1))
    ll = LinkedList(ctx)
    rng = np.random.default_rng(nb)
    # half of the beads in one corner: crowded cells
    x = rng.uniform(0.0, 1.0, (nb, 3)) * npts * p.dx * np.where(rng.uniform(size=(nb, 1)) < 0.5, 0.1, 1.0)
    ll.link(x)
    head, lst, _ = ll.lists()
    M = np.array(ll.M)
    c = np.minimum((x / (npts * p.dx) * M).astype(int), M - 1)
    cell = c[:, 0] + c[:, 1] * M[0] + c[:, 2] * M[0] * M[1]
    head0, lst0 = np.full(ll.ncell, -1), np.zeros(nb, int)
    for b in range(nb):
        lst0[b] = head0[cell[b]]
        head0[cell[b]] = b
    assert np.array_equal(head, head0) and np.array_equal(lst, lst0)
    ctx.close()
