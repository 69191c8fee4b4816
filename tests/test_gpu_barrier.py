"""The collision barrier with a lane per cell range and with eight lanes per bead, bit for bit
against the oracle: both sides of the line between them (48 beads per SM), boxes so small that
several neighbour slots meet in one cell, and beads on the box faces."""
import numpy as np
import pytest
import torch

from filsim_b200.configs import params_for
from filsim_b200.fcm import Context, LinkedList
from filsim_b200.suspension import fcm_positions

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npts,beads", [(16, 5), (16, 11), (32, 33), (128, "line"), (128, "over"), (160, 14001)])
def test_bit_exact(oracle, gpu_lib, npts, beads):
    line = 48 * torch.cuda.get_device_properties(0).multi_processor_count
    beads = {"line": line, "over": line + 1}.get(beads, beads)
    p = params_for(npts, **({"cell_width": 4.0} if beads == 5 else {}))  # two cells a side
    rng = np.random.default_rng(beads)
    X = rng.uniform(-0.5, 1.5, (beads, 3)) * npts * p.dx
    X[::5, 1] = npts * p.dx  # on a face
    fil, seg = np.arange(beads, dtype=np.int32) // 5, np.arange(beads, dtype=np.int32) % 5
    Y, F0 = fcm_positions(p, X), rng.standard_normal((beads, 3))
    head, lst, mp = oracle.cells_link(p, X)
    ref = oracle.collision_barrier(p, Y, F0, fil, seg, head, lst, mp, 5, max_pairs=1 << 18)
    ctx = Context(p, max_beads=beads, max_filaments=beads)
    ll = LinkedList(ctx)
    ll.link(X)
    F, Yd = torch.as_tensor(F0.copy(), device="cuda"), torch.as_tensor(Y, device="cuda")
    assert ll.apply_collision_barrier(Yd, F, 5, fil, seg) == ref["min_dist2"]
    assert np.array_equal(F.cpu().numpy(), ref["F"])
    pairs, n = ll.pairs(Yd, 5, fil, seg)
    assert n == ref["npairs"] and np.array_equal(pairs, ref["pairs"])
