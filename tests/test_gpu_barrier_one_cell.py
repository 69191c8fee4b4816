"""The collision barrier in boxes with one collision cell along one, two and three axes, where a
bead's neighbour cell is its own: the bead meets itself at distance 0, its force is not a number,
the closest distance is 0 and the pairs are those of the oracle, in its order. Both of the
barrier's forms (lanes per cell range, eight lanes per bead)."""
import numpy as np
import pytest
import torch

from filsim_b200.configs import params_for
from filsim_b200.fcm import Context, LinkedList
from filsim_b200.suspension import fcm_positions

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,width,beads,cells", [((16, 16, 16), 7.0, 2, (1, 1, 1)), ((16, 64, 64), 7.0, 9, (1, 4, 4)),
                                                    ((48, 16, 32), 5.0, 5, (5, 1, 3)), ((16, 16, 64), 8.0, 4, (1, 1, 4)),
                                                    ((16, 512, 512), 5.0, 7200, (1, 55, 55))])
def test_matches_the_oracle(oracle, gpu_lib, dims, width, beads, cells):
    p = params_for(dims, cell_width=width)
    assert tuple(oracle.cells_dims(p)) == cells
    rng = np.random.default_rng(beads)
    L = np.array(dims) * p.dx
    if beads > 1000:  # a lattice in y and z, so that no bead's events outgrow its list
        n = int(np.ceil(np.sqrt(beads)))
        yz = np.stack(np.meshgrid(np.arange(n), np.arange(n), indexing="ij"), -1).reshape(-1, 2)[:beads] * (L[1] / n)
        X = np.concatenate([rng.uniform(0, 1, (beads, 1)) * L[0], yz], 1)
    else:
        X = rng.uniform(0, 1, (beads, 3)) * L
    fil, seg = np.arange(beads, dtype=np.int32), np.zeros(beads, np.int32)
    Y, F0 = fcm_positions(p, X), rng.standard_normal((beads, 3))
    head, lst, mp = oracle.cells_link(p, X)
    ref = oracle.collision_barrier(p, Y, F0, fil, seg, head, lst, mp, 5, max_pairs=1 << 18)
    assert np.isnan(ref["F"]).all()
    ctx = Context(p, max_beads=beads, max_filaments=beads)
    ll = LinkedList(ctx)
    ll.link(X)
    F, Yd = torch.as_tensor(F0.copy(), device="cuda"), torch.as_tensor(Y, device="cuda")
    assert ll.apply_collision_barrier(Yd, F, 5, fil, seg) == ref["min_dist2"] == 0.0
    assert np.array_equal(F.cpu().numpy(), ref["F"], equal_nan=True)
    pairs, n = ll.pairs(Yd, 5, fil, seg)
    assert n == ref["npairs"] and np.array_equal(pairs, ref["pairs"])
    ctx.close()
