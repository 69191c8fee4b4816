"""The history's dot products on both sides of the length where a CTA per column gives way to
blocks of partial sums (4,096 beads), with no, one and many columns: x = J0^-1 b + C (D . b)."""
import numpy as np
import pytest

from filsim_b200.configs import sediment_params
from filsim_b200.fcm import Context, Simulation
from filsim_b200.suspension import Suspension

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nfil,nw", [(1, 2), (5, 7), (1024, 4), (4097, 1), (1366, 3)])
@pytest.mark.parametrize("cols", [0, 1, 17, 33])
def test_apply_adds_the_columns(gpu_lib, nfil, nw, cols):
    p = sediment_params(64, broyden_maxiter=40)
    rng = np.random.default_rng(nfil + cols)
    X = rng.uniform(0, 30, (nfil * nw, 3))
    q = np.tile([1.0, 0.0, 0.0, 0.0], (nfil * nw, 1))
    s = Suspension(np.arange(nfil + 1) * nw, X, q, kap=1.0, c=1.0)
    sim = Simulation(Context(p, max_beads=s.np, max_filaments=s.nfil), s)
    sim.build_jacobian(9)
    n6 = 6 * s.np
    C, D = rng.standard_normal((cols, n6)), rng.standard_normal((cols, n6))
    for i in range(cols):
        sim.set_cols(C[i], D[i], i)
    b = rng.standard_normal(n6)
    want = sim.broyden_apply(b, 0).cpu().numpy() + (D @ b) @ C
    got = sim.broyden_apply(b, cols).cpu().numpy()
    # sums of at most 64 terms a thread and a tree, here and in numpy: 128 eps of their absolute terms
    bound = 128 * np.finfo(float).eps * ((np.abs(D) @ np.abs(b)) @ np.abs(C) + np.abs(want)).max()
    assert np.abs(got - want).max() <= bound
