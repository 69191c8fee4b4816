"""The filaments' approximate Jacobian, factored from both ends as a block tridiagonal matrix,
against the oracle's dense inverse: filament lengths at the edges of the two chains (one bead:
the identity; two: no second chain) and at the longest accepted one, alone and mixed in one
suspension, in both time schemes."""
import numpy as np
import pytest

from filsim_b200.configs import sediment_params
from filsim_b200.fcm import Context, Simulation
from filsim_b200.suspension import Suspension

pytestmark = pytest.mark.gpu


def bent_case(lengths, seed):
    """Parallel filaments of the given lengths, then rotations, orientations, torques and
    tensions of a bent state (the Jacobian reads no positions)."""
    p = sediment_params(64)
    rng = np.random.default_rng(seed)
    X, q = [], []
    for f, nw in enumerate(lengths):
        for i in range(nw):
            X.append([2.2 * i, 4.0 * (f % 6), 4.0 * (f // 6)])
            v = rng.standard_normal(4) * [0.1, 0.3, 0.3, 0.3] + [1, 0, 0, 0]
            q.append(v / np.linalg.norm(v))
    s = Suspension(np.concatenate([[0], np.cumsum(lengths)]), X, q, kap=np.linspace(0.1, 30.0, len(lengths)), c=2.0)
    s.set_arrays({"Us": 0.2 * rng.standard_normal((s.np, 3)), "TAU": rng.standard_normal((s.np, 3)),
                  "lam": 5.0 * rng.standard_normal((s.nlink, 3))})
    return p, s


@pytest.mark.parametrize("nt", [1, 9])
@pytest.mark.parametrize("lengths", [[1], [2], [3], [4, 5], [31, 32, 33], [47], [48], [7, 1, 48, 2, 1, 16, 3, 2, 30]])
def test_inverse_and_apply_match(oracle, gpu_lib, lengths, nt):
    p, s = bent_case(lengths, seed=100 + sum(lengths))
    sysw = oracle.System(p, s)
    ctx = Context(p, max_beads=s.np, max_filaments=s.nfil)
    sim = Simulation(ctx, s)
    sysw.build_jacobian(nt)
    sim.build_jacobian(nt)
    b = np.random.default_rng(7).standard_normal(6 * s.np)
    x = sim.broyden_apply(b, 0).cpu().numpy()
    for f, nw in enumerate(lengths):
        # 1e-10: with 80-bit solves as the reference, both routes solve such systems to 1e-13
        # (one bead has no tension for the oracle's position rows to couple to: the identity)
        want, got = sysw.jinv(f) if nw > 1 else np.eye(6), sim.jinv(f)
        assert np.abs(got - want).max() <= 1e-10 * np.abs(want).max(), (f, nw)
        lo = 6 * int(s.fil_start[f])
        xf = want @ b[lo:lo + 6 * nw]
        assert np.abs(x[lo:lo + 6 * nw] - xf).max() <= 1e-10 * np.abs(xf).max(), (f, nw)
