"""Flexible CG on a parity-split level 0, whose x moves every second step
(k_fcg_step_split, k_fcg_flush): after 1, 2, 3 and 4 steps the solution and
its recomputed residual equal those of the natural-rows kernels, which update x
every step.  The two group their reductions differently, so the scalars agree
to the rounding of sums of 32768 terms."""
import numpy as np
import pytest

import briscola_b200 as bb
from briscola_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("steps", [1, 2, 3, 4])
def test_x_after_odd_and_even_steps(native, steps, precision):
    mesh, b, _ = workloads.channel(32, seed=4)
    out = {}
    for rows in ("split", "natural"):
        c = bb.Context(mesh, bb.make_options({"relTol": 0.0, "tolerance": 0, "minIter": steps, "maxIter": steps,
                                              "nSweepsPre": 2, "nSweepsPost": 2, "cycleType": "V", "coarseLevel": 1,
                                              "precision": precision, "krylov": "fcg", "rowLayout": rows,
                                              "autotune": "off"}))
        for _ in range(2):  # the second solve replays the graph on stale directions
            x = np.zeros_like(b)
            rep = c.solve(b, x, zero_guess=True)
        out[rows] = (x, rep.rel_residual)
        c.close()
    xs, xn = out["split"][0], out["natural"][0]
    assert np.linalg.norm(xs - xn) <= 1e-9 * np.linalg.norm(xn)
    assert abs(out["split"][1] - out["natural"][1]) <= 1e-6 * out["natural"][1]
