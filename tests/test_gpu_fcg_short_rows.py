"""Flexible CG where the longest rows have 4, 8 or 12 cells (the grid of the
quad kernels then has more blocks than that of the one-cell kernels), on one
brick and on several, against the direct solution of the box by cosine
transforms."""
import numpy as np
import pytest
from scipy.fft import dctn, idctn

import briscola_b200 as bb
from briscola_b200.mesh import NEUMANN, Brick, Mesh

pytestmark = pytest.mark.gpu


def _direct(f, h):
    """x of zero mean with the 7-point Neumann Laplacian of x equal to f"""
    lam = sum(((2 * np.cos(np.pi * np.arange(n) / n) - 2) / h**2).reshape([-1 if d == a else 1 for a in range(3)])
              for d, n in enumerate(f.shape))
    lam[0, 0, 0] = 1.0
    q = dctn(f, type=2) / lam
    q[0, 0, 0] = 0.0
    return idctn(q, type=2)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("bricks,n1,n2", [((64,), 64, 8), ((64,), 32, 4), ((128, 128), 64, 8), ((32, 96), 32, 8),
                                          ((48, 16, 64), 48, 12)])
def test_flexible_cg_on_short_rows(native, bricks, n1, n2, precision):
    h = 1.0 / n1
    parts, at = [], 0
    for n0 in bricks:
        pts = [h * np.arange(at, at + n0 + 1.0), h * np.arange(n1 + 1.0), h * np.arange(n2 + 1.0)]
        parts.append(Brick(pts, (NEUMANN,) * 6, (at, 0, 0)))
        at += n0
    f = np.random.default_rng(at + n2).standard_normal((at, n1, n2))
    f -= f.mean()
    b = np.ascontiguousarray(h**3 * f).ravel()
    c = bb.Context(Mesh(parts), bb.make_options({"relTol": 1e-10, "tolerance": 0, "cycleType": "V", "nSweepsPre": 2,
                                                 "nSweepsPost": 2, "coarseLevel": 0, "precision": precision,
                                                 "krylov": "fcg", "maxIter": 60, "autotune": "off"}))
    x = np.zeros_like(b)
    rep = c.solve(b, x, zero_guess=True)
    c.close()
    assert rep.status == 0 and rep.rel_residual <= 2e-10
    ref = _direct(f, h).ravel()
    # |x - ref| <= |A^-1| |r|, the smallest eigenvalue being that of the longest axis
    inv = 1.0 / ((2 - 2 * np.cos(np.pi / max(at, n1, n2))) / h**2)
    assert np.linalg.norm(x - ref) <= 2e-10 * inv * np.linalg.norm(f)
