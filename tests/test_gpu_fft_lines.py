"""The FFT solver's line kernels at the edges of their ranges, against the
oracle's restatement: the paired transforms (bfft_pair.cu) at every length
they take, with line counts that leave a last tile nearly empty and rows whose
lines are not adjacent pairs, and the tridiagonal solves (bfft_tri.cu) around
the chunk sizes, for a line per thread block and beyond the longest of them
(2048 rows; longer lines are marched by a thread each, bfft.cu)."""
import numpy as np
import pytest

from briscola_b200 import fft
from briscola_b200.mesh import DIRICHLET, NEUMANN, PERIODIC, Brick, geometric_points, uniform_points
from oracle import fft_oracle as F

pytestmark = pytest.mark.gpu

D, N, P = (DIRICHLET,) * 2, (NEUMANN,) * 2, (PERIODIC,) * 2


def _check(n, bc, s):
    # cubic cells, the longest side n_max of them: the operator's condition
    # number is at most 3 (2 n_max / pi)^2, and two backward-stable direct
    # solves differ by that many eps; 1e-12 where it is smaller
    tol = max(1e-12, 3 * (2 * max(n) / np.pi) ** 2 * np.finfo(float).eps)
    pts = [uniform_points(m, m / max(n)) for m in n]
    pts[s] = geometric_points(n[s], 2.0, n[s] / max(n))
    faces = sum(bc, ())
    rng = np.random.default_rng(3)
    f = rng.standard_normal(n)
    h = [np.diff(p) for p in pts]
    V = h[0][:, None, None] * h[1][None, :, None] * h[2][None, None, :]
    if D not in bc:
        f -= (f * V).sum() / V.sum()
    solver = fft.FFTPoissonSolver(Brick(pts, faces))
    assert solver.solve_direction == s
    x = solver.solve(None, f)
    ref = F.solve(f, pts, faces)
    assert np.linalg.norm(x - ref) <= tol * np.linalg.norm(ref)
    return solver, f, x


@pytest.mark.parametrize("kind", [P, N, D])
@pytest.mark.parametrize("m", [16, 32, 64, 128, 256, 512])
def test_paired_transforms(m, kind):
    _check((m, 6, 32), (kind, N, P), 1)  # along x: strided lines in adjacent pairs
    _check((32, 5, m), (N, D, kind), 1)  # along z: rows, an odd number of them
    _check((32, m, 7), (P, kind, N), 2)  # odd rows: no adjacent pairs, solve along z


@pytest.mark.parametrize("ns", [2, 3, 4, 5, 63, 64, 65, 255, 256, 257, 512, 513, 1030, 2048, 2049, 3000])
def test_tridiagonal_chunks(ns):
    _check((8, ns, 4), (P, N, P), 1)
    _check((ns, 4, 8), (D, P, N), 0)
    _check((4, 8, ns), (N, P, D), 2)


def test_arrays_on_8_bytes():
    """device arrays that start on 8 bytes, not 16: the same solution"""
    import torch

    n = (32, 12, 64)
    solver, f, x = _check(n, (P, N, P), 1)
    m = int(np.prod(n))
    b = torch.empty(m + 1, dtype=torch.float64, device="cuda")[1:]
    b.copy_(torch.from_numpy(f.ravel()))
    out = torch.empty(m + 1, dtype=torch.float64, device="cuda")[1:]
    solver.solve(out, b)
    assert np.array_equal(out.cpu().numpy().reshape(n), x)
