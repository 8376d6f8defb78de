"""The coarse end of a V or F cycle in one thread-block cluster (bmg_tail.cu)
against the per-pass launches, over the shapes its planning takes: levels on
one CTA and spread over several, extents that halve down to 2 and 3, rows of
odd and even length, levels that stop halving along an axis, periodic,
Dirichlet and variable-coefficient systems, V and F cycles, both precisions,
and coarse solves spread over the cluster."""
import numpy as np
import pytest

import briscola_b200 as bb
from briscola_b200 import workloads
from briscola_b200.mesh import DIRICHLET, NEUMANN, PERIODIC, Brick, Mesh, tanh_points, uniform_points

pytestmark = pytest.mark.gpu

P, N, D = (PERIODIC,) * 2, (NEUMANN,) * 2, (DIRICHLET,) * 2


def _mesh(n, bc):
    pts = [uniform_points(n[0]), tanh_points(n[1], 1.2), uniform_points(n[2])]
    return Mesh([Brick(pts, sum(bc, ()))])


CASES = [
    ((8, 8, 8), (N, N, N), 1), ((16, 16, 16), (P, N, P), 1), ((32, 32, 32), (N, N, N), 1),
    ((32, 16, 8), (P, D, P), 0), ((24, 12, 6), (D, N, N), 0), ((12, 24, 48), (N, N, D), 0),
    ((6, 48, 16), (N, N, P), 1), ((64, 4, 16), (P, N, N), 0),
    ((3, 24, 24), (N, D, N), 0), ((32, 32, 2), (N, N, P), 1), ((64, 32, 16), (P, N, P), 3),
]


@pytest.mark.parametrize("cycle", ["V", "F"])
@pytest.mark.parametrize("n,bc,coarse", CASES)
def test_cluster_tail_matches_per_pass(native, n, bc, coarse, cycle):
    mesh = _mesh(n, bc)
    rng = np.random.default_rng(5)
    V = mesh.bricks[0].cell_volumes()
    f = rng.standard_normal(n)
    b = np.ascontiguousarray((-V * workloads.zero_mean(f, V)).ravel())
    lam = [rng.uniform(0.5, 1.5, s) for s in ((n[0] + 1, n[1], n[2]), (n[0], n[1] + 1, n[2]), (n[0], n[1], n[2] + 1))]
    for d in range(3):  # one coefficient on both ends of a periodic axis
        if bc[d] == P:
            np.moveaxis(lam[d], d, 0)[-1] = np.moveaxis(lam[d], d, 0)[0]
    for precision in ("fp64", "mixed"):
        for coef in (None, lam):
            out = []
            for fuse in ("on", "off"):
                c = bb.Context(mesh, bb.make_options({
                    "relTol": 0.0, "tolerance": 0, "minIter": 3, "maxIter": 3, "nSweepsPre": 2 if cycle == "V" else 0,
                    "nSweepsPost": 2, "cycleType": cycle, "coarseLevel": coarse, "precision": precision,
                    "fuseCoarse": fuse, "autotune": "off"}))
                if coef is not None:
                    c.set_coefficients(coef)
                x = np.zeros_like(b)
                rep = c.solve(b, x, zero_guess=True)
                out.append((x, rep.kernel_launches))
                c.close()
            assert out[0][1] < out[1][1]  # the cluster ran
            # the same operations cell by cell
            assert np.array_equal(out[0][0], out[1][0]), (precision, coef is not None)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [(512, 8, 8), (8, 128, 256), (128, 8, 256), (2, 2, 512), (2, 2, 1024)])
def test_coefficients_given_to_a_context_that_fits_without_them(native, n, precision):
    """face coefficients take shared memory in the cluster: a context planned
    without them plans again when they come and when they go"""
    mesh = _mesh(n, (N, N, N))
    rng = np.random.default_rng(6)
    V = mesh.bricks[0].cell_volumes()
    b = np.ascontiguousarray((-V * workloads.zero_mean(rng.standard_normal(n), V)).ravel())
    lam = [rng.uniform(0.5, 1.5, s) for s in ((n[0] + 1, n[1], n[2]), (n[0], n[1] + 1, n[2]), (n[0], n[1], n[2] + 1))]
    out = {}
    for fuse in ("on", "off"):
        c = bb.Context(mesh, bb.make_options({
            "relTol": 0.0, "tolerance": 0, "minIter": 2, "maxIter": 2, "nSweepsPre": 2, "nSweepsPost": 2,
            "cycleType": "V", "coarseLevel": 0, "precision": precision, "fuseCoarse": fuse, "autotune": "off"}))
        out[fuse] = []
        for coef in (None, lam, None):
            c.set_coefficients(coef)
            for _ in range(2):  # the second one replays the graph
                x = np.zeros_like(b)
                rep = c.solve(b, x, zero_guess=True)
                out[fuse].append((x, rep.cycles, rep.final_l2))
        c.close()
    for on, off in zip(out["on"], out["off"]):
        assert on[1] == off[1] == 2 and np.isfinite(on[2])
        assert np.array_equal(on[0], off[0])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,bc", [((24, 16, 16), (N, N, N)), ((48, 8, 16), (D, N, P)), ((24, 24, 8), (N, D, N))])
def test_level_0_in_the_cluster_from_a_guess(native, n, bc, precision):
    """level 0 read into the cluster with its ghosts, where the last of its
    CTAs own no plane"""
    mesh = _mesh(n, bc)
    rng = np.random.default_rng(7)
    V = mesh.bricks[0].cell_volumes()
    b = np.ascontiguousarray((-V * workloads.zero_mean(rng.standard_normal(n), V)).ravel())
    guess = rng.standard_normal(b.size)
    out = []
    for fuse in ("on", "off"):
        c = bb.Context(mesh, bb.make_options({
            "relTol": 0.0, "tolerance": 0, "minIter": 2, "maxIter": 2, "nSweepsPre": 2, "nSweepsPost": 2,
            "cycleType": "V", "coarseLevel": 0, "precision": precision, "fuseCoarse": fuse, "autotune": "off"}))
        x = guess.copy()
        rep = c.solve(b, x)
        out.append((x, rep.kernel_launches))
        c.close()
    assert out[0][1] < out[1][1]
    assert np.array_equal(out[0][0], out[1][0])


@pytest.mark.parametrize("mode", ["guess", "replace"])
@pytest.mark.parametrize("level", [1, 2, 3, 4])
def test_levels_below_a_level_solver(native, level, mode):
    """a level solver at a level that would fit the cluster: the levels below
    it run there, and the solver is called as often as with a launch per pass"""
    import torch

    from briscola_b200 import learned

    mesh = learned.cube_mesh(64)
    b = np.random.default_rng(8).standard_normal(64**3)
    b -= b.mean()
    out = []
    for fuse in ("on", "off"):
        c = bb.Context(mesh, bb.make_options({
            "relTol": 0.0, "tolerance": 0, "minIter": 3, "maxIter": 3, "nSweepsPre": 2, "nSweepsPost": 2,
            "cycleType": "V", "coarseLevel": 1, "precision": "mixed", "krylov": "fcg", "fuseCoarse": fuse,
            "graph": "off", "autotune": "off"}))
        calls = []

        def smooth_guess(stream, rhs, x, shape):
            torch.cuda.synchronize()
            r = torch.empty(int(np.prod(shape)), dtype=torch.float32, device="cuda")
            learned._copy_from_ptr(r, rhs)
            calls.append(shape)
            learned._copy_to_ptr(x, (r * (-0.1 / 64**2 * 4**level)).contiguous())
            torch.cuda.synchronize()

        c.set_level_solver(level, smooth_guess, mode)
        x = np.zeros_like(b)
        rep = c.solve(b, x, zero_guess=True)
        out.append((x, len(calls), rep.kernel_launches))
        c.close()
    assert out[0][1] == out[1][1] == 3
    assert np.array_equal(out[0][0], out[1][0])
    if mode == "guess" and level < 3:  # (the coarse solve's level is 4)
        assert out[0][2] < out[1][2]
