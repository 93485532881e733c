"""The Gram-Schmidt kernels of the Krylov solvers where their tiles end, and the
product with the matrix in all its groups of rows (one to four rows, 8 and 16
lanes): fewer
unknowns than one tile of 128 rows, a few rows past a tile, more tiles than
blocks, Krylov spaces of 1, 3, 4 and 5 vectors around the four columns that a
warp takes at once and of 37 around the 32 of a block, independent problems
with tiles of their own, and FP32 vectors.

With all of the space kept, GMRES minimises the residual over it, so the
residual after m iterations is the least over the Krylov space, found here by
least squares on the same space built with the same preconditioner: one
GMRES(1) step from b returns a multiple of M^-1 b.  The matrix has unit
diagonals and off-diagonal row sums of at most 1/2, so the preconditioned
matrix is within a factor of 3 of the identity; in FP64 any order of the sums
moves the residual by less than 1e-6 of itself and 1e-9 of b (N eps < 1e-10 a
dot, 5 dots deep), and an FP32 preconditioner, whose vectors differ by their
rounding (6e-8 an entry), by less than 1e-3 and 1e-6.
"""
import numpy as np
import pytest

from goma_gb300 import problem as pb
from tests.test_gpu_line_sweeps import cavity, cube, system, union

pytestmark = pytest.mark.gpu

CASES = {
    "cavity 1x1": lambda: cavity(1, 1),
    "cavity 3x3": lambda: cavity(3, 3),
    "cavity 9x4": lambda: cavity(9, 4),
    "cube 4x2x3": lambda: cube(4, 2, 3),
    "cavity 130x70": lambda: cavity(130, 70),
    "reacting 2x2x2": lambda: pb.reacting_channel_3d(2, 2, 2),
    "bratu 5x5": lambda: pb.bratu_square_2d(5),
    "40 cavities 2x2": lambda: union(cavity(2, 2), 40),
    "3 cavities 20x17": lambda: union(cavity(20, 17), 3),
}


def matrix(ija, N, a):
    from scipy.sparse import csr_matrix
    rows = np.repeat(np.arange(N), np.diff(ija[:N + 1]))
    return csr_matrix((np.concatenate([a[N + 1:], a[:N]]),
                       (np.concatenate([rows, np.arange(N)]),
                        np.concatenate([ija[N + 1:], np.arange(N)]))), (N, N))


@pytest.mark.parametrize("fp32", [False, True], ids=["fp64", "fp32"])
@pytest.mark.parametrize("m", [1, 3, 4, 5])
@pytest.mark.parametrize("name", list(CASES))
def test_m_iterations_minimise_the_residual(name, m, fp32):
    from goma_gb300.newton import GomaNewton
    prob = CASES[name]()
    ija, N, a, b = system(prob, 7)
    gn = GomaNewton(prob)
    A = matrix(ija, N, a)
    nseg = {"40 cavities 2x2": 40, "3 cavities 20x17": 3}.get(name, 1)
    solve = lambda r, k: gn.linear_solve(a, r, krylov_dim=k, max_linear_its=k, linear_tol=1e-30,
                                         fp32_preconditioner=fp32)[0]
    x = solve(b, m)
    # the space: z_0 = M^-1 b, z_{i+1} = M^-1 (A z_i), per problem
    W = np.empty((m, N))
    v = b
    for i in range(m):
        z = solve(v, 1)
        for s in np.split(np.arange(N), nseg):
            W[i, s] = z[s] / np.linalg.norm(z[s])
        v = A @ W[i]
    for s in np.split(np.arange(N), nseg):
        As = A[s][:, s]
        B = np.stack([As @ W[i, s] for i in range(m)], 1)
        best = np.linalg.norm(b[s] - B @ np.linalg.lstsq(B, b[s], rcond=None)[0])
        got, nb = np.linalg.norm(b[s] - As @ x[s]), np.linalg.norm(b[s])
        assert got <= best * (1 + (1e-3 if fp32 else 1e-6)) + (1e-6 if fp32 else 1e-9) * nb
    gn.close()


@pytest.mark.parametrize("name", list(CASES))
def test_a_space_of_37_vectors(name):
    from goma_gb300.newton import GomaNewton
    prob = CASES[name]()
    ija, N, a, b = system(prob, 8)
    gn = GomaNewton(prob)
    x = gn.linear_solve(a, b, krylov_dim=37, max_linear_its=200, linear_tol=1e-11)[0]
    r = b - matrix(ija, N, a) @ x
    nseg = {"40 cavities 2x2": 40, "3 cavities 20x17": 3}.get(name, 1)
    for s in np.split(np.arange(N), nseg):
        assert np.linalg.norm(r[s]) <= 1.1e-11 * np.linalg.norm(b[s])
    gn.close()
