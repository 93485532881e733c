"""The sync-free ILU(0) sweeps by lines of nodes against the oracle's ILU(0)
and a row-by-row substitution, where the tables can go wrong: lines of one,
two and three nodes, a whole plane as one line, nodes with 2 to 10 unknowns
(tasks of one to four rows, near columns beyond 8), independent problems (the
many-lines launch), a renumbered mesh and the multicoloured order.

One GMRES iteration returns a multiple of M^-1 b, so its direction is
compared.  The matrix has unit diagonals and off-diagonal row sums of at most
1/2: no pivot comes near the floor and every row's rounding error is at most
(row length) eps, doubled by the sums of the other rows, in the factors and
in each of the two sweeps: below 6 * 700 * eps < 1e-12 in FP64, 5e-4 in FP32.
"""
import numpy as np
import pytest

import oracle
from goma_gb300 import problem as pb

pytestmark = pytest.mark.gpu


def union(prob, copies):
    """`copies` of a problem side by side in one mesh."""
    m = prob.mesh
    nn = m.num_nodes
    m.coords = np.concatenate([m.coords + 3.0 * k for k in range(copies)])
    m.conn = np.ascontiguousarray(np.concatenate([m.conn + nn * k for k in range(copies)]), np.int32)
    m.node_sets = [np.concatenate([s + nn * k for k in range(copies)]).astype(np.int32)
                   for s in m.node_sets]
    return prob


def renumbered(prob, length):
    """Nodes in segments of `length`, every third segment first."""
    m = prob.mesh
    segs = [np.arange(a, min(m.num_nodes, a + length)) for a in range(0, m.num_nodes, length)]
    order = np.concatenate([segs[k] for r in range(3) for k in range(r, len(segs), 3)])
    new = np.empty(m.num_nodes, np.int64)
    new[order] = np.arange(m.num_nodes)
    m.coords = m.coords[order]
    m.conn = np.ascontiguousarray(new[m.conn], np.int32)
    m.node_sets = [np.sort(new[s]).astype(np.int32) for s in m.node_sets]
    return prob


def cavity(nx, ny):
    return pb.lid_cavity_2d(0, mesh=pb.box_mesh(2, nx, ny))


def cube(nx, ny, nz):
    return pb.boussinesq_cube_3d(0, mesh=pb.box_mesh(3, nx, ny, nz))


CASES = {
    "cavity 1x1": (lambda: cavity(1, 1), 0),
    "cavity 1x5": (lambda: cavity(1, 5), 0),
    "cavity 9x4": (lambda: cavity(9, 4), 0),
    "cavity 40x3": (lambda: cavity(40, 3), 0),
    "bratu 5x5": (lambda: pb.bratu_square_2d(5), 0),
    "cube 1x1x1": (lambda: cube(1, 1, 1), 0),
    "cube 1x3x2": (lambda: cube(1, 3, 2), 0),
    "cube 4x2x3": (lambda: cube(4, 2, 3), 0),
    "reacting 2x2x2": (lambda: pb.reacting_channel_3d(2, 2, 2), 0),
    "230 cavities 2x2": (lambda: union(cavity(2, 2), 230), 0),
    "260 reacting 1x1x1": (lambda: union(pb.reacting_channel_3d(1, 1, 1), 260), 0),
    "cavity 7x7 renumbered by 1": (lambda: renumbered(cavity(7, 7), 1), 0),
    "cube 3x3x2 renumbered by 3": (lambda: renumbered(cube(3, 3, 2), 3), 0),
    "cavity 6x6 multicoloured": (lambda: cavity(6, 6), 1),
    "cube 2x3x2 multicoloured": (lambda: cube(2, 3, 2), 1),
}


def system(prob, seed):
    """A well-conditioned matrix on the problem's pattern (MSR) and a vector."""
    from goma_gb300.newton import msr_pattern_host
    ija = msr_pattern_host(prob).astype(np.int64)
    N = int(ija[0]) - 1
    rng = np.random.default_rng(seed)
    a = np.zeros(len(ija))
    a[:N] = 1.0
    rows = np.repeat(np.arange(N), np.diff(ija[:N + 1]))
    a[N + 1:] = rng.uniform(-0.5, 0.5, len(rows)) / np.bincount(rows, minlength=N)[rows]
    return ija, N, a, rng.uniform(-1, 1, N)


def substitute(ija, N, lu, b):
    y = np.empty(N)
    for i in range(N):
        c, v = ija[ija[i]:ija[i + 1]], lu[ija[i]:ija[i + 1]]
        low = c < i
        y[i] = b[i] - v[low] @ y[c[low]]
    z = np.empty(N)
    for i in range(N - 1, -1, -1):
        c, v = ija[ija[i]:ija[i + 1]], lu[ija[i]:ija[i + 1]]
        up = c > i
        z[i] = (y[i] - v[up] @ z[c[up]]) / lu[i]
    return z


@pytest.mark.parametrize("fp32", [False, True], ids=["fp64", "fp32"])
@pytest.mark.parametrize("name", list(CASES))
def test_line_sweeps_apply_the_ilu0_inverse(name, fp32):
    from goma_gb300.newton import GomaNewton
    make, ordering = CASES[name]
    prob = make()
    ija, N, a, b = system(prob, 3)
    gn = GomaNewton(prob)
    gn.set_ilu_ordering(ordering)
    opts = dict(krylov_dim=1, max_linear_its=1, linear_tol=1e-30, fp32_preconditioner=fp32)

    def direction(mode):
        gn.set_triangular_solve(mode)
        d = gn.linear_solve(a, b, **opts)[0]
        return d

    d = direction(0)
    if ordering == 0:
        ref = substitute(ija, N, oracle.Oracle(prob).ilu0(a), b)
    else:  # the multicoloured factors: the level-by-level sweeps
        ref = direction(1)
    # independent problems have a factor each
    from numpy.linalg import norm
    nseg = {"230 cavities 2x2": 230, "260 reacting 1x1x1": 260}.get(name, 1)
    for u, w in zip(np.split(d, nseg), np.split(ref, nseg)):
        u, w = u / norm(u), w / norm(w)
        assert norm(u * np.sign(u @ w) - w) < (5e-4 if fp32 else 1e-12)
    gn.close()
