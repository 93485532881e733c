"""2-D assembly where an element's centroid node is also a corner of another
element: the pressure rows of that node belong to the first element alone.  The
gathered rows against the scalar kernel, which adds them element by element, to
1e-12 of a row's largest entry as for any mesh."""
import numpy as np
import pytest

from goma_gb300 import problem as pb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("energy", [False, True], ids=["flow", "energy"])
def test_rows_of_a_shared_centroid(energy):
    from goma_gb300.newton import GomaNewton
    mesh = pb.box_mesh(2, 2, 2)
    c = mesh.conn[0, 8]  # the node of element 0's pressures and of the datum
    x0, y0 = mesh.coords[c]
    # corners, sides, centroid of [x0, x0 + 0.3] x [y0, y0 + 0.4]
    loc = np.array([(0, 0), (2, 0), (2, 2), (0, 2), (1, 0), (2, 1), (1, 2), (0, 1), (1, 1)])
    new = mesh.num_nodes + np.arange(-1, 8)
    new[0] = c
    mesh.coords = np.concatenate([mesh.coords, ([x0, y0] + loc * [0.15, 0.2])[1:]])
    mesh.conn = np.ascontiguousarray(np.concatenate([mesh.conn, [new]]), np.int32)
    m = pb.Material(density=2.0, viscosity=0.6, heat_capacity=1.1, conductivity=0.3)
    bcs = list(pb.CAVITY2D_BCS) + ([(pb.VAR_T, 2, 1.0)] if energy else [])
    gn = GomaNewton(pb.Problem(mesh, m, energy, bcs, (0, 0.5)))
    x = gn.dirichlet_init(np.random.default_rng(6).uniform(-1, 1, gn.N))
    gn.set_assembly_path(1)
    R1, a1 = gn.matrix_fill_full(x)
    gn.set_assembly_path(0)
    R0, a0 = gn.matrix_fill_full(x)
    assert np.abs(R0 - R1).max() <= 1e-12 * np.abs(R1).max()
    ija = gn.msr_pattern().astype(np.int64)
    for i in range(gn.N):
        row = np.append(a1[ija[i]:ija[i + 1]], a1[i])
        got = np.append(a0[ija[i]:ija[i + 1]], a0[i])
        assert np.abs(got - row).max() <= 1e-12 * np.abs(row).max(), i
    gn.close()
