"""Species rows of 3-D elements by sum factorisation against the dense kernel
(path 1): 1 to 4 species, every source, steady and transient, perturbed
meshes of one element to a few per colour, with and without the energy
equation, Dirichlet species rows, residual only.  Both sum a few thousand FP64
products an entry: 1e-12 of the row's largest entry (R: of the largest
residual)."""
import numpy as np
import pytest

from goma_gb300 import problem as pb

pytestmark = pytest.mark.gpu

ARR, CON, NON = (pb.SPECIES_SOURCE_ARRHENIUS, pb.SPECIES_SOURCE_CONSTANT,
                 pb.SPECIES_SOURCE_NONE)
CASES = {
    "1x1x1 one": (1, 1, 1, True, [(ARR, (2.0, 1.5, -1.0, 0.0))]),
    "3x2x2 two": (3, 2, 2, True, [(ARR, (2.0, 1.5, -1.0, 0.0)), (ARR, (2.0, 1.5, 1.0, 0.0))]),
    "1x4x2 three": (1, 4, 2, True, [(NON, ()), (ARR, (1.0, 0.5, -2.0, 2.0)), (CON, (0.4,))]),
    "2x2x3 four": (2, 2, 3, True, [(CON, (0.2,)), (ARR, (1.0, 0.5, 1.0, 3.0)),
                                   (ARR, (3.0, 1.0, -1.0, 2.0)), (NON, ())]),
    "2x3x2 two without energy": (2, 3, 2, False, [(CON, (0.7,)), (NON, ())]),
}


@pytest.mark.parametrize("transient", [False, True], ids=["steady", "transient"])
@pytest.mark.parametrize("name", list(CASES))
def test_species_rows_match_the_dense_kernel(name, transient):
    from goma_gb300.newton import GomaNewton
    nx, ny, nz, energy, src = CASES[name]
    mesh = pb.box_mesh(3, nx, ny, nz, 1.2, 1.0, 0.9, amp=0.15, seed=3)
    mat = pb.Material(density=1.5, viscosity=0.3, conductivity=0.2,
                      diffusivity=tuple(0.02 * (w + 1) for w in range(len(src))),
                      species_source=tuple(src))
    bcs = [(pb.VAR_U1, 1, 1.0), (pb.VAR_U2, 3, 0.0), (pb.VAR_Y(0), 1, 1.0)]
    bcs += [(pb.VAR_T, 1, 2.0)] if energy else []
    gn = GomaNewton(pb.Problem(mesh, mat, energy, bcs, (0, 0.0), len(src)))
    rng = np.random.default_rng(6)
    x = gn.dirichlet_init(rng.uniform(0.5, 1.5, gn.N))
    xdot = rng.uniform(-1, 1, gn.N)

    def fill(path, jac=True):
        gn.set_assembly_path(path)
        if transient:
            return gn.matrix_fill_full_transient(x, xdot, 0.05, 0.5, jacobian=jac)
        return gn.matrix_fill_full(x, jacobian=jac)

    R1, a1 = fill(1)
    R0, a0 = fill(0)
    assert np.abs(R0 - R1).max() <= 1e-12 * np.abs(R1).max()
    ija = gn.msr_pattern().astype(np.int64)
    d = np.abs(a0 - a1)
    for i in range(gn.N):
        row = np.append(a1[ija[i]:ija[i + 1]], a1[i])
        assert max(d[i], d[ija[i]:ija[i + 1]].max()) <= 1e-12 * np.abs(row).max(), i
    assert np.array_equal(fill(0, False)[0], R0)
    gn.close()
