"""The 2-D assembly by element blocks and gathered rows against the scalar
kernel (path 1) over the forms both take: one element, one-element-wide
strips, element counts around four a block and around the launch that gives
every element a block of its own, Carreau with a = 2 and without, energy with
every heat source, Boussinesq, species, transient terms, per-element
densities, integrated conditions, residual only, a caller's stream.

Both sum a few hundred FP64 products an entry: they agree to 1e-12 of the
row's largest entry (R: of the largest residual)."""
import numpy as np
import pytest

from goma_gb300 import problem as pb

pytestmark = pytest.mark.gpu

WALLS = list(pb.CAVITY2D_BCS)
HOT = [(pb.VAR_T, 2, 1.0), (pb.VAR_T, 4, 0.0)]


def make(nx, ny, energy=False, carreau=None, heat=pb.HEAT_SOURCE_NONE, bouss=False, species=0,
         ibc=False, seed=1):
    mesh = pb.box_mesh(2, nx, ny, 1, 1.0 + 0.1 * nx, 1.0, amp=0.15, seed=seed)
    m = pb.Material(density=3.0, viscosity=0.7, heat_capacity=1.3, conductivity=0.4)
    if carreau:
        m.viscosity_model = pb.VISC_CARREAU
        m.mu0, m.mu_inf, m.lam, (m.aexp, m.nexp) = 1.1, 0.05, 0.9, carreau
    m.heat_source_model, m.heat_source = heat, (0.8, 0.6)
    m.momentum_source = (0.3, -0.9, 0.0)
    if bouss:
        m.momentum_source_model = pb.SOURCE_BOUSSINESQ
        m.volume_expansion, m.reference_temperature = 0.7, 0.2
    if species:
        m.diffusivity = (1e-2,) * species
        m.species_source = ((pb.SPECIES_SOURCE_ARRHENIUS, (2.0, 1.5, -1.0, 0.0)),
                            (pb.SPECIES_SOURCE_CONSTANT, (0.3,)))[:species]
    bcs = WALLS + (HOT if energy else []) + ([(pb.VAR_Y(0), 4, 1.0)] if species else [])
    ibcs = [(pb.IBC_QCONV, 1, 2.0, 0.5), (pb.IBC_FLOW_PRESSURE, 2, 1.5, 0.0)] if ibc else []
    return pb.Problem(mesh, m, energy, bcs, (0, 0.0), species, ibcs)


CASES = {
    "1x1": dict(nx=1, ny=1),
    "1x5": dict(nx=1, ny=5),
    "3x1 energy": dict(nx=3, ny=1, energy=True),
    "5x5 carreau a=2": dict(nx=5, ny=5, carreau=(2.0, 0.5)),
    "6x3 carreau a=1.7": dict(nx=6, ny=3, carreau=(1.7, 0.6)),
    "4x4 carreau energy bouss": dict(nx=4, ny=4, energy=True, carreau=(2.0, 0.4), bouss=True),
    "7x5 energy bouss exp": dict(nx=7, ny=5, energy=True, bouss=True,
                                 heat=pb.HEAT_SOURCE_EXPONENTIAL),
    "5x4 energy const ibc": dict(nx=5, ny=4, energy=True, heat=pb.HEAT_SOURCE_CONSTANT, ibc=True),
    "4x3 species": dict(nx=4, ny=3, energy=True, species=2),
    "24x25": dict(nx=24, ny=25),
    "32x19": dict(nx=32, ny=19),
    "41x15 carreau": dict(nx=41, ny=15, carreau=(2.0, 0.5)),
}


@pytest.mark.parametrize("transient", [False, True], ids=["steady", "transient"])
@pytest.mark.parametrize("name", list(CASES))
def test_blocks_match_the_scalar_kernel(name, transient):
    from goma_gb300.newton import GomaNewton
    prob = make(**CASES[name])
    gn = GomaNewton(prob)
    rng = np.random.default_rng(2)
    x = gn.dirichlet_init(rng.uniform(0.2, 1.0, gn.N))
    xdot = rng.uniform(-1, 1, gn.N)

    def fill(jac=True):
        if transient:
            return gn.matrix_fill_full_transient(x, xdot, 0.05, 0.5, jacobian=jac)
        return gn.matrix_fill_full(x, jacobian=jac)

    def check():
        gn.set_assembly_path(1)
        R1, a1 = fill()
        gn.set_assembly_path(0)
        R0, a0 = fill()
        assert np.abs(R0 - R1).max() <= 1e-12 * np.abs(R1).max()
        ija = gn.msr_pattern().astype(np.int64)
        N = gn.N
        d = np.abs(a0 - a1)
        for i in range(N):
            row = np.append(a1[ija[i]:ija[i + 1]], a1[i])
            err = max(d[i], d[ija[i]:ija[i + 1]].max())
            assert err <= 1e-12 * np.abs(row).max(), i
        if prob.ibcs:
            return  # their kernel adds side by side, in no fixed order
        # a repeat and the residual alone are the same bit for bit
        R2, a2 = fill()
        assert np.array_equal(R2, R0) and np.array_equal(a2, a0)
        assert np.array_equal(fill(False)[0], R0)

    check()
    gn.set_element_density(rng.uniform(0.5, 5.0, prob.mesh.num_elems))
    check()
    gn.close()


def test_two_streams_have_their_own_blocks():
    """Assemblies queued on two streams at once, without a wait between them,
    give what they give one after another."""
    import torch
    from goma_gb300.newton import GomaNewton
    gn = GomaNewton(make(40, 40))
    rng = np.random.default_rng(4)
    xs = [torch.from_numpy(gn.dirichlet_init(rng.uniform(-1, 1, gn.N))).cuda() for _ in range(2)]
    def buffers():
        return (torch.zeros(gn.N, dtype=torch.float64, device="cuda"),
                torch.zeros(gn.nnz, dtype=torch.float64, device="cuda"))
    ref = [buffers() for _ in range(2)]
    out = [buffers() for _ in range(2)]
    torch.cuda.synchronize()
    for x, (R, v) in zip(xs, ref):
        gn.matrix_fill_full_device(x.data_ptr(), R.data_ptr(), v.data_ptr())
        gn.status()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for _ in range(5):
        for x, (R, v), s in zip(xs, out, streams):
            gn.matrix_fill_full_device(x.data_ptr(), R.data_ptr(), v.data_ptr(), s.cuda_stream)
    torch.cuda.synchronize()
    for (R, v), (R1, v1) in zip(ref, out):
        assert torch.equal(R, R1) and torch.equal(v, v1)
    gn.close()
