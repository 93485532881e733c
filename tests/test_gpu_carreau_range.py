"""The Carreau viscosity's derivative at both ends of its powers' range, 2-D: the
element blocks take two of the four powers from the others by division, and past
their range give what the scalar kernel's powers give.  (lambda g)^a overflows
where (lambda g)^(a - 1) does not, or underflows.

The flow is a shear u = rate y, whose advection u . grad u is zero only as the
difference of terms of the size density rate^2 (u <= rate): a residual entry is
held to 1e-12 of the larger of the residual and these terms on an element, a
matrix entry to 1e-12 of its row's largest, as elsewhere."""
import numpy as np
import pytest

from tests.test_gpu_assembly_2d import make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("a, n, rate", [
    (40.0, 0.5, 6.5e7),     # rate^40 = 3e312, rate^39 = 5e304
    (100.0, 0.4, 1.25e3),   # 5e309, 4e306
    (2.0, 0.5, 1e-150),     # 1e-300
    (40.0, 0.5, 1e-8),      # underflows to 0
    (2.0, 1.4, 1e60),       # thickening
], ids=lambda v: "%g" % v)
def test_shear_at_the_ends_of_the_range(a, n, rate):
    from goma_gb300.newton import GomaNewton
    prob = make(4, 3, carreau=(a, n))
    prob.material.lam = 1.0
    gn = GomaNewton(prob)
    x = np.zeros(gn.N)
    fu = np.empty(prob.mesh.num_nodes + 1, np.int32)
    import ctypes
    gn._L.gb_first_unknown(gn.h, fu.ctypes.data_as(ctypes.POINTER(ctypes.c_int)))
    x[fu[:-1]] = rate * prob.mesh.coords[:, 1]  # u = rate y
    gn.set_assembly_path(1)
    R1, a1 = gn.matrix_fill_full(x)
    gn.set_assembly_path(0)
    R0, a0 = gn.matrix_fill_full(x)
    assert np.isfinite(R1).all() and np.isfinite(a1).all()
    m = prob.mesh
    corner = m.coords[m.conn[:, :4]]
    d1, d2 = corner[:, 2] - corner[:, 0], corner[:, 3] - corner[:, 1]
    area = 0.5 * np.abs(d1[:, 0] * d2[:, 1] - d1[:, 1] * d2[:, 0]).max()
    scale = max(np.abs(R1).max(), prob.material.density * rate ** 2 * area)
    assert np.abs(R0 - R1).max() <= 1e-12 * scale
    ija = gn.msr_pattern().astype(np.int64)
    for i in range(gn.N):
        row = np.append(a1[ija[i]:ija[i + 1]], a1[i])
        got = np.append(a0[ija[i]:ija[i + 1]], a0[i])
        assert np.abs(got - row).max() <= 1e-12 * np.abs(row).max(), i
    gn.close()
