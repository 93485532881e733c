"""2-D assemblies without room for the element blocks: a limit on the pool's
allocations takes the Jacobian's blocks away, or the residual's too.  The
Jacobian is then the scalar kernel's, and the residual is the one that a
residual-only assembly gives in the same conditions, bit for bit."""
import pytest

from tests import fake_runtime

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["flow", "energy and species"])
def test_residual_with_and_without_the_jacobian(kind, tmp_path):
    fake_runtime.run("""
    import os
    from tests.test_gpu_assembly_2d import make
    gn = GomaNewton(make(7, 5, **%r))
    rng = np.random.default_rng(3)
    x = gn.dirichlet_init(rng.uniform(0.2, 1.0, gn.N))
    full, vals = gn.matrix_fill_full(x)
    alone = gn.matrix_fill_full(x, jacobian=False)[0]
    assert np.array_equal(full, alone)
    gn.set_assembly_path(1)
    scalar, scalar_vals = gn.matrix_fill_full(x)
    gn.set_assembly_path(0)
    # room for a residual's blocks only: at most 240 of 6,504 bytes an element
    os.environ["POOL_LIMIT"] = str(240 * gn.problem.mesh.num_elems)
    R, a = gn.matrix_fill_full(x)
    assert np.array_equal(gn.matrix_fill_full(x, jacobian=False)[0], full)
    assert np.array_equal(R, full) and np.array_equal(a, scalar_vals)
    assert not np.array_equal(a, vals)  # the limit was in force
    # room for nothing
    os.environ["POOL_LIMIT"] = "0"
    R, a = gn.matrix_fill_full(x)
    assert np.array_equal(R, scalar) and np.array_equal(a, scalar_vals)
    assert np.array_equal(gn.matrix_fill_full(x, jacobian=False)[0], scalar)
    """ % ({"energy": True, "species": 2} if kind != "flow" else {},), tmp_path, "limit_pool.c")


def test_a_bad_element_is_counted_once(tmp_path):
    fake_runtime.run("""
    import os
    prob = cavity(4, 4)
    prob.mesh.coords[prob.mesh.conn[5]] = 0.25 - prob.mesh.coords[prob.mesh.conn[5]][:, ::-1]
    gn = GomaNewton(prob)
    def message():
        try:
            gn.matrix_fill_full(np.zeros(gn.N))
        except _lib.GbError as e:
            return str(e)
    one = message()
    assert "non-positive" in one
    os.environ["POOL_LIMIT"] = str(240 * prob.mesh.num_elems)
    assert message() == one
    """, tmp_path, "limit_pool.c")
