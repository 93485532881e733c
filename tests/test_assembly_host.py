"""The host side of the 2-D assembly, on a CUDA runtime without a GPU
(fake_cudart.c)."""
import os

import pytest

from goma_gb300 import _lib
from tests import fake_runtime

pytestmark = pytest.mark.skipif(not os.path.exists(_lib.LIB_PATH),
                                reason="libgbnewton.so is not built")


MESHES = """
    def fan(n):
        # n quadrilaterals around node 0
        t = np.pi * np.arange(2 * n) / n
        rim = np.stack([np.cos(t), np.sin(t)], 1)
        mid = 0.5 * (rim + np.roll(rim, -1, 0))
        centroid = 0.25 * (rim[0::2] + rim[1::2] + np.roll(rim[0::2], -1, 0))
        i = np.arange(n)
        j, c = (i + 1) % n, 1 + 2 * i        # the next spoke; first corner on the rim
        m = pb.box_mesh(2, 1, 1)
        m.coords = np.concatenate([[[0.0, 0.0]], rim, mid, 0.5 * rim[0::2], centroid])
        m.conn = np.ascontiguousarray(np.stack(
            [0 * i, c, c + 1, 1 + 2 * j, 1 + 4 * n + i, 2 * n + c, 2 * n + c + 1, 1 + 4 * n + j,
             1 + 5 * n + i], 1), np.int32)
        m.node_sets = [np.array([1], np.int32) for _ in m.node_sets]
        return m
    big = GomaNewton(pb.lid_cavity_2d(0, mesh=fan(60)))
    small = GomaNewton(cavity(3, 3))
    rp, _ = big.csr_pattern()
    assert 4 * 8 * (rp[2] - rp[0]) > 48 * 1024  # the row kernel: four nodes a block
"""


@pytest.mark.parametrize("call", ["fill", "solve"])
def test_a_call_between_another_ones_launches(call, tmp_path):
    """A kernel's limit of dynamic shared memory belongs to the process: a
    second thread with a mesh of shorter rows, here between any attribute that
    the first sets and its launch, leaves the first one's launches possible."""
    fake_runtime.run(MESHES + """
    def fill(g):
        return g._L.gb_matrix_fill_full_device(g.h, g.d_x, g.d_R, g.d_vals, None)
    def solve(g):
        opts, its, rr = g.newton_opts(), ctypes.c_int(), ctypes.c_double()
        return g._L.gb_linear_solve_device(g.h, g.d_vals, g.d_R, g.d_x, ctypes.byref(opts),
                                           ctypes.byref(its), ctypes.byref(rr))
    call, calls, inside = %s, [], []
    @ctypes.CFUNCTYPE(None)
    def other_thread():
        if not inside:
            inside.append(1)
            calls.append(call(small))
            inside.pop()
    ctypes.c_void_p.in_dll(fake, "fake_attribute_set").value = ctypes.cast(
        other_thread, ctypes.c_void_p).value
    own = [call(big) for _ in range(3)]
    assert calls and not any(calls) and not any(own), (own, calls)
    """ % call, tmp_path)


def test_a_failed_launch_gives_the_element_blocks_back(tmp_path):
    """Whichever of the two launches fails, the call returns an error and holds
    no memory; the next call works."""
    fake_runtime.run("""
    gn = GomaNewton(cavity(5, 4))
    fill = lambda: gn._L.gb_matrix_fill_full_device(gn.h, gn.d_x, gn.d_R, gn.d_vals, None)
    live, fail = ll("fake_pool_live"), integer("fake_fail_launch")
    for nth in (0, 1):
        fail.value = nth
        assert fill() == -1
        assert live.value == 0
        assert fill() == 0 and live.value == 0
    """, tmp_path)


def test_blocks_of_captured_assemblies(tmp_path):
    """They come from the pool no more than they are nodes of the graph: one
    piece a captured stream, freed at the first assembly after the graph is gone,
    or with the context, whichever of the two goes first."""
    fake_runtime.run("""
    gn = GomaNewton(cavity(5, 4))
    fill = lambda st=None: gn.matrix_fill_full_device(gn.d_x, gn.d_R, gn.d_vals, st)
    capture, live, pool = ll("fake_capture"), ll("fake_malloc_live"), ll("fake_pool_live")
    fill()
    before = live.value
    for k in (1, 2):
        capture.value = k
        fill()
        fill()
        assert live.value == before + 1 and pool.value == 0
        fill(4096 * k)
        assert live.value == before + 2
        capture.value = 0
        fill()
        assert live.value == before + 2
        fake.fake_graph_gone()
        fill()
        assert live.value == before and pool.value == 0
    capture.value = 3
    fill()
    capture.value = 0
    gn.close()
    assert live.value == 0, live.value
    fake.fake_graph_gone()
    assert live.value == 0
    """, tmp_path)


def test_launches_of_an_assembly_are_counted(tmp_path):
    """bench.py's count: two for the element blocks, one a colour for the scalar
    kernel, also where it takes over for want of room."""
    fake_runtime.run("""
    import bench
    gn = GomaNewton(cavity(5, 4))
    count = lambda: bench.assembly_launches(gn, gn.d_x, None)
    assert count() == 2
    gn.set_assembly_path(1)
    assert count() == gn.num_colors == 4
    gn.set_assembly_path(0)
    limit = ll("fake_pool_limit")
    limit.value = 20 * 168
    assert count() == gn.num_colors + 2
    limit.value = 0
    assert count() == gn.num_colors
    limit.value = -1
    assert count() == 2
    """, tmp_path)
