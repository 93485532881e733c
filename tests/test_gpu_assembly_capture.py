"""A captured assembly is a graph of kernels like any other: it can be
instantiated more than once at a time and be a child of another graph, and each
of these replays to the bits of a direct call."""
import ctypes

import numpy as np
import pytest

from goma_gb300 import problem as pb

pytestmark = pytest.mark.gpu


def check(rc):
    assert rc == 0, rc


CASES = {
    "2-D": lambda: pb.lid_cavity_2d(0, mesh=pb.box_mesh(2, 9, 7)),
    "2-D species": lambda: __import__("tests.test_gpu_assembly_2d", fromlist=["make"]).make(
        4, 3, energy=True, species=2),
    "3-D species": lambda: pb.reacting_channel_3d(2, 2, 2),
}


@pytest.mark.parametrize("jacobian", [True, False], ids=["jacobian", "residual"])
@pytest.mark.parametrize("name", list(CASES))
def test_instances_and_a_child_graph(name, jacobian):
    import torch
    from goma_gb300.newton import GomaNewton
    gn = GomaNewton(CASES[name]())
    rt = ctypes.CDLL("libcudart.so.13")
    x = torch.from_numpy(gn.dirichlet_init(np.random.default_rng(5).uniform(0.2, 1, gn.N))).cuda()
    R = torch.zeros(gn.N, dtype=torch.float64, device="cuda")
    v = torch.zeros(gn.nnz, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    st = torch.cuda.Stream()
    s = ctypes.c_void_p(st.cuda_stream)

    def fill():
        gn.matrix_fill_full_device(x.data_ptr(), R.data_ptr(), v.data_ptr() if jacobian else None,
                                   st.cuda_stream)
    fill()
    st.synchronize()
    want = R.clone(), v.clone()
    torch.cuda.synchronize()
    graph, parent, node = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p()
    check(rt.cudaStreamBeginCapture(s, 0))  # the strictest mode
    fill()
    check(rt.cudaStreamEndCapture(s, ctypes.byref(graph)))
    check(rt.cudaGraphCreate(ctypes.byref(parent), 0))
    check(rt.cudaGraphAddChildGraphNode(ctypes.byref(node), parent, None, ctypes.c_size_t(0),
                                        graph))
    instances = []
    for g in (graph, graph, parent):
        instances.append(ctypes.c_void_p())
        check(rt.cudaGraphInstantiate(ctypes.byref(instances[-1]), g, ctypes.c_ulonglong(0)))
    check(rt.cudaGraphDestroy(graph))
    check(rt.cudaGraphDestroy(parent))
    for e in instances * 2:
        R.fill_(float("nan"))
        v.fill_(float("nan") if jacobian else 0.0)
        torch.cuda.synchronize()
        check(rt.cudaGraphLaunch(e, s))
        st.synchronize()
        assert torch.equal(R, want[0]) and torch.equal(v, want[1])
        fill()  # a direct call between has blocks of its own
        st.synchronize()
        assert torch.equal(R, want[0]) and torch.equal(v, want[1])
    for e in instances:
        check(rt.cudaGraphExecDestroy(e))
    gn.status()
    gn.close()
