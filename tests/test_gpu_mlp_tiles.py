"""The network's kernels at the edges of their tiles and of the rules between
them: batches around a tile of 64 rows and of one row, widths around 64 (one
column of tiles more or less) and around the 8 of the narrow kernels, widths
that are not a multiple of four (no 16-byte loads or stores), unaligned
inputs, batches of one split, of two and of 32 uneven ones.

Against float64 (oracle/mlp_ref.py).  Every output is a sum of at most K FP32
products per layer, |terms| <= 1 in the mean: the bounds are those of the
tests of the network's shapes, 1e-5 on the outputs, 1e-4 of the largest
gradient."""
import numpy as np
import pytest

from oracle import mlp_ref

pytestmark = pytest.mark.gpu

CASES = [((8, 256, 3, 1), 4096), ((8, 256, 3, 1), 4161), ((9, 72, 2, 9), 63), ((9, 72, 2, 9), 65),
         ((8, 63, 2, 8), 257), ((1, 65, 2, 2), 64), ((3, 7, 2, 5), 300), ((20, 8, 1, 3), 131),
         ((5, 130, 1, 12), 1), ((12, 64, 2, 64), 1030), ((2, 9, 1, 1), 383)]


@pytest.mark.parametrize("shift", [0, 1], ids=["aligned", "unaligned"])
@pytest.mark.parametrize("shape,n", CASES)
def test_forward_and_gradients(shape, n, shift):
    import torch
    from goma_gb300.mlp import GpuMLP
    net = GpuMLP(*shape, seed=11)
    widths = net.widths
    rng = np.random.default_rng(n)
    X = rng.uniform(-1, 1, (n, widths[0])).astype(np.float32)
    T = rng.uniform(-1, 1, (n, widths[-1])).astype(np.float32)
    M = (rng.uniform(0, 1, (n, widths[-1])) < 0.6).astype(np.float32)
    M[0] = 1.0

    def dev(a):
        b = torch.zeros(a.size + shift, device="cuda")
        b[shift:] = torch.from_numpy(a).cuda().flatten()
        return b[shift:].view(a.shape)

    p = net.params()
    p[:] = rng.uniform(-0.2, 0.2, p.size)  # biases that are not zero
    net.set_params(p)
    x, t, m = dev(X), dev(T), dev(M)
    H = mlp_ref.forward(p, widths, X)
    y = net.forward(x).cpu().numpy()
    assert np.abs(y - H[-1]).max() <= 1e-5 * max(1.0, np.abs(H[-1]).max())
    loss = net.loss_grad(x, t, m)
    loss_ref, g_ref = mlp_ref.loss_and_grad(p, widths, X, T, M)
    assert abs(loss - loss_ref) <= 1e-5 * loss_ref
    assert np.abs(net.grads() - g_ref).max() <= 1e-4 * np.abs(g_ref).max()
    net.close()


@pytest.mark.parametrize("shape,n", [((8, 256, 3, 1), 4161), ((9, 72, 2, 9), 65),
                                     ((3, 20, 18, 2), 300)])
def test_a_training_step_is_the_gradient_and_an_adam_step(shape, n):
    """All layers' sums and the step in one launch (up to 16 layers), against
    the gradient's own launches and a step after them: the same operations."""
    import torch
    from goma_gb300.mlp import GpuMLP
    rng = np.random.default_rng(n)
    x, t, m = (torch.from_numpy(rng.uniform(0.1, 1, (n, k)).astype(np.float32)).cuda()
               for k in (shape[0], shape[3], shape[3]))
    nets = [GpuMLP(*shape, seed=4) for _ in range(2)]
    for k in range(2):
        nets[0].train(x, t, m, 1, batch=n, lr=1e-2)
        nets[1].loss_grad(x, t, m)
        nets[1].adam_step(lr=1e-2)
        assert np.array_equal(nets[0].grads(), nets[1].grads())
        assert np.array_equal(nets[0].params(), nets[1].params())
    for net in nets:
        net.close()
