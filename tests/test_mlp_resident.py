"""The tuner network's passes with the whole network in shared memory: at the
edges of the rows a block (2, 4, 8, 16), past one turn of the grid, and at the
size where the network no longer fits; against the CPU oracle, tolerances as
in test_mlp.py. The gradients written to host memory are the device's."""
import ctypes as C

import numpy as np
import pytest

from oracle import mlp_ref

torch = pytest.importorskip("torch")

from race_gb300 import tuner  # noqa: E402


@pytest.mark.gpu
@pytest.mark.parametrize("dims,batch", [((34, 128, 3, 1), b) for b in (2, 3, 304, 305, 608, 1216, 1217, 2433, 5000)] +
                         [((35, 127, 2, 3), 306), ((36, 132, 2, 4), 1218), ((2, 6, 1, 130), 19)] +
                         [((16, h, 3, 1), 100) for h in (160, 164, 168)])  # 164 and more: tiles
def test_resident_passes_match_cpu_oracle(dims, batch):
    net, other = tuner.Mlp(*dims, seed=6), tuner.Mlp(*dims, seed=6)
    theta = net.get_params().astype(np.float64)
    rng = np.random.Generator(np.random.PCG64(batch))
    X = rng.normal(size=(batch, dims[0])).astype(np.float32)
    T = rng.normal(size=(batch, dims[3])).astype(np.float32)
    Xt, Tt = torch.tensor(X, device="cuda"), torch.tensor(T, device="cuda")
    acts = mlp_ref.forward(theta, X.astype(np.float64), dims)
    np.testing.assert_allclose(net.forward(Xt).cpu().numpy(), acts[-1], rtol=0,
                               atol=1e-5 * max(1.0, np.abs(acts[-1]).max()))
    loss_ref, g_ref = mlp_ref.loss_grad(theta, X.astype(np.float64), T.astype(np.float64), dims)
    loss, g = net.loss_grad(Xt, Tt)
    assert abs(loss - loss_ref) <= 1e-5 * max(1.0, loss_ref)
    assert np.max(np.abs(g - g_ref)) <= 1e-4 * np.max(np.abs(g_ref))
    assert other.loss_grad(Xt, Tt, want_grad=False)[0] == loss
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    for one in (net, other):
        one._check(one._lib.race_mlp_adam_step(one._h, 1e-3, 0.9, 0.999, 1e-8, s))
    np.testing.assert_array_equal(net.get_params(), other.get_params())
