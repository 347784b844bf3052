"""The tuner network's fused passes at the edges of their tiles (rows a
block, 128-result and 32-term weight tiles, 32-row gradient slices, chunks of
rows) and the networks that keep one kernel per product, against the CPU
oracle. Tolerances as in test_mlp.py: FP32 sums against float64."""
import numpy as np
import pytest

from oracle import mlp_ref

torch = pytest.importorskip("torch")

from race_gb300 import tuner  # noqa: E402


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(34, 128, 3, 1), (1, 1, 1, 1), (33, 129, 2, 5), (3, 31, 15, 2), (130, 257, 1, 129),
                                  (5, 1024, 1, 3),                        # widest fused
                                  (5, 1028, 1, 3), (4, 8, 16, 1)])       # one kernel per product
@pytest.mark.parametrize("batch", [1, 5, 33, 512, 513, 609, 1300])
def test_fused_passes_match_cpu_oracle(dims, batch):
    if dims[1] > 1000 and batch > 600:
        pytest.skip("covered by the narrower networks")
    net = tuner.Mlp(*dims, seed=4)
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
    assert net.loss_grad(Xt, Tt, want_grad=False)[0] == loss
