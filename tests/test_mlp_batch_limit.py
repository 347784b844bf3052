"""The largest batch of the tuner network and one row more, which every pass
refuses: the passes count rows and outputs in 32 bits."""
import pytest

torch = pytest.importorskip("torch")

from race_gb300 import tuner  # noqa: E402
from race_gb300._lib import RaceError  # noqa: E402

LIMIT = 65535 * 32


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(2, 4, 1, 1), (2, 1100, 1, 1)])  # fused; one kernel per product
def test_one_row_too_many_is_refused(dims):
    net = tuner.Mlp(*dims, seed=1)
    X, T = torch.ones((LIMIT + 1, 2), device="cuda"), torch.ones((LIMIT + 1, 1), device="cuda")
    with pytest.raises(RaceError):
        net.forward(X)
    with pytest.raises(RaceError):
        net.loss_grad(X, T)
    y = net.forward(X[:LIMIT])
    assert torch.equal(y[-1], net.forward(X[:1])[0]) and bool((y == y[0]).all())
