"""The tuner network's training pass captured in a CUDA graph after nothing
but predictions of that batch size (one chain of rows and chunks of rows), and
a captured pass that is still replayed after a larger batch has run."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from race_gb300 import tuner  # noqa: E402


def _grad(net, X, T, stream):
    net._check(net._lib.race_mlp_loss_grad(net._h, C.c_void_p(X.data_ptr()), C.c_void_p(T.data_ptr()), X.shape[0],
                                           None, None, C.c_void_p(stream.cuda_stream)))


def _stepped(net, stream):
    net._check(net._lib.race_mlp_adam_step(net._h, 1e-3, 0.9, 0.999, 1e-8, C.c_void_p(stream.cuda_stream)))
    stream.synchronize()
    return net.get_params()


def _data(batch):
    rng = np.random.Generator(np.random.PCG64(batch))
    return (torch.tensor(rng.normal(size=(batch, d)).astype(np.float32), device="cuda") for d in (34, 1))


@pytest.mark.gpu
@pytest.mark.parametrize("warm,batch", [(300, 300), (600, 600), (5000, 600), (5000, 5000)])
def test_training_pass_captured_after_predictions(warm, batch):
    net, eager = tuner.Mlp(seed=3), tuner.Mlp(seed=3)
    (X, T), (W, V) = _data(batch), _data(warm)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        net.forward(W)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        _grad(net, X, T, stream)
    _grad(net, W, V, stream)  # as large as the predictions: nothing moves
    with torch.cuda.stream(stream):
        graph.replay()
    _grad(eager, X, T, stream)
    np.testing.assert_array_equal(_stepped(net, stream), _stepped(eager, stream))
