"""Wide tuner networks on both sides of the line between fused passes and one
kernel per product (width, depth and rows), against the CPU oracle with the
tolerances of test_mlp.py; the gradients on the device are the caller's. For
the speed of it, 64 rows of a wide network against 512 rows of it: a pass over
fewer rows does not take longer."""
import ctypes as C

import numpy as np
import pytest

from oracle import mlp_ref

torch = pytest.importorskip("torch")

from race_gb300 import tuner  # noqa: E402


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(34, 640, 3, 1), (34, 768, 3, 2), (9, 1024, 2, 3), (1024, 900, 2, 1024), (1024, 64, 1, 1024)])
@pytest.mark.parametrize("batch", [1, 32, 33, 150, 161, 256, 257])
def test_wide_passes_match_cpu_oracle(dims, batch):
    net, other = tuner.Mlp(*dims, seed=4), tuner.Mlp(*dims, seed=4)
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


@pytest.mark.gpu
def test_few_rows_of_a_wide_network_take_no_longer_than_many():
    net, ev = tuner.Mlp(1024, 1024, 4, 1024, seed=1), [torch.cuda.Event(enable_timing=True) for _ in range(2)]

    def time(batch):
        X, ms = torch.ones((batch, 1024), device="cuda"), []
        for _ in range(8):
            ev[0].record()
            net.forward(X)
            ev[1].record()
            torch.cuda.synchronize()
            ms.append(ev[0].elapsed_time(ev[1]))
        return min(ms)

    assert time(64) < 0.7 * time(512)  # 0.48 measured; 0.88 by blocks of two rows


@pytest.mark.gpu
def test_wide_prediction_in_a_capture():
    """Captured without a pass before it, and again after one."""
    net = tuner.Mlp(34, 1024, 3, 1, seed=2)
    X = torch.tensor(np.random.Generator(np.random.PCG64(1)).normal(size=(40, 34)).astype(np.float32), device="cuda")
    Y, stream, got = torch.empty((40, 1), device="cuda"), torch.cuda.Stream(), []
    for _ in range(2):
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            net._check(net._lib.race_mlp_forward(net._h, C.c_void_p(X.data_ptr()), 40, C.c_void_p(Y.data_ptr()),
                                                 C.c_void_p(stream.cuda_stream)))
        Y.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            graph.replay()
        stream.synchronize()
        got.append(Y.cpu().numpy().copy())
        want = net.forward(X).cpu().numpy()
    assert np.any(want) and all(np.array_equal(g, want) for g in got)
