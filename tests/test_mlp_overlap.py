"""Predictions written over their own inputs (outputs narrower, as wide and
wider than the inputs, and starting inside them), through the resident and the
tiled passes, past one turn of the grid: the same as written elsewhere."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from race_gb300 import tuner  # noqa: E402


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(34, 128, 3, 1), (4, 32, 2, 4), (4, 32, 2, 64), (3, 300, 2, 7)])
@pytest.mark.parametrize("batch", [5, 700, 20000])
@pytest.mark.parametrize("offset", [0, 3])
def test_outputs_over_inputs(dims, batch, offset):
    net = tuner.Mlp(*dims, seed=2)
    rng = np.random.Generator(np.random.PCG64(batch))
    X = torch.tensor(rng.normal(size=(batch, dims[0])).astype(np.float32), device="cuda")
    want = net.forward(X)
    room = torch.zeros(offset + batch * max(dims[0], dims[3]), device="cuda")
    room[:X.numel()] = X.reshape(-1)
    net._check(net._lib.race_mlp_forward(net._h, C.c_void_p(room.data_ptr()), batch,
                                         C.c_void_p(room.data_ptr() + 4 * offset),
                                         C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    assert torch.equal(room[offset:offset + want.numel()].view_as(want), want)
