"""The matrix power's plain launches on both sides of the line between the
one-chunk-a-warp kernel and the striding one (32 warps an SM), odd and even
powers (which run backwards), FP64 against the oracle's chain and FP32/BF16
against the wavefront schedule, bit for bit."""
import numpy as np
import pytest

from oracle import oracle as orc
from race_gb300 import matgen

torch = pytest.importorskip("torch")

from race_gb300 import interface as ri  # noqa: E402


@pytest.mark.gpu
@pytest.mark.parametrize("side", [1, 5, 53, 54, 55])
@pytest.mark.parametrize("power", [1, 2, 3])
@pytest.mark.parametrize("vdt", ["float64", "float32", "bfloat16"])
def test_plain_launches(side, power, vdt):
    A = matgen.laplace3d_7pt(side, side, side + 1)
    rc = ri.Interface(A.n, 1, ri.POWER, A.row_ptr, A.col, symm_hint=True)
    assert rc.RACEColor(power, 300e6) == 0
    P = A.permuted(rc.getPerm(), rc.getInvPerm())
    x0 = matgen.uniform_vector(A.n, 3)
    x = torch.zeros((power + 1) * A.n, dtype=torch.float64, device="cuda")
    x[: A.n] = torch.tensor(x0, device="cuda")
    fid = rc.registerFunction(ri.MPK, ri.Operands(ri.DeviceCsr.from_csr(P, "cuda", getattr(torch, vdt)), x), power=power)
    got = {}
    for schedule in ("wavefront", "sweeps"):
        rc.setMpkSchedule(fid, schedule)
        for _ in range(2):
            x[A.n:] = 0
            assert rc.executeFunction(fid) == 0
        got[schedule] = x.cpu().numpy().reshape(power + 1, A.n)
    np.testing.assert_array_equal(got["sweeps"], got["wavefront"])
    if vdt == "float64":
        np.testing.assert_array_equal(got["sweeps"], orc.mpk_plain(P, x0, power))


@pytest.mark.gpu
@pytest.mark.parametrize("vdt", ["float64", "float32"])
@pytest.mark.parametrize("schedule", ["wavefront", "sweeps"])
def test_captured_and_replayed(vdt, schedule):
    """Captured once, replayed with new inputs; then the same powers from the
    single-power entry point."""
    A, power = matgen.stencil3d_27pt(17), 5
    rc = ri.Interface(A.n, 1, ri.POWER, A.row_ptr, A.col, symm_hint=True)
    assert rc.RACEColor(power, 300e6) == 0
    P = A.permuted(rc.getPerm(), rc.getInvPerm())
    x = torch.zeros((power + 1) * A.n, dtype=torch.float64, device="cuda")
    fid = rc.registerFunction(ri.MPK, ri.Operands(ri.DeviceCsr.from_csr(P, "cuda", getattr(torch, vdt)), x), power=power)
    rc.setMpkSchedule(fid, schedule)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    rc.setStream(stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        assert rc.executeFunctionAsync(fid) == 0
    for seed in (1, 2, 3):
        x0 = matgen.uniform_vector(A.n, seed)
        with torch.cuda.stream(stream):
            x[: A.n] = torch.tensor(x0, device="cuda")
            x[A.n:] = 0
            graph.replay()
        stream.synchronize()
        assert rc.getStatus() == 0
        got = x.cpu().numpy().copy()
        if vdt == "float64":
            np.testing.assert_array_equal(got.reshape(power + 1, A.n), orc.mpk_plain(P, x0, power))
        with torch.cuda.stream(stream):
            x[A.n:] = 0
        for k in range(power):
            rc.spmvPowerLayout(fid, k)
        stream.synchronize()
        np.testing.assert_array_equal(x.cpu().numpy(), got)
