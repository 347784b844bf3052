"""Gauss-Seidel and Kaczmarz without the SELL copy of the thread rows
(RACE_GPU_SWEEP_SELL=0), on an order of many waves: registration stays inside
its tables, and both layouts give the same bits in both executors' sums."""
import numpy as np
import pytest

from race_gb300 import matgen

torch = pytest.importorskip("torch")

from race_gb300 import interface as ri  # noqa: E402


@pytest.mark.gpu
@pytest.mark.parametrize("kernel", [ri.GS, ri.KACZ])
@pytest.mark.parametrize("vdt", ["float64", "float32"])
def test_sweeps_without_the_sell_copy(kernel, vdt, monkeypatch):
    A, got = matgen.stencil3d_27pt(11), {}
    for sell in ("1", "0"):
        monkeypatch.setenv("RACE_GPU_SWEEP_SELL", sell)
        rc = ri.Interface(A.n, 16, ri.TWO, A.row_ptr, A.col, symm_hint=True)
        assert rc.RACEColor() == 0
        P = A.permuted(rc.getPerm(), rc.getInvPerm())
        dt = getattr(torch, vdt)
        x, b = (torch.tensor(matgen.uniform_vector(A.n, k), device="cuda").to(dt) for k in (0, 1))
        fid = rc.registerFunction(kernel, ri.Operands(ri.DeviceCsr.from_csr(P, "cuda", dt), x, b))
        assert fid >= 0 and rc.getSweepInfo(fid)["waves"] > 30, rc.getSweepInfo(fid)
        for mode in (ri.SWEEP_WAVE, ri.SWEEP_LEAF):
            rc.setSweepMode(mode)
            for rev in (False, True):
                assert rc.executeFunction(fid, rev) == 0
        got[sell] = x.cpu().numpy()
    np.testing.assert_array_equal(got["0"], got["1"])
