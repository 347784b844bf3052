"""race_get_mpk_layout's matrix bytes with hub rows: every array that the
powers read is in them, the FP32 copy of long FP32/BF16 hub rows included."""
import numpy as np
import pytest

from test_zz_mpk_hub_tiles import _matrix

torch = pytest.importorskip("torch")

from race_gb300 import interface as ri  # noqa: E402


@pytest.mark.gpu
@pytest.mark.parametrize("vdt,size", [("float64", 8), ("float32", 4), ("bfloat16", 2)])
@pytest.mark.parametrize("lens", [(300, 1024), (300, 1025, 4000)])
def test_matrix_bytes(vdt, size, lens, monkeypatch):
    monkeypatch.setenv("RACE_GPU_MPK_COL16", "0")
    A = _matrix(9000, lens)
    rc = ri.Interface(A.n, 1, ri.POWER, A.row_ptr, A.col, symm_hint=True)
    assert rc.RACEColor(2, 1e9) == 0
    P = A.permuted(rc.getPerm(), rc.getInvPerm())
    x = torch.zeros(3 * A.n, dtype=torch.float64, device="cuda")
    fid = rc.registerFunction(ri.MPK, ri.Operands(ri.DeviceCsr.from_csr(P, "cuda", getattr(torch, vdt)), x), power=2)
    got = rc.getMpkLayout(fid)
    hubs = [k for k in np.diff(P.row_ptr) if k > 256]
    copies = 4 * sum(k for k in hubs if k > 1024) if size < 8 else 0
    assert got["matrix_bytes"] == (got["sell_slots"] * (size + 4) + 4 * A.n + 12 * got["chunks"] + 4 * len(hubs) +
                                   (size + 4) * sum(hubs) + copies)
