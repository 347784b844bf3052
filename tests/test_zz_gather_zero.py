"""The sign of a zero in the gather execution of SymmSpMV: an entry of b whose
own row has no entries, folded by a warp over more than 96 updates that leave
-0 behind, keeps it as the sequential walk does."""
import numpy as np
import pytest

from race_gb300 import matgen
from test_zz_gather_lists import _walk

torch = pytest.importorskip("torch")

from race_gb300 import interface as ri  # noqa: E402


@pytest.mark.gpu
@pytest.mark.parametrize("vdt", ["float64", "float32"])
def test_an_empty_row_keeps_a_negative_zero(vdt):
    n, hub = 300, 150
    i = np.arange(n - 1)
    others = np.delete(np.arange(n), [hub - 1, hub, hub + 1])
    r, c = np.concatenate([i, np.full(others.size, hub)]), np.concatenate([i + 1, others])
    rr, cc = np.concatenate([r, c]), np.concatenate([c, r]).astype(np.int32)
    A = matgen._assemble(n, rr, cc, np.ones(rr.size), np.full(n, 400.0), "star")
    rc = ri.Interface(n, 4, ri.TWO, A.row_ptr, A.col, symm_hint=True)
    assert rc.RACEColor() == 0
    P = A.permuted(rc.getPerm(), rc.getInvPerm())
    y = int(np.argmax(np.diff(P.row_ptr)))
    # every other row updates y; y's own row is empty
    rows = np.repeat(np.arange(n), np.diff(P.row_ptr))
    keep = rows != y
    M = matgen.Csr(n, np.concatenate([[0], np.cumsum(np.bincount(rows[keep], minlength=n))]).astype(np.int32),
                   P.col[keep], P.val[keep], "star")
    ft = np.float64 if vdt == "float64" else np.float32
    dt = getattr(torch, vdt)
    x, b = (torch.full((n,), -0.0, dtype=dt, device="cuda") for _ in range(2))
    fid = rc.registerFunction(ri.SYMMSPMV, ri.Operands(ri.DeviceCsr.from_csr(M, "cuda", dt), x, b))
    assert rc.getSweepInfo(fid)["mode"] == "gather" and rc.executeFunction(fid) == 0
    ref = np.full(n, -0.0, ft)
    _walk(ri.SYMMSPMV, rc, False, M, M.val.astype(ft), np.full(n, -0.0, ft), ref, ft)
    got = b.cpu().numpy()
    assert np.signbit(ref[y]) and np.signbit(got[y])
    np.testing.assert_array_equal(np.signbit(got), np.signbit(ref))
