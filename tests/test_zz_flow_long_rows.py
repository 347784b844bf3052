"""Kaczmarz rows above 512 entries that follow one another on shared columns:
their segments' updates must read the words of the rows before them. Lengths
at the edges of segments (256 entries), of the update's rounds (128) and of
the 512-entry line; repeated runs give the sequential walk's bits each time."""
import numpy as np
import pytest

from race_gb300 import matgen
from test_zz_flow import _walk

torch = pytest.importorskip("torch")

from race_gb300 import interface as ri  # noqa: E402

LENS = (512, 513, 640, 641, 767, 768, 769, 1024, 1025, 1281, 2047)  # with the diagonal


def _matrix(n=2400):
    rng = np.random.Generator(np.random.PCG64(12))
    rows, cols = [np.arange(n - 1)], [np.arange(1, n)]
    for i, length in enumerate(LENS):
        hub = 2 + 4 * i  # chain neighbours: two of its entries
        rows.append(np.full(length - 3, hub))
        cols.append(rng.choice(np.arange(60, n), size=length - 3, replace=False))
    r, c = np.concatenate(rows), np.concatenate(cols)
    v = rng.standard_normal(r.size)
    rr, cc, vv = np.concatenate([r, c]), np.concatenate([c, r]).astype(np.int32), np.concatenate([v, v])
    return matgen._assemble(n, rr, cc, vv, np.bincount(rr, weights=np.abs(vv), minlength=n) + 1.0, "long")


@pytest.mark.gpu
@pytest.mark.parametrize("vdt", ["float64", "float32", "bfloat16"])
def test_long_kaczmarz_rows_follow_one_another(vdt):
    A = _matrix()
    assert set(LENS) <= set(np.diff(A.row_ptr).tolist())
    ft = np.float64 if vdt == "float64" else np.float32
    rc = ri.Interface(A.n, 16, ri.TWO, A.row_ptr, A.col, symm_hint=True)
    assert rc.RACEColor() == 0
    rc.setSweepMode(ri.SWEEP_WAVE)
    P = A.permuted(rc.getPerm(), rc.getInvPerm())
    xdt = torch.float64 if ft is np.float64 else torch.float32
    dm = ri.DeviceCsr.from_csr(P, "cuda", getattr(torch, vdt))
    val = dm.val.to(xdt).cpu().numpy()
    x0, b0 = (matgen.uniform_vector(A.n, k).astype(ft) for k in (0, 1))
    x, b = torch.tensor(x0, device="cuda"), torch.tensor(b0, device="cuda")
    fid = rc.registerFunction(ri.KACZ, ri.Operands(dm, x, b))
    assert fid >= 0
    ref, want = x0.copy(), []
    for rev in (False, True):
        _walk(ri.KACZ, False, rc, rev, P, val, ref, b0, ft)
        want.append(ref.copy())
    for _ in range(20):
        x.copy_(torch.tensor(x0))
        for rev in (False, True):
            assert rc.executeFunction(fid, rev) == 0
            np.testing.assert_array_equal(x.cpu().numpy(), want[rev])
