"""Gather execution of large matrices with short rows (a thread per entry of b
on the plain lists): around the row count and the row lengths at which it
takes over, with rows without entries, forward and reverse, against the wave
executor, bit for bit."""
import numpy as np
import pytest

from race_gb300 import matgen

torch = pytest.importorskip("torch")

from race_gb300 import interface as ri  # noqa: E402


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(725, 723, 1), (725, 724, 1), (81, 80, 81), (1049, 1000, 1)])
@pytest.mark.parametrize("vdt", ["float64", "float32", "bfloat16"])
def test_short_rows_of_large_matrices(shape, vdt):
    A = matgen.laplace3d_7pt(*shape)  # five entries a row in one plane, seven in several
    xdt = torch.float64 if vdt == "float64" else torch.float32
    rc = ri.Interface(A.n, 256, ri.TWO, A.row_ptr, A.col, symm_hint=True)
    assert rc.RACEColor() == 0
    P = A.permuted(rc.getPerm(), rc.getInvPerm())
    for kernel in (ri.SPMV, ri.SPMTV, ri.SYMMSPMV):
        M = P.upper() if kernel == ri.SYMMSPMV else P
        rp, col, val = np.asarray(M.row_ptr), np.asarray(M.col), np.asarray(M.val)
        keep = np.ones(col.size, bool)
        for r in (0, 31, A.n // 2, A.n - 1):  # rows without entries
            keep[rp[r]:rp[r + 1]] = False
        lens = np.diff(np.concatenate([[0], np.cumsum(keep)])[rp])
        dm = ri.DeviceCsr(A.n, torch.tensor(np.concatenate([[0], np.cumsum(lens)]).astype(np.int32), device="cuda"),
                          torch.tensor(col[keep], device="cuda"),
                          torch.tensor(val[keep], device="cuda").to(getattr(torch, vdt)))
        x, b = (torch.tensor(matgen.uniform_vector(A.n, k), device="cuda").to(xdt) for k in (0, 1))
        fid = rc.registerFunction(kernel, ri.Operands(dm, x, b))
        assert fid >= 0
        b0, got = b.clone(), []
        for mode in (ri.SWEEP_GATHER, ri.SWEEP_WAVE):
            rc.setSweepMode(mode)
            b.copy_(b0)
            for rev in (False, True):
                assert rc.executeFunction(fid, rev) == 0
            got.append(b.cpu().numpy())
        np.testing.assert_array_equal(*got, err_msg=str(kernel))
