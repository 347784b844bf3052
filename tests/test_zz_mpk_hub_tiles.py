"""Hub rows of the matrix power at the edges of the blocks' tiles (FP32, BF16:
896 entries) and of the four stages they go through, and in larger matrices
whose chunks stride, with the hub rows before the chunks or in warps of their
own (a row above 1,024 entries): both schedules give the sums restated in
test_zz_mpk_hubs.py, bit for bit, and the same short rows."""
import numpy as np
import pytest

from race_gb300 import matgen
from test_zz_mpk_hubs import _hub

torch = pytest.importorskip("torch")

from race_gb300 import interface as ri  # noqa: E402

EDGES = tuple(896 * k + d for k in (2, 3, 4, 5, 7) for d in (-1, 0, 1))


def _matrix(n, lens):
    rng = np.random.Generator(np.random.PCG64(n + len(lens)))
    rows, cols = [np.arange(n - 1)], [np.arange(1, n)]
    far = np.arange(128, n)  # beyond every hub and its chain neighbours
    for i, length in enumerate(lens):
        rows.append(np.full(length - 3, 2 + 4 * i))  # chain neighbours: two of its entries
        cols.append(rng.choice(far, size=length - 3, replace=False))
    r, c = np.concatenate(rows), np.concatenate(cols)
    v = rng.standard_normal(r.size)
    rr, cc, vv = np.concatenate([r, c]), np.concatenate([c, r]).astype(np.int32), np.concatenate([v, v])
    diag = np.bincount(rr, weights=np.abs(vv), minlength=n) + 1.0
    return matgen._assemble(n, rr, cc, vv / diag.max(), diag / diag.max(), "tiles")


@pytest.mark.gpu
@pytest.mark.parametrize("n,lens", [(30000, EDGES), (170000, EDGES + (257, 1024, 1025, 8192)), (170000, (300,)),
                                    (240000, (1024, 300)), (240000, (1025, 600)), (660000, (3135, 1025, 257))])
@pytest.mark.parametrize("vdt", ["float32", "bfloat16", "float64"])
def test_hub_rows_at_tile_edges(n, lens, vdt):
    A, power = _matrix(n, lens), 2
    rc = ri.Interface(A.n, 1, ri.POWER, A.row_ptr, A.col, symm_hint=True)
    assert rc.RACEColor(power, 1e9) == 0
    P = A.permuted(rc.getPerm(), rc.getInvPerm())
    assert set(lens) <= set(np.diff(P.row_ptr).tolist())
    hubs = np.flatnonzero(np.diff(P.row_ptr) > 256)
    ft = np.float64 if vdt == "float64" else np.float32
    dm = ri.DeviceCsr.from_csr(P, "cuda", getattr(torch, vdt))
    val = dm.val.to(torch.float64 if vdt == "float64" else torch.float32).cpu().numpy()
    x = torch.zeros((power + 1) * n, dtype=torch.float64, device="cuda")
    x[:n] = torch.tensor(matgen.uniform_vector(n, 5), device="cuda")
    fid = rc.registerFunction(ri.MPK, ri.Operands(dm, x), power=power)
    got = []
    for schedule in ("sweeps", "wavefront"):
        rc.setMpkSchedule(fid, schedule)
        for _ in range(2):
            x[n:] = 0
            assert rc.executeFunction(fid) == 0
        got.append(x.cpu().numpy().reshape(power + 1, n))
    np.testing.assert_array_equal(*got)
    for k in range(power):
        xk = got[0][k].astype(ft)
        ref = [_hub(P.col[P.row_ptr[h]:P.row_ptr[h + 1]], val[P.row_ptr[h]:P.row_ptr[h + 1]], xk, ft) for h in hubs]
        np.testing.assert_array_equal(got[0][k + 1][hubs], np.array(ref, np.float64), err_msg=f"power {k + 1}")
