"""Hub rows of the matrix power (rows above 256 entries) at the edges of their
segments (FP64: 512 entries) and of the blocks' tiles (FP32, BF16: rows above
4,096 entries, tiles of 2,048): both schedules give, bit for bit, the order
restated here; in FP64 the other rows are the oracle's sequential sums."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as orc
from race_gb300 import matgen

torch = pytest.importorskip("torch")

from race_gb300 import interface as ri  # noqa: E402

_libm = ctypes.CDLL("libm.so.6")
_libm.fma.restype, _libm.fma.argtypes = ctypes.c_double, [ctypes.c_double] * 3
_libm.fmaf.restype, _libm.fmaf.argtypes = ctypes.c_float, [ctypes.c_float] * 3

LENS = (256, 257, 511, 512, 513, 1024, 1025, 4096, 4097, 6143, 6144, 6145, 33 * 512 + 7)  # with the diagonal


def _matrix(n):
    rng = np.random.Generator(np.random.PCG64(n))
    rows, cols = [np.arange(n - 1)], [np.arange(1, n)]
    far = np.arange(128, n)  # beyond every hub and its chain neighbours
    for i, length in enumerate(LENS):
        hub = 2 + 4 * i  # chain neighbours: two of its entries
        c = rng.choice(far, size=length - 3, replace=False)
        rows.append(np.full(c.size, hub))
        cols.append(c)
    r, c = np.concatenate(rows), np.concatenate(cols)
    v = rng.standard_normal(r.size)
    rr, cc, vv = np.concatenate([r, c]), np.concatenate([c, r]).astype(np.int32), np.concatenate([v, v])
    diag = np.bincount(rr, weights=np.abs(vv), minlength=n) + 1.0
    return matgen._assemble(n, rr, cc, vv / diag.max(), diag / diag.max(), "hubs")


def _butterfly(p, ft):
    for o in (16, 8, 4, 2, 1):
        p = [ft(p[i] + p[i ^ o]) for i in range(32)]
    return p[0]


def _hub(col, val, x, ft):
    fma = _libm.fma if ft is np.float64 else _libm.fmaf
    seg = 512 if ft is np.float64 else len(col)
    sums = []
    for s in range(0, len(col), seg):
        p = [ft(0)] * 32
        for i in range(s, min(s + seg, len(col))):
            p[(i - s) % 32] = ft(fma(val[i], x[col[i]], p[(i - s) % 32]))
        sums.append(_butterfly(p, ft))
    if len(sums) == 1:
        return sums[0]
    p = [ft(0)] * 32
    for g, t in enumerate(sums):
        p[g % 32] = ft(p[g % 32] + t)
    return _butterfly(p, ft)


@pytest.mark.gpu
@pytest.mark.parametrize("n,vdt", [(30000, "float64"), (170000, "float64"), (30000, "float32"), (40000, "bfloat16")])
def test_hub_rows(n, vdt):
    A, power = _matrix(n), 2
    rc = ri.Interface(A.n, 1, ri.POWER, A.row_ptr, A.col, symm_hint=True)
    assert rc.RACEColor(power, 1e9) == 0
    P = A.permuted(rc.getPerm(), rc.getInvPerm())
    lens = np.diff(P.row_ptr)
    assert set(LENS) <= set(lens.tolist())
    hubs = np.flatnonzero(lens > 256)
    ft = np.float64 if vdt == "float64" else np.float32
    dm = ri.DeviceCsr.from_csr(P, "cuda", getattr(torch, vdt))
    val = dm.val.to(torch.float64 if ft is np.float64 else torch.float32).cpu().numpy()
    x = torch.zeros((power + 1) * n, dtype=torch.float64, device="cuda")
    x[:n] = torch.tensor(matgen.uniform_vector(n, 5), device="cuda")
    fid = rc.registerFunction(ri.MPK, ri.Operands(dm, x), power=power)
    for schedule in ("sweeps", "wavefront"):
        rc.setMpkSchedule(fid, schedule)
        for _ in range(2):
            x[n:] = 0
            assert rc.executeFunction(fid) == 0
        Y = x.cpu().numpy().reshape(power + 1, n)
        for k in range(power):
            xk = Y[k].astype(ft)
            if ft is np.float64:
                ref = orc.mpk_plain(P, xk, 1)[1]
                for h in hubs:
                    s, e = P.row_ptr[h], P.row_ptr[h + 1]
                    ref[h] = _hub(P.col[s:e], val[s:e], xk, ft)
                np.testing.assert_array_equal(Y[k + 1], ref, err_msg=f"{schedule} power {k + 1}")
            else:
                ref = [_hub(P.col[P.row_ptr[h]:P.row_ptr[h + 1]], val[P.row_ptr[h]:P.row_ptr[h + 1]], xk, ft)
                       for h in hubs]
                np.testing.assert_array_equal(Y[k + 1][hubs], np.array(ref, np.float64), err_msg=f"{schedule} {k + 1}")
