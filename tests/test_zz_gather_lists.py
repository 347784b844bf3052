"""Gather execution of SpMV, SpMTV and SymmSpMV where an entry of b changes
from a thread to a warp (96 updates or entries), around the groups of four and
the folds' rounds of 128, and with columns and values that are not 16-byte
aligned: forward and reverse, FP64, FP32 and BF16 values, bit for bit the
bodies of the sequential walk."""
import ctypes

import numpy as np
import pytest

from race_gb300 import matgen

torch = pytest.importorskip("torch")

from race_gb300 import interface as ri  # noqa: E402

_libm = ctypes.CDLL("libm.so.6")
_libm.fma.restype, _libm.fma.argtypes = ctypes.c_double, [ctypes.c_double] * 3
_libm.fmaf.restype, _libm.fmaf.argtypes = ctypes.c_float, [ctypes.c_float] * 3


def _matrix(n=901):
    rng = np.random.Generator(np.random.PCG64(n))
    edges = set()
    # hubs at both ends: long own rows in the upper triangle, and long lists
    for i, deg in enumerate((95, 96, 97, 98, 127, 128, 129, 260, 600)):
        for hub in (3 * i, n - 1 - 3 * i):
            for c in rng.choice(np.arange(40, n - 40), size=deg, replace=False):
                edges.add((min(hub, int(c)), max(hub, int(c))))
    e = np.array(sorted(edges))
    v = rng.standard_normal(len(e))
    rows, cols = np.concatenate([e[:, 0], e[:, 1]]), np.concatenate([e[:, 1], e[:, 0]]).astype(np.int32)
    vals = np.concatenate([v, v])
    return matgen._assemble(n, rows, cols, vals, np.bincount(rows, weights=np.abs(vals), minlength=n) + 1.0, "lists")


def _walk(kernel, rc, rev, P, val, x, b, ft):
    fma = (lambda u, v, w: ft(_libm.fma(u, v, w))) if ft is np.float64 else (lambda u, v, w: ft(_libm.fmaf(u, v, w)))
    pp, lo, hi = rc.getPhases(rev)
    for a, z in zip(lo, hi):
        for r in (range(a, z) if a <= z else range(a, z, -1)):
            s, e = int(P.row_ptr[r]), int(P.row_ptr[r + 1])
            t = ft(0)
            if kernel == ri.SPMV:
                for j in range(s, e):
                    t = fma(val[j], x[P.col[j]], t)
                b[r] = t
            elif kernel == ri.SPMTV:
                for j in range(s, e):
                    b[P.col[j]] = fma(val[j], x[r], b[P.col[j]])
            elif e > s:
                b[r] = fma(val[s], x[r], b[r])
                for j in range(s + 1, e):
                    t = fma(val[j], x[P.col[j]], t)
                    b[P.col[j]] = fma(val[j], x[r], b[P.col[j]])
                b[r] = ft(b[r] + t)


def _shifted(t):
    """The same values one element past an aligned address."""
    u = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:]
    u.copy_(t)
    return u


@pytest.mark.gpu
@pytest.mark.parametrize("vdt", ["float64", "float32", "bfloat16"])
@pytest.mark.parametrize("shifted", [False, True])
def test_gather_lists_bit_exact(vdt, shifted):
    A = _matrix()
    ft = np.float64 if vdt == "float64" else np.float32
    xdt = torch.float64 if vdt == "float64" else torch.float32
    rc = ri.Interface(A.n, 8, ri.TWO, A.row_ptr, A.col, symm_hint=True)
    assert rc.RACEColor() == 0
    P = A.permuted(rc.getPerm(), rc.getInvPerm())
    for kernel, M in ((ri.SPMV, P), (ri.SPMTV, P), (ri.SYMMSPMV, P.upper())):
        dm = ri.DeviceCsr.from_csr(M, "cuda", getattr(torch, vdt))
        if shifted:
            dm = ri.DeviceCsr(M.n, dm.row_ptr, _shifted(dm.col), _shifted(dm.val))
        val = dm.val.to(xdt).cpu().numpy()
        x0, b0 = (matgen.uniform_vector(A.n, k).astype(ft) for k in (0, 1))
        x, b = torch.tensor(x0, device="cuda"), torch.tensor(b0, device="cuda")
        fid = rc.registerFunction(kernel, ri.Operands(dm, x, b))
        ref = b0.copy()
        for rev in (False, True):
            assert rc.getSweepInfo(fid, rev)["mode"] == "gather"
            assert rc.executeFunction(fid, rev) == 0
            _walk(kernel, rc, rev, M, val, x0, ref, ft)
            np.testing.assert_array_equal(b.cpu().numpy(), ref, err_msg=f"{kernel} rev={rev}")
        # values changed in place are the ones that are used
        dm.val.mul_(2)
        val = val * ft(2)
        assert rc.executeFunction(fid) == 0
        _walk(kernel, rc, False, M, val, x0, ref, ft)
        np.testing.assert_array_equal(b.cpu().numpy(), ref)
