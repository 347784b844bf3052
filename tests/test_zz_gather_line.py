"""Gather execution where most entries of b are above 96 updates or entries
and threads fold them: bands at the edges of the lines (96, 128, 192) against
the wave executor, and with a row above 512 entries, which that executor sums
in segments, against the sequential walk, bit for bit. For the speed of it, a
band just above 96 entries a row against one just below: four entries a row
more are not a matter of ten times (within a factor of 3; 1.04 by the work)."""
import numpy as np
import pytest

from race_gb300 import matgen
from test_zz_gather_lists import _walk

torch = pytest.importorskip("torch")

from race_gb300 import interface as ri  # noqa: E402


def _band(n, half, hub=0):
    """2 half + 1 entries a row; the first `hub` rows also in a long row n/2."""
    i = np.arange(n)
    rows = np.concatenate([i[: n - d] for d in range(1, half + 1)] + [np.full(hub, n // 2)])
    cols = np.concatenate([i[d:] for d in range(1, half + 1)] + [np.arange(hub)])
    v = np.random.Generator(np.random.PCG64(half)).standard_normal(rows.size)
    r, c = np.concatenate([rows, cols]), np.concatenate([cols, rows]).astype(np.int32)
    vv = np.concatenate([v, v])
    return matgen._assemble(n, r, c, vv, np.bincount(r, weights=np.abs(vv), minlength=n) + 1.0, "band")


def _functions(A, vdt, kernels=(ri.SPMV, ri.SPMTV, ri.SYMMSPMV)):
    rc = ri.Interface(A.n, 4, ri.TWO, A.row_ptr, A.col, symm_hint=True)
    assert rc.RACEColor() == 0
    P = A.permuted(rc.getPerm(), rc.getInvPerm())
    xdt = torch.float64 if vdt == "float64" else torch.float32
    for kernel in kernels:
        x, b = (torch.tensor(matgen.uniform_vector(A.n, k), device="cuda").to(xdt) for k in (0, 1))
        M = P.upper() if kernel == ri.SYMMSPMV else P
        fid = rc.registerFunction(kernel, ri.Operands(ri.DeviceCsr.from_csr(M, "cuda", getattr(torch, vdt)), x, b))
        assert fid >= 0
        yield kernel, rc, fid, M, x, b


@pytest.mark.gpu
@pytest.mark.parametrize("vdt", ["float64", "float32", "bfloat16"])
@pytest.mark.parametrize("half,hub", [(48, 0), (64, 0), (97, 0), (130, 0), (60, 700)])
def test_long_rows_bit_exact(vdt, half, hub):
    for kernel, rc, fid, M, x, b in _functions(_band(2500, half, hub), vdt):
        b0, got = b.clone(), []
        if hub:
            ft, ref = (np.float64 if vdt == "float64" else np.float32), b.cpu().numpy()
            val = torch.tensor(M.val).to(getattr(torch, vdt)).to(b.dtype).numpy()
            for rev in (False, True):
                assert rc.executeFunction(fid, rev) == 0
                _walk(kernel, rc, rev, M, val, x.cpu().numpy(), ref, ft)
            np.testing.assert_array_equal(b.cpu().numpy(), ref)
            continue
        for mode in (ri.SWEEP_GATHER, ri.SWEEP_WAVE):
            rc.setSweepMode(mode)
            b.copy_(b0)
            for rev in (False, True):
                assert rc.executeFunction(fid, rev) == 0
            got.append(b.cpu().numpy())
        np.testing.assert_array_equal(*got)


@pytest.mark.gpu
@pytest.mark.parametrize("kernel", [ri.SPMV, ri.SPMTV])
def test_a_few_entries_more_a_row_cost_a_few_percent(kernel):
    def time(half):
        (_, rc, fid, *_), = _functions(_band(60000, half), "float64", (kernel,))
        ev, ms = [torch.cuda.Event(enable_timing=True) for _ in range(2)], []
        for _ in range(8):
            ev[0].record()
            assert rc.executeFunctionAsync(fid) == 0
            ev[1].record()
            torch.cuda.synchronize()
            ms.append(ev[0].elapsed_time(ev[1]))
        return min(ms)

    assert time(49) < 3 * time(47)
