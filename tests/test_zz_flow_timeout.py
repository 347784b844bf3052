"""Waits of the dataflow sweeps that run out: with a limit of 64 polls a chain
of thousands of dependent rows must end with RACE_ERR_TIMEOUT, and an engine
with the default limit then computes the same function."""
import numpy as np
import pytest

from race_gb300 import _lib, matgen

torch = pytest.importorskip("torch")

from race_gb300 import interface as ri  # noqa: E402

TIMEOUT = 101


def _chain(n=20000):
    i = np.arange(n - 1)
    rows, cols = np.concatenate([i, i + 1]), np.concatenate([i + 1, i]).astype(np.int32)
    return matgen._assemble(n, rows, cols, np.full(2 * n - 2, -1.0), np.full(n, 3.0), "chain")


def _engine(A, dist=ri.TWO):
    rc = ri.Interface(A.n, 1, dist, A.row_ptr, A.col, symm_hint=True)
    assert rc.RACEColor() == 0
    return rc, A.permuted(rc.getPerm(), rc.getInvPerm())


def _function(rc, P, kernel, dt=torch.float64):
    x, b = (torch.tensor(matgen.uniform_vector(P.n, k), device="cuda").to(dt) for k in (0, 1))
    fid = rc.registerFunction(kernel, ri.Operands(ri.DeviceCsr.from_csr(P, "cuda", dt), x, b))
    return fid, x


@pytest.mark.gpu
@pytest.mark.parametrize("kernel", [ri.GS, ri.KACZ])
@pytest.mark.parametrize("mode", [ri.SWEEP_WAVE, ri.SWEEP_LEAF])
@pytest.mark.parametrize("vdt", ["float64", "float32"])
def test_a_wait_that_runs_out_ends_the_sweep(kernel, mode, vdt, monkeypatch):
    A, got = _chain(), {}
    assert _lib.lib()  # the library is there
    for limit in ("0", "4194304"):
        monkeypatch.setenv("RACE_GPU_SWEEP_MAX_POLLS", limit)
        rc, P = _engine(A)
        rc.setSweepMode(mode)
        fid, x = _function(rc, P, kernel, getattr(torch, vdt))
        got[limit] = [rc.executeFunction(fid, rev) for rev in (False, True)]
    assert got == {"0": [TIMEOUT, TIMEOUT], "4194304": [0, 0]}
    assert bool(torch.isfinite(x).all())
