"""Waits of the dataflow sweeps that run out: with a limit of 64 polls a chain
of thousands of dependent rows must end with RACE_ERR_TIMEOUT, and an engine
with the default limit then computes the same function. Launches behind the
failed one do not hide it: it is reported once, also from replays of a graph."""
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


def _diagonal(rc, n):
    """A Gauss-Seidel function whose rows wait for nothing: x = b / 2."""
    i = torch.arange(n + 1, dtype=torch.int32, device="cuda")
    x, b = torch.zeros(n, dtype=torch.float64, device="cuda"), torch.ones(n, dtype=torch.float64, device="cuda")
    mat = ri.DeviceCsr(n, i, i[:-1].contiguous(), torch.full((n,), 2.0, dtype=torch.float64, device="cuda"))
    return rc.registerFunction(ri.GS, ri.Operands(mat, x, b)), x, rc.registerFunction(ri.SPMV, ri.Operands(mat, b, x))


@pytest.mark.gpu
def test_a_failed_sweep_is_reported_behind_later_launches(monkeypatch):
    monkeypatch.setenv("RACE_GPU_SWEEP_MAX_POLLS", "0")
    A = _chain()
    rc, P = _engine(A)
    chain, _ = _function(rc, P, ri.GS)
    diag, x, spmv = _diagonal(rc, A.n)
    for later in ([(diag, False)], [(diag, False), (diag, True)], [(spmv, False)]):
        assert rc.executeFunctionAsync(chain) == 0
        for fid, rev in later:
            assert rc.executeFunctionAsync(fid, rev) == 0
        assert rc.getStatus() == TIMEOUT
        assert rc.getStatus() == 0  # once
        if later[0][0] == diag:
            assert bool((x == 0).all())  # not run behind the failed one
    x.zero_()
    assert rc.executeFunction(diag) == 0 and bool((x == 0.5).all())
    assert rc.executeFunctionAsync(chain) == 0
    assert rc.executeFunction(spmv) == TIMEOUT  # a synchronous call reports it too
    assert rc.executeFunction(spmv) == 0 and bool((x == 2.0).all())


@pytest.mark.gpu
def test_a_failed_replay_is_reported(monkeypatch):
    monkeypatch.setenv("RACE_GPU_SWEEP_MAX_POLLS", "0")
    A = _chain()
    rc, P = _engine(A)
    chain, _ = _function(rc, P, ri.GS)
    torch.cuda.synchronize()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    rc.setStream(stream)
    with torch.cuda.graph(graph, stream=stream):
        assert rc.executeFunctionAsync(chain) == 0
    assert rc.getStatus() == 0
    for _ in range(2):
        with torch.cuda.stream(stream):
            graph.replay()
        assert rc.getStatus() == TIMEOUT
        assert rc.getStatus() == 0
