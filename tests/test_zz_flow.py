"""Dataflow sweeps (Gauss-Seidel, Kaczmarz) against a scalar restatement of
the two row bodies on the engine's own phases, bit for bit: the sequential
sums of wave mode (long rows in segments of 256) and the lane sums and
butterfly of leaf mode, in FP64, FP32 and BF16 values, forward and backward,
also replayed from a CUDA graph. Row lengths cross the limits of the task
kinds (8, 16, 32 products, thread rows, warp folds, segments). Rows without
entries, and a Kaczmarz operand that names a column twice (which keeps the
wave executor), run as the sequential walk does."""
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


def _matrix(n=900, seed=3):
    """Symmetric pattern whose row lengths run from 1 to about 700."""
    rng = np.random.Generator(np.random.PCG64(seed))
    edges = set()
    for hub, deg in ((7, 690), (400, 515), (401, 512), (500, 300), (501, 129), (502, 65), (503, 34), (504, 33),
                     (505, 32), (506, 17), (507, 16), (508, 9), (509, 8)):
        for c in rng.choice(n - 20, size=deg, replace=False):
            if c != hub:
                edges.add((min(hub, int(c)), max(hub, int(c))))
    for _ in range(2 * n):
        a, b = (int(v) for v in rng.integers(0, n - 20, size=2))
        if a != b:
            edges.add((min(a, b), max(a, b)))
    e = np.array(sorted(edges))
    v = rng.standard_normal(len(e))
    rows, cols = np.concatenate([e[:, 0], e[:, 1]]), np.concatenate([e[:, 1], e[:, 0]]).astype(np.int32)
    vals = np.concatenate([v, v])
    diag = np.bincount(rows, weights=np.abs(vals), minlength=n) + 1.0
    return matgen._assemble(n, rows, cols, vals, diag, "flow")


def _butterfly(p, ft):
    p = list(p)
    for o in (16, 8, 4, 2, 1):
        p = [ft(p[i] + p[i ^ o]) for i in range(32)]
    return p[0]


def _walk(kernel, leaf, rc, rev, P, val, x, b, ft):
    """The phases' rows in order with the executor's sums in type ft."""
    fma = (lambda u, v, w: ft(_libm.fma(u, v, w))) if ft is np.float64 else (lambda u, v, w: ft(_libm.fmaf(u, v, w)))
    pp, lo, hi = rc.getPhases(rev)
    for a, z in zip(lo, hi):
        for r in (range(a, z) if a <= z else range(a, z, -1)):
            s, e = int(P.row_ptr[r]), int(P.row_ptr[r + 1])
            if s == e:
                continue
            c, v, gs = P.col[s:e], val[s:e], kernel == ri.GS
            k0 = 1 if gs else 0
            if leaf or e - s > 512:
                step = e - s if leaf else 256
                dot = nrm = None
                parts = []
                for q in range(0, e - s, step):
                    p, w = [ft(0)] * 32, [ft(0)] * 32
                    first = k0 if q == 0 else 0
                    for i, k in enumerate(range(q + (first if leaf else 0), min(q + step, e - s))):
                        if not leaf and gs and k == 0:
                            continue
                        u = -v[k] if gs and leaf else v[k]
                        p[i % 32] = fma(u, x[c[k]], p[i % 32])
                        w[i % 32] = fma(v[k], v[k], w[i % 32])
                    parts.append((_butterfly(p, ft), _butterfly(w, ft)))
                if leaf:
                    dot, nrm = parts[0]
                else:
                    p, w = [ft(0)] * 32, [ft(0)] * 32
                    for i, (d, m) in enumerate(parts):
                        p[i % 32], w[i % 32] = ft(p[i % 32] + d), ft(w[i % 32] + m)
                    dot, nrm = _butterfly(p, ft), _butterfly(w, ft)
                if gs:
                    x[r] = ft((b[r] + dot) / v[0]) if leaf else ft((b[r] - dot) / v[0])
                    continue
                sc = ft(ft(dot - b[r]) / nrm)
            elif gs:
                t = b[r]
                for k in range(1, e - s):
                    t = fma(-v[k], x[c[k]], t)
                x[r] = ft(t / v[0])
                continue
            else:
                sc, nrm = ft(-b[r]), ft(0)
                for k in range(e - s):
                    sc, nrm = fma(v[k], x[c[k]], sc), fma(v[k], v[k], nrm)
                sc = ft(sc / nrm)
            for k in range(e - s):
                x[c[k]] = fma(-sc, v[k], x[c[k]])


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["wave", "leaf"])
@pytest.mark.parametrize("vdt", ["float64", "float32", "bfloat16"])
def test_flow_sweeps_bit_exact(mode, vdt):
    A = _matrix()
    lens = np.diff(A.row_ptr)
    assert lens.min() == 1 and lens.max() > 600
    ft = np.float64 if vdt == "float64" else np.float32
    xdt = torch.float64 if vdt == "float64" else torch.float32
    for kernel, dist in ((ri.GS, 1), (ri.KACZ, 2)):
        rc = ri.Interface(A.n, 16, dist, A.row_ptr, A.col, symm_hint=True)
        assert rc.RACEColor() == 0
        rc.setSweepMode(ri.SWEEP_WAVE if mode == "wave" else ri.SWEEP_LEAF)
        P = A.permuted(rc.getPerm(), rc.getInvPerm())
        dm = ri.DeviceCsr.from_csr(P, "cuda", getattr(torch, vdt))
        val = dm.val.to(xdt).cpu().numpy()
        x0, b0 = (matgen.uniform_vector(A.n, k).astype(ft) for k in (0, 1))
        x, b = torch.tensor(x0, device="cuda"), torch.tensor(b0, device="cuda")
        fid = rc.registerFunction(kernel, ri.Operands(dm, x, b))
        assert fid >= 0
        ref = x0.copy()
        for rev in (False, True):
            assert rc.executeFunction(fid, rev) == 0
            _walk(kernel, mode == "leaf", rc, rev, P, val, ref, b0, ft)
            np.testing.assert_array_equal(x.cpu().numpy(), ref, err_msg=f"{kernel} rev={rev}")
        # captured once, replayed twice: every replay is one more sweep
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        rc.setStream(stream)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            assert rc.executeFunctionAsync(fid) == 0
        for _ in range(2):
            graph.replay()
            _walk(kernel, mode == "leaf", rc, False, P, val, ref, b0, ft)
        torch.cuda.synchronize()
        assert rc.getStatus() == 0
        np.testing.assert_array_equal(x.cpu().numpy(), ref)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [ri.SWEEP_WAVE, ri.SWEEP_LEAF])
def test_flow_rows_without_entries_keep_their_value(mode):
    A = matgen.chain_with_empty_rows()
    rc = ri.Interface(A.n, 4, ri.ONE, A.row_ptr, A.col, symm_hint=True)
    assert rc.RACEColor() == 0
    rc.setSweepMode(mode)
    P = A.permuted(rc.getPerm(), rc.getInvPerm())
    x0, b0 = matgen.uniform_vector(A.n, 0), matgen.uniform_vector(A.n, 1)
    x = torch.tensor(x0, device="cuda")
    fid = rc.registerFunction(ri.GS, ri.Operands(ri.DeviceCsr.from_csr(P), x, torch.tensor(b0, device="cuda")))
    ref = x0.copy()
    for rev in (False, True):
        assert rc.executeFunction(fid, rev) == 0
        _walk(ri.GS, mode == ri.SWEEP_LEAF, rc, rev, P, P.val, ref, b0, np.float64)
    np.testing.assert_array_equal(x.cpu().numpy(), ref)


@pytest.mark.gpu
def test_kaczmarz_with_a_column_named_twice(mats):
    A = mats["lap7_16"]
    rc = ri.Interface(A.n, 16, ri.TWO, A.row_ptr, A.col, symm_hint=True)
    assert rc.RACEColor() == 0
    rc.setSweepMode(ri.SWEEP_WAVE)
    P = A.permuted(rc.getPerm(), rc.getInvPerm())
    r = int(np.argmax(np.diff(P.row_ptr) >= 4))
    s = int(P.row_ptr[r])
    P.col[s + 2] = P.col[s + 1]  # within the colored pattern
    x0, b0 = matgen.uniform_vector(A.n, 0), matgen.uniform_vector(A.n, 1)
    x = torch.tensor(x0, device="cuda")
    fid = rc.registerFunction(ri.KACZ, ri.Operands(ri.DeviceCsr.from_csr(P), x, torch.tensor(b0, device="cuda")))
    assert fid >= 0
    pp, lo, hi = rc.getPhases(False)
    ref, b = x0.copy(), b0.copy()
    for a, z in zip(lo, hi):
        orc.run_kernel(orc.K_KACZ, int(a), int(z), P, ref, b)
    assert rc.executeFunction(fid) == 0
    np.testing.assert_array_equal(x.cpu().numpy(), ref)
