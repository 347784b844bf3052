"""Operand types that no sweep kernel exists for are refused, by every kernel
and mode, before anything is launched: vectors that are neither FP64 nor FP32."""
import ctypes as C

import pytest

from race_gb300 import _lib, matgen

torch = pytest.importorskip("torch")

from race_gb300 import interface as ri  # noqa: E402


@pytest.mark.gpu
@pytest.mark.parametrize("kernel", [ri.SPMV, ri.SPMTV, ri.SYMMSPMV, ri.GS, ri.KACZ])
@pytest.mark.parametrize("vec_type", [ri.VAL_BF16, 7])
def test_unknown_vector_types_are_refused(kernel, vec_type):
    A = matgen.laplace3d_7pt(6)
    rc = ri.Interface(A.n, 4, ri.TWO, A.row_ptr, A.col, symm_hint=True)
    assert rc.RACEColor() == 0
    P = A.permuted(rc.getPerm(), rc.getInvPerm())
    x, b = (torch.full((A.n,), v, dtype=torch.float64, device="cuda") for v in (1.0, 2.0))
    args = ri.Operands(ri.DeviceCsr.from_csr(P, "cuda", torch.bfloat16), x, b)
    ops, fid = args.to_c(), C.c_int(-1)
    ops.vec_type = vec_type
    code = _lib.lib().race_register_function(rc._h, kernel, C.byref(ops), 1, C.byref(fid))
    if code == 0:
        for mode in (ri.SWEEP_AUTO, ri.SWEEP_WAVE, ri.SWEEP_LEAF):
            rc.setSweepMode(mode)
            for rev in (False, True):
                assert rc.executeFunction(fid.value, rev) == _lib.RACE_ERR_INVALID_ARG
    else:
        assert code == _lib.RACE_ERR_INVALID_ARG
    torch.cuda.synchronize()
    assert bool((x == 1.0).all()) and bool((b == 2.0).all())
