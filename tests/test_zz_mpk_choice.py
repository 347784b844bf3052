"""RACE_MPK_AUTO times both schedules and may settle on their first runs. A
kernel that the process has not used yet is loaded at its first launch, so the
code of both must be loaded before the first event (seen by a preloaded
counter of the runtime's calls), and the choice for a small matrix, whose
wavefront is about four times slower, is the same whatever ran before."""
import os
import shutil
import subprocess
import sys
import textwrap

import pytest

COUNTER = textwrap.dedent("""
    #define _GNU_SOURCE
    #include <dlfcn.h>
    static int loads = 0, loadsBeforeEvent = -1;
    int cudaFuncGetAttributes(void *attributes, const void *kernel) {
        ++loads;
        return ((int (*)(void *, const void *))dlsym(RTLD_NEXT, "cudaFuncGetAttributes"))(attributes, kernel);
    }
    int cudaEventRecord(void *event, void *stream) {
        if (loadsBeforeEvent < 0) loadsBeforeEvent = loads;
        return ((int (*)(void *, void *))dlsym(RTLD_NEXT, "cudaEventRecord"))(event, stream);
    }
    void start(void) { loads = 0; loadsBeforeEvent = -1; }
    int loaded(void) { return loadsBeforeEvent; }
""")
CHILD = textwrap.dedent("""
    import ctypes as C
    import os
    import sys
    import torch
    from race_gb300 import interface as ri, matgen

    calls = C.CDLL(os.environ["LD_PRELOAD"])

    def choice(A, power, vdt):
        rc = ri.Interface(A.n, 1, ri.POWER, A.row_ptr, A.col, symm_hint=True)
        assert rc.RACEColor(power, 300e6) == 0
        P = A.permuted(rc.getPerm(), rc.getInvPerm())
        x = torch.zeros((power + 1) * A.n, dtype=torch.float64, device="cuda")
        x[:A.n] = torch.tensor(matgen.uniform_vector(A.n, 1), device="cuda")
        fid = rc.registerFunction(ri.MPK, ri.Operands(ri.DeviceCsr.from_csr(P, "cuda", vdt), x), power=power)
        calls.start()
        assert rc.executeFunction(fid) == 0
        return rc.getMpkLayout(fid)["schedule"], calls.loaded()

    vdt = getattr(torch, sys.argv[1])
    first = choice(matgen.laplace3d_7pt(57), 4, vdt)  # the striding kernel of larger matrices
    small = matgen.laplace3d_7pt(24)
    got = [choice(small, 4, vdt) for _ in range(3)]
    assert [g[0] for g in got] == ["sweeps"] * 3, got
    assert all(g[1] == 2 for g in [first, *got]), (first, got)
    print("loaded first")
""")


@pytest.mark.gpu
@pytest.mark.parametrize("vdt", ["float64", "float32", "bfloat16"])
def test_choice_does_not_depend_on_what_ran_before(vdt, tmp_path):
    if not shutil.which("gcc"):
        pytest.skip("no gcc")
    src, so = tmp_path / "calls.c", tmp_path / "calls.so"
    src.write_text(COUNTER)
    subprocess.check_call(["gcc", "-shared", "-fPIC", "-O1", str(src), "-o", str(so), "-ldl"])
    r = subprocess.run([sys.executable, "-c", CHILD, vdt], capture_output=True, text=True, timeout=300,
                       env={**os.environ, "LD_PRELOAD": str(so)})
    assert r.returncode == 0 and "loaded first" in r.stdout, r.stdout + r.stderr
