"""Shared memory beyond 48 KB is granted to a kernel for one device, so every
network must ask for its own: a second network of the process repeats the
first one's requests (it may live on another GPU). The requests are counted by
a preloaded cudaFuncSetAttribute that passes them on."""
import os
import shutil
import subprocess
import sys
import textwrap

import pytest

COUNTER = textwrap.dedent("""
    #define _GNU_SOURCE
    #include <dlfcn.h>
    static int count = 0;
    int cudaFuncSetAttribute(const void *kernel, int attribute, int value) {
        ++count;
        return ((int (*)(const void *, int, int))dlsym(RTLD_NEXT, "cudaFuncSetAttribute"))(kernel, attribute, value);
    }
    int requests(void) { return count; }
""")
CHILD = textwrap.dedent("""
    import ctypes as C
    import os
    import torch
    from race_gb300 import tuner

    requests = C.CDLL(os.environ["LD_PRELOAD"]).requests

    def passes(dims, batch):
        before, net = requests(), tuner.Mlp(*dims, seed=1)
        X, T = torch.ones((batch, dims[0]), device="cuda"), torch.ones((batch, dims[3]), device="cuda")
        for _ in range(2):
            net.forward(X)
            net.loss_grad(X, T)
        return requests() - before

    for dims, batch, kernels in (((34, 128, 3, 1), 239, 2), ((8, 300, 2, 3), 2000, 2)):  # resident; tiles
        got = [passes(dims, batch) for _ in range(3)]
        assert got == [kernels] * 3, (dims, got)
    print("every network asked")
""")


@pytest.mark.gpu
def test_every_network_asks_for_its_shared_memory(tmp_path):
    if not shutil.which("gcc"):
        pytest.skip("no gcc")
    src, so = tmp_path / "counter.c", tmp_path / "counter.so"
    src.write_text(COUNTER)
    subprocess.check_call(["gcc", "-shared", "-fPIC", "-O1", str(src), "-o", str(so), "-ldl"])
    r = subprocess.run([sys.executable, "-c", CHILD], capture_output=True, text=True, timeout=300,
                       env={**os.environ, "LD_PRELOAD": str(so)})
    assert r.returncode == 0 and "every network asked" in r.stdout, r.stdout + r.stderr
