"""Issue order and item sizes of batches: members of very different sizes
(from one row), powers and level groups, at item sizes from a single pass of a
warp to several passes, against the oracle's chains bit for bit."""
import numpy as np
import pytest

from oracle import oracle as orc
from race_gb300 import matgen

torch = pytest.importorskip("torch")

from race_gb300 import interface as ri  # noqa: E402


@pytest.mark.gpu
@pytest.mark.parametrize("vdt,nrhs", [("float64", 1), ("float64", 32), ("float32", 2), ("float32", 8),
                                      ("float32", 32), ("bfloat16", 16)])
@pytest.mark.parametrize("big", [False, True])
def test_batch_members_of_any_size(vdt, nrhs, big):
    mats = [matgen.aniso2d(1, 1, 5), matgen.aniso2d(3, 2, 9), matgen.laplace3d_7pt(9), matgen.aniso2d(33, 31, 9),
            matgen.powerlaw_chung_lu(700, seed=4), matgen.aniso2d(150, 90, 5)]
    if big:  # enough rows that several passes make an item
        mats.insert(3, matgen.aniso2d(700, 300 if nrhs > 4 else 900, 5))
    xdt = torch.float64 if vdt == "float64" else torch.float32
    batch, members = ri.Batch(), []
    for i, A in enumerate(mats):
        p = 1 + (3 * i) % 5
        rc = ri.Interface(A.n, 1, ri.POWER, A.row_ptr, A.col, symm_hint=True)
        assert rc.RACEColor(p, 1e9 if i % 2 else 2e4, 2.0) == 0  # one level group, and many
        P = A.permuted(rc.getPerm(), rc.getInvPerm())
        X0 = matgen.uniform_block(A.n, nrhs, seed=i).astype(np.float64 if vdt == "float64" else np.float32)
        dm = ri.DeviceCsr.from_csr(P, "cuda", getattr(torch, vdt))
        x = torch.zeros((p + 1) * A.n * nrhs, dtype=xdt, device="cuda")
        x[: A.n * nrhs] = torch.tensor(X0.reshape(-1), device="cuda")
        fid = rc.registerMpkBlock(ri.Operands(dm, x), p, nrhs)
        assert fid >= 0
        batch.add(rc, fid)
        members.append((rc, fid, P, p, X0, dm, x))
    batch.graphLaunch()
    assert batch.getStatus() == 0
    for alone in (False, True):
        for rc, fid, P, p, X0, dm, x in members:
            if alone:
                x[P.n * nrhs:] = 0
                assert rc.executeFunction(fid) == 0
            val = None if vdt == "float64" else dm.val.float().cpu().numpy()
            ref = orc.mpk_block(P, X0, p) if val is None else orc.mpk_block(P, X0, p, val=val)
            np.testing.assert_array_equal(x.cpu().numpy().reshape(p + 1, P.n, nrhs), ref)
