"""A pivot below the normal numbers (2^-1022), whose reciprocal is not finite, is a positive
pivot like any other: G = D C D with one d_k = 1e-155 has the factor D chol(C).

Bound: G_kk = 1e-310 keeps 44 bits, so the pivot's relative error is 2^-44 times the condition
of C's Schur complement (below 50 here), and it enters the other entries of column k; the
row's entries of 1e-155 are normal numbers.  1e-10 of the scaled entry's row norm (one)."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n,k", [(1, 0), (20, 3), (100, 15), (100, 64), (300, 17), (300, 130), (300, 299)])
def test_factor(cg, tmp_path, n, k, mode):
    torch = pytest.importorskip("torch")
    synth = importlib.import_module("chimes_lsq-myllfork_gb300.synth")
    sess = cg.Session(cg.Model(synth.make_workload("water-2b", str(tmp_path), nframes=1)), 0)
    rng = np.random.default_rng(n + k)
    X = rng.standard_normal((4 * n + 8, n))
    C = X.T @ X
    C /= np.sqrt(np.outer(np.diag(C), np.diag(C)))
    D = np.ones(n)
    D[k] = 1e-155
    G = D[:, None] * C * D[None, :]
    assert 0.0 < G[k, k] < 2.0**-1022
    dG = torch.from_numpy(G).cuda()
    dL = torch.empty((n, n), dtype=torch.float64, device="cuda")
    sess.tune("cholesky_tensor_updates", mode)
    used = sess.cholesky(dG.data_ptr(), n, 0.0, dL.data_ptr())
    torch.cuda.synchronize()
    assert used == 0.0
    L = np.triu(dL.cpu().numpy()).T     # column-major L: the row-major upper triangle is L^T
    want = np.linalg.cholesky(C)
    assert np.abs(L / D[:, None] - want).max() <= 1e-10
