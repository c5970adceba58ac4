"""Factor and solves at the edges of the 16-column steps, 64-column halves and 128-column
panels, and of the one-block and the chained substitution.

Bounds (Higham, Accuracy and Stability of Numerical Algorithms, theorems 10.3 and 8.5),
u = 2^-53: |L L^T - G|_ij <= c u sqrt(G_ii G_jj) and |L L^T x - h| <= c u |L| |L^T| |x|
with c = n + 1 and 2 n.  A factor of 4 and 8 more roundings cover the square-root-free
form, the reciprocals, and the digit products' dropped digits (below 2^-54 of the row
scales per panel).  The products are evaluated in long double."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 15, 16, 17, 63, 64, 65, 79, 127, 128, 129, 191, 192, 193, 255, 256, 257, 320, 385]


@pytest.fixture(scope="module")
def sess(cg, tmp_path_factory):
    import importlib
    synth = importlib.import_module("chimes_lsq-myllfork_gb300.synth")
    return cg.Session(cg.Model(synth.make_workload("water-2b", str(tmp_path_factory.mktemp("edges")), nframes=1)), 0)


def _matrix(n):
    rng = np.random.default_rng(n)
    X = rng.standard_normal((2 * n + 8, n)) * np.exp(rng.uniform(-9, 9, size=n))[None, :]
    return X.T @ X, rng.standard_normal(n)


def _factor(sess, torch, G, ridge, mode):
    n = G.shape[0]
    sess.tune("cholesky_tensor_updates", mode)
    dG, L = torch.from_numpy(G).cuda(), torch.full((n, n), float("nan"), dtype=torch.float64, device="cuda")
    try:
        return sess.cholesky(dG.data_ptr(), n, ridge, L.data_ptr()), L
    finally:
        sess.tune("cholesky_tensor_updates", 1)


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n", SIZES)
def test_factor_and_solves(cg, sess, n, mode):
    torch = pytest.importorskip("torch")
    G, h = _matrix(n)
    used, dL = _factor(sess, torch, G, 0.0, mode)
    assert used == 0.0
    dh, dx = torch.from_numpy(h).cuda(), torch.empty(n, dtype=torch.float64, device="cuda")
    sess.cholesky_solve(dL.data_ptr(), n, dh.data_ptr(), dx.data_ptr())
    torch.cuda.synchronize()
    U = np.triu(dL.cpu().numpy()).astype(np.longdouble)   # column-major L: the row-major upper triangle is L^T
    x = dx.cpu().numpy().astype(np.longdouble)
    unit = 4 * (n + 8) * 2.0**-53
    d = np.sqrt(np.diag(G))
    assert np.all(np.abs(U.T @ U - G) <= unit * np.outer(d, d))
    assert np.all(np.abs(U.T @ (U @ x) - h) <= 2 * unit * (np.abs(U).T @ (np.abs(U) @ np.abs(x))))


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n,bad", [(1, 0), (64, 63), (100, 64), (129, 128), (257, 200), (257, 256)])
def test_a_pivot_that_is_not_positive_raises_the_ridge(cg, sess, n, bad, mode):
    """A diagonal matrix with one entry of -0.5: the ridge grows tenfold from 0.01 to 1."""
    torch = pytest.importorskip("torch")
    G = np.diag(np.linspace(1.0, 2.0, n))
    G[bad, bad] = -0.5
    used, dL = _factor(sess, torch, G, 0.01, mode)
    assert used == pytest.approx(1.0)
    np.testing.assert_allclose(np.diag(dL.cpu().numpy()), np.sqrt(np.diag(G) + 1.0), rtol=4 * 2.0**-53)
