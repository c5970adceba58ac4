"""The FP64 Gram as digit products (csrc/dense64.cu k_syrk_digits) against extended
precision, at tile and chunk edges: row counts around 16 and 32, column counts around 64,
K slices added atomically and single slices, columns of very different size, a zero
column, a column with one spike, and a non-finite entry.

Bound, in units of the columns' largest entries m_i m_j.  Entries are scaled to
X = x 2^(63 - e) with 2^e <= 2.01 m: rounding X costs a term 2 * 2.01 * 2^-64 <= 2^-61.9,
the digit pairs that are not formed 7 * 2^14 * 256^-10 * (2 * 2.01)^2 <= 2^-59.1.  Every
32 rows a value is rounded to 2^-(56 + up) of the scaled product, up = min(8, 9 -
ceil(log2 rows)): half of that times (2 * 2.01)^2.  The conversion and the additions to G
add 2^-51 of |G|.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gram(cg, sess, torch, A, b):
    n = A.shape[1]
    dA, db = torch.from_numpy(A).cuda(), torch.from_numpy(b).cuda()
    G = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    h = torch.zeros(n, dtype=torch.float64, device="cuda")
    sess.gram(cg.CG_FP64, dA.data_ptr(), n, A.shape[0], n, db.data_ptr(), 0, G.data_ptr(), h.data_ptr())
    torch.cuda.synchronize()
    return G.cpu().numpy(), h.cpu().numpy()


@pytest.mark.parametrize("K,m", [(4097, 100), (1000, 201), (33, 1111), (9600, 65), (16, 1601), (20000, 64)])
def test_matches_extended_precision(cg, tmp_path, K, m):
    torch = pytest.importorskip("torch")
    import importlib
    synth = importlib.import_module("chimes_lsq-myllfork_gb300.synth")
    sess = cg.Session(cg.Model(synth.make_workload("water-2b", str(tmp_path), nframes=1, seed=3)), 0)
    rng = np.random.default_rng(K + m)
    A = rng.standard_normal((K, m)) * np.exp(3.0 * rng.standard_normal(m))
    A[rng.random((K, m)) < 0.3] = 0.0
    A[:, m // 2] = 0.0
    A[K // 3, m - 1] = 1.0e6 * np.abs(A[:, m - 1]).max() + 1.0
    b = rng.standard_normal(K)
    G, h = _gram(cg, sess, torch, A, b)
    Q = A.astype(np.longdouble)
    sel = np.unique(np.concatenate([rng.integers(0, m, 40), [0, m // 2, m - 1, min(63, m - 1), min(64, m - 1)]]))
    R = (Q[:, sel].T @ Q).astype(np.float64)   # rows `sel` of G
    mx = np.abs(A).max(axis=0)
    up_bits = min(8, 9 - int(np.ceil(np.log2(-(-K // 16) * 16))))
    unit = K * (2.0 ** -61.9 + 2.0 ** -59.1) + (K / 32 + 1) * 4.02 ** 2 * 2.0 ** -(57 + up_bits)
    tol = unit * np.outer(mx[sel], mx) + 2.0 ** -51 * np.abs(R)
    up = np.arange(m)[None, :] >= sel[:, None]
    assert np.all((np.abs(G[sel] - R) <= tol)[up])
    assert np.all(np.abs(h - (Q.T @ b.astype(np.longdouble)).astype(np.float64)) <= K * 2.0 ** -52 * (np.abs(A).T @ np.abs(b)))


@pytest.mark.parametrize("frac", [0.9940, 0.99415, 0.9945, 0.9961, 0.99999, 1.0])
def test_entries_just_below_a_power_of_two(cg, tmp_path, frac):
    """The scaled leading digit at the end of its range: every entry of a column frac times
    a power of two, both signs."""
    torch = pytest.importorskip("torch")
    import importlib
    synth = importlib.import_module("chimes_lsq-myllfork_gb300.synth")
    sess = cg.Session(cg.Model(synth.make_workload("water-2b", str(tmp_path), nframes=1, seed=3)), 0)
    rng = np.random.default_rng(2)
    A = np.where(rng.random((2048, 160)) < 0.5, -1.0, 1.0) * frac * np.exp2(rng.integers(-3, 4, 160))
    G, _ = _gram(cg, sess, torch, A, np.ones(2048))
    R = A.T @ A
    up = np.triu(np.ones(R.shape, bool))
    assert np.all((np.abs(G - R) <= 1e-12 * np.sqrt(np.outer(np.diag(R), np.diag(R))))[up])


def test_non_finite_columns(cg, tmp_path):
    torch = pytest.importorskip("torch")
    import importlib
    synth = importlib.import_module("chimes_lsq-myllfork_gb300.synth")
    sess = cg.Session(cg.Model(synth.make_workload("water-2b", str(tmp_path), nframes=1, seed=3)), 0)
    A = np.random.default_rng(1).standard_normal((2000, 150))
    A[7, 5], A[9, 100] = np.nan, np.inf
    G, _ = _gram(cg, sess, torch, A, np.ones(2000))
    bad = np.zeros(150, bool)
    bad[[5, 100]] = True
    up = np.triu(np.ones((150, 150), bool))
    assert np.array_equal(~np.isfinite(G) & up, (bad[:, None] | bad[None, :]) & up)


@pytest.mark.parametrize("n", [1, 63, 64, 65, 129, 820])
def test_gram_finish_mirrors_the_upper_triangle(cg, tmp_path, n):
    torch = pytest.importorskip("torch")
    import ctypes
    import importlib
    synth = importlib.import_module("chimes_lsq-myllfork_gb300.synth")
    sess = cg.Session(cg.Model(synth.make_workload("water-2b", str(tmp_path), nframes=1, seed=3)), 0)
    G = torch.randn((n, n), dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(n))
    U = torch.triu(G)
    assert cg.lib().cg_gram_finish(sess._h, ctypes.c_void_p(G.data_ptr()), n) == 0
    torch.cuda.synchronize()
    assert torch.equal(G, U + torch.triu(U, 1).T)
