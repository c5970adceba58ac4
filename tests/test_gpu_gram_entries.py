"""Each entry of the FP64 Gram (csrc/dense64.cu k_syrk_digits) to what FP64 sums give for it,
also where a column's largest entries meet small ones of the other column: spikes of 2^10 to
2^60 over entries of size one in rows where the others are zero, small or ordinary, weighted
rows, entries spread over 40 powers of two, columns without a common row, and K slices
of up to 30,000 rows.

Bound: K rounding errors of a sum are at most 2^-53 of a partial sum of |x_ki x_kj| each; taken
as independent, 8 sqrt(K) 2^-53 S_ij holds with probability 1 - 2 exp(-32) (Higham, Mary, SIAM
J. Sci. Comput. 41, 2019), S = |A|^T |A|.  The digit sums' own worst case is less: in units
of a 32-row block's powers of two 32 (7 * 2^14 * 256^-10 * 2^2.01 + 2^-63) <= 2^-55.8, with nb units whose
root of squares is at most 97 S: below sqrt(nb) 2^-49 S <= 2.9 sqrt(K) 2^-53 S, and one rounding."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gram(cg, tmp_path, torch, A):
    synth = importlib.import_module("chimes_lsq-myllfork_gb300.synth")
    sess = cg.Session(cg.Model(synth.make_workload("water-2b", str(tmp_path), nframes=1, seed=3)), 0)
    n = A.shape[1]
    dA, db = torch.from_numpy(A).cuda(), torch.zeros(A.shape[0], dtype=torch.float64, device="cuda")
    G = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    h = torch.zeros(n, dtype=torch.float64, device="cuda")
    sess.gram(cg.CG_FP64, dA.data_ptr(), n, A.shape[0], n, db.data_ptr(), 0, G.data_ptr(), h.data_ptr())
    torch.cuda.synchronize()
    return G.cpu().numpy()


def _check(A, G, pairs):
    K = A.shape[0]
    for i, j in pairs:
        x, y = A[:, i].astype(np.longdouble), A[:, j].astype(np.longdouble)
        want, S = (x * y).sum(), float((np.abs(x) * np.abs(y)).sum())
        assert abs(G[i, j] - want) <= 8 * np.sqrt(K) * 2.0**-53 * S, (i, j, float(G[i, j] - want) / (S + 1e-300))


def _pairs(rng, m, first, n=40):
    p = {(min(a, b), max(a, b)) for a, b in rng.integers(0, m, (n, 2))}
    return sorted(p | {(i, j) for i in first for j in range(m) if j >= i and (j % 7 == 0 or j < 8)})


@pytest.mark.parametrize("s", [10, 20, 30, 45, 60])
@pytest.mark.parametrize("K,m", [(2048, 150), (5000, 97)])
def test_spikes(cg, tmp_path, K, m, s):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(s + m)
    A = rng.standard_normal((K, m))
    rows = rng.choice(K, 6, replace=False)
    A[rows[:2], 1:] = 0.0            # two spikes of column 0 that meet zeros,
    A[rows[2:4], 1:] *= 2.0**-s      # two that meet small entries,
    A[rows[4:], 1:70] = 0.0          # and two that meet ordinary ones in some columns
    A[rows, 0] = 2.0**s
    A[rng.choice(K, 3), 3] = -(2.0**s)
    G = _gram(cg, tmp_path, torch, A)
    _check(A, G, _pairs(rng, m, [0, 3]))


def test_weighted_rows_and_wide_spread(cg, tmp_path):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(11)
    K, m = 3000, 140
    A = rng.standard_normal((K, m)) * np.exp2(rng.uniform(-40, 0, (K, m)))
    A[rng.random(K) < 0.02] *= 300.0
    A[: K // 2, 10:20] = 0.0         # columns without a common row
    A[K // 2:, 20:30] = 0.0
    G = _gram(cg, tmp_path, torch, A)
    assert np.all(G[10:20, 20:30] == 0.0)
    _check(A, G, _pairs(rng, m, [0, 12, 64], 60))


def test_long_slices_of_a_wide_matrix(cg, tmp_path):
    """Enough tiles that a CTA keeps all rows of its outputs."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(12)
    K, m = 30011, 2500
    A = rng.standard_normal((K, m), dtype=np.float32).astype(np.float64)
    rows = rng.choice(K, 12, replace=False)
    A[rows, ::5] *= 2.0**20
    A[rows, 1::5] = 0.0
    G = _gram(cg, tmp_path, torch, A)
    _check(A, G, _pairs(rng, m, [], 40) + [(0, 1), (5, 6), (0, 2), (0, 5), (1, 6), (64, 65), (2495, 2496)])


@pytest.mark.parametrize("scale", [2.0**-480, 2.0**480])
def test_range_of_exponents(cg, tmp_path, scale):
    """Entries near the ends of the exponents' range: sums far above the smallest normal number."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(13)
    A = rng.standard_normal((1500, 170)) * scale
    G = _gram(cg, tmp_path, torch, A)
    _check(A / scale, G / scale / scale, _pairs(rng, 170, [0]))


def test_infinite_entries_as_in_fp64_sums(cg, tmp_path):
    """Infinities give infinities of the right sign, or NaN where FP64 sums do."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(14)
    A = np.abs(rng.standard_normal((2000, 150))) + 0.1
    A[9, 100], A[11, 7] = np.inf, -np.inf
    A[9, 20] = 0.0
    G = np.triu(_gram(cg, tmp_path, torch, A))
    with np.errstate(invalid="ignore"):
        R = np.triu(A.T @ A)
    assert np.array_equal(np.isnan(G), np.isnan(R))
    assert np.array_equal(G == np.inf, R == np.inf) and np.array_equal(G == -np.inf, R == -np.inf)
