"""Neighbour lists (csrc/geom.cu k_neigh) with more than 65,536 images of the cell: a cell
0.26 A thick and 20 image layers (68,921 images), whose last images along the short edge are
still within the cut-off, against a plain FP64 enumeration and the CPU oracle's rows.
Pair counts are equal; FP64 rows to 1e-12 of their column's largest entry."""
import importlib
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3])
def test_pairs_beyond_65536_images(cg, oracle, tmp_path, n):
    synth = importlib.import_module("chimes_lsq-myllfork_gb300.synth")
    layers, cut, smin = 20, 5.0, 0.8
    cell = np.diag([0.26, 6.0, 6.5])
    rng = np.random.default_rng(n)
    x = rng.uniform(0.1, 0.9, (n, 3)) @ cell
    types = [k % 2 for k in range(n)]
    fm = str(tmp_path / "fm_setup.in")
    with open(tmp_path / "traj.xyzf", "w") as f:
        f.write(f"{n}\n" + " ".join(f"{v:.6f}" for v in np.diag(cell)) + "\n")
        for t, r in zip(types, x):
            f.write("OH"[t] + " " + " ".join(f"{v:.17g}" for v in r) + " 0.0 0.0 0.0\n")
    synth.write_fm_setup(fm, str(tmp_path / "traj.xyzf"), 1, ["O", "H"], [16.0, 1.0], 6, 0, 0, smin, cut, 1.4,
                         nlayers=layers)
    model = cg.Model(fm)
    sess = cg.Session(model, 0)
    A = sess.assemble(cg.Frames.read(model), cg.CG_FP64)
    want, last = 0, 0
    r1 = range(-layers, layers + 1)
    side = 2 * layers + 1
    for n1, n2, n3 in itertools.product(r1, r1, r1):
        if abs(n2) > 1 or abs(n3) > 1:
            continue
        d = np.linalg.norm(x[None] + np.array([n1, n2, n3]) @ cell - x[:, None], axis=2)
        hits = int(((d < cut) & (d > smin)).sum())
        want += hits
        if ((n1 + layers) * side + n2 + layers) * side + n3 + layers > 65536:
            last += hits
    assert last > 0                       # pairs with images beyond 2^16 exist
    assert sess.last_counts()["pairs"] == want
    O, _ = oracle.assemble(fm, nthreads=8)
    assert A.shape == O.shape
    assert np.all(np.abs(A - O) <= 1e-12 * np.abs(O).max(axis=0)[None, :])
