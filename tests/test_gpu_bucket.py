"""The per-frame bucket sort (csrc/geom.cu k_bucket) is stable whatever the number of CTAs
per frame: FP32 rows, whose sums run in bucket order, of a frame in batches for each
number of CTAs (8, 4, 2, 1) equal those of the frame alone bit for bit.  Frames of 1 to 90
atoms: none, few and many items per warp."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = (1, 3, 33, 90, 64)


@pytest.mark.parametrize("nframes", [2, 45, 100, 170])
def test_rows_do_not_depend_on_the_batch(cg, tmp_path, nframes):
    synth = importlib.import_module("chimes_lsq-myllfork_gb300.synth")
    fm = str(tmp_path / "fm_setup.in")
    synth.write_fm_setup(fm, "traj.xyzf", nframes, ["O", "H"], [16.0, 1.0], 6, 4, 2, 0.8, 5.0, 3.0)
    model = cg.Model(fm)
    sess = cg.Session(model, 0)
    rng = np.random.default_rng(7)
    geo = []
    for n in SIZES:
        L = max((n / 0.05) ** (1 / 3), 6.0)
        geo.append((n, rng.integers(0, 2, n), rng.uniform(0, L, (n, 3)), (np.eye(3) * L).reshape(9)))

    def rows(idx):
        fr = cg.Frames.from_arrays(model, [geo[i][0] for i in idx], np.concatenate([geo[i][1] for i in idx]),
                                   np.concatenate([geo[i][2] for i in idx]), np.stack([geo[i][3] for i in idx]))
        return sess.assemble(fr.independent(), cg.CG_FP32)

    idx = [k % len(SIZES) for k in range(nframes)]
    A = rows(idx)
    alone = [rows([i]) for i in range(len(SIZES))]
    assert any(a.any() for a in alone)
    assert A.shape[0] == sum(alone[i].shape[0] for i in idx)
    r = 0
    for i in idx:
        m = 3 * geo[i][0]
        np.testing.assert_array_equal(A[r:r + m], alone[i][:m])
        r += alone[i].shape[0]
