"""Many-body A rows as digit products on the tensor cores (csrc/tensor_rows.cu) against the
CPU oracle, where groups, chunks and grids end: owner groups of one to thousands of
clusters (8 a step, 16 a chunk), more than 512 clusters of a (frame, type) group, orders
that fill their padded grids in part, small cells (PERM_SCALE), and the row options.

Tolerances: FP64 1e-12 of the entry and of its column's scale, FP32 2e-5 of the column
scale, as for every other form of these rows."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = {
    "order5": ("water-3b", dict(nframes=1, order=(6, 5, 0))),
    "order7_energy_only": ("water-3b", dict(nframes=1, order=(6, 7, 0), fitstrs=None)),
    "dense_3body": ("water-3b", dict(nframes=1, smax=(5.0, 6.0, None))),
    "small_cell": ("chno-4b", dict(nframes=2, sizes=[9, 11], triclinic=False, order=(6, 8, 4))),
    "two_species": ("chno-4b", dict(nframes=3, sizes=[33, 90, 34], triclinic=False, species2=True, order=(6, 6, 4))),
    "diagonal_stress": ("chno-4b", dict(nframes=2, sizes=[35, 61], triclinic=False, fitstrs="true", fitener=False,
                                        order=(6, 8, 4))),
    "no_extra_rows": ("chno-4b", dict(nframes=1, sizes=[40], triclinic=False, fitstrs=None, fitener=False,
                                      order=(6, 8, 4))),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_rows_match_oracle(cg, oracle, tmp_path, name):
    synth = importlib.import_module("chimes_lsq-myllfork_gb300.synth")
    kind, over = CASES[name]
    fm = synth.make_workload(kind, str(tmp_path), seed=77, labels=False, **over)
    model = cg.Model(fm)
    frames = cg.Frames.read(model)
    sess = cg.Session(model, 0)
    O, _ = oracle.assemble(fm, nthreads=8)
    colmax = np.abs(O).max(axis=0)
    A = sess.assemble(frames, cg.CG_FP64)
    assert A.shape == O.shape
    err = np.abs(A - O)
    assert np.all(err <= 1e-12 * np.abs(O) + 1e-12 * colmax[None, :]), err.max()
    assert np.array_equal(A, sess.assemble(frames, cg.CG_FP64))   # bit-reproducible
    A32 = sess.assemble(frames, cg.CG_FP32).astype(np.float64)
    assert (np.abs(A32 - O) / (colmax[None, :] + 1e-300)).max() < 2e-5


def test_coincident_atoms_stay_visible(cg, tmp_path):
    """Two atoms at one place have no direction: the rows that the per-power form makes
    non-finite are non-finite here too, and the others agree."""
    synth = importlib.import_module("chimes_lsq-myllfork_gb300.synth")
    fm = synth.make_workload("water-3b", str(tmp_path), nframes=1, seed=5, labels=False)
    model = cg.Model(fm)
    rng = np.random.default_rng(3)
    xyz, types, cell, _ = synth.water_frame(rng, 40, 12.0, 0.1)
    xyz[5] = xyz[1]
    frames = cg.Frames.from_arrays(model, [len(xyz)], types, xyz, cell.reshape(1, 9))
    sess = cg.Session(model, 0)
    A = sess.assemble(frames, cg.CG_FP64)
    sess.tune("force_range", 0)
    B = sess.assemble(frames, cg.CG_FP64)
    bad = ~np.isfinite(B)
    assert bad.any() and not np.isfinite(A[bad]).any()
    n3 = 3 * len(xyz)
    rows = ~bad[:n3].any(axis=1)
    assert rows.sum() > n3 // 3
    scale = np.abs(B[:n3][rows]).max(axis=0) + 1e-300
    d = np.abs(A[:n3][rows] - B[:n3][rows])
    assert np.nanmax(d / scale[None, :]) <= 1e-12
