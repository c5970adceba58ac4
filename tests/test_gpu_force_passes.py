"""Many-body force rows by passes over several cluster types (csrc/assemble.cu k_force_rg,
k_force_pt) at orders whose loops run at run time and at the usual one, with types of no, a
few and more than one pass of clusters (32 in FP32, 16 in FP64).

Tolerances: FP64 1e-12 of the entry and of its column's scale, FP32 2e-5 of the column
scale, as for every other form of these rows."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [0, 1, 2])
@pytest.mark.parametrize("o3,o4", [(2, 2), (4, 3), (9, 2), (8, 4)])
def test_rows_match_oracle(cg, oracle, tmp_path, o3, o4, form):
    synth = importlib.import_module("chimes_lsq-myllfork_gb300.synth")
    fm = synth.make_workload("chno-4b", str(tmp_path), seed=o3, labels=False, nframes=2, sizes=[21, 70],
                             triclinic=False, order=(4, o3, o4))
    model = cg.Model(fm)
    frames = cg.Frames.read(model)
    sess = cg.Session(model, 0)
    sess.tune("force_range", form)
    O, _ = oracle.assemble(fm, nthreads=8)
    colmax = np.abs(O).max(axis=0)
    A = sess.assemble(frames, cg.CG_FP64)
    assert np.all(np.abs(A - O) <= 1e-12 * np.abs(O) + 1e-12 * colmax[None, :])
    A32 = sess.assemble(frames, cg.CG_FP32).astype(np.float64)
    assert (np.abs(A32 - O) / (colmax[None, :] + 1e-300)).max() < 2e-5
