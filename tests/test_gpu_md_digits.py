"""The FP64 MD contraction on the tensor cores (csrc/md_tensor.cu) against the CPU oracle:
tiles of 64 clusters filled by one cluster to many, 16-cluster row tiles, several frames
in one call, small cells (PERM_SCALE), coefficients of very different size, and lists
reused over steps (the serving loop, against one force call's first step).  Tolerance: 1e-10 of
max |F| and of each scalar's largest value, as for the other FP64 form."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,species2,spread", [((6,), True, 0.0), ((9, 12, 40), False, 0.0), ((33, 64, 17), True, 6.0),
                                                   ((220,), False, 3.0)])
def test_forces_match_oracle(cg, oracle, tmp_path, sizes, species2, spread):
    synth = importlib.import_module("chimes_lsq-myllfork_gb300.synth")
    fm = synth.make_workload("chno-4b", str(tmp_path), nframes=len(sizes), seed=len(sizes), sizes=list(sizes),
                             triclinic=False, species2=species2, labels=False)
    model = cg.Model(fm)
    names = ["C", "H"] if species2 else ["C", "H", "N", "O"]
    nat, types, xyz, cell = synth.frames_arrays(str(tmp_path / "traj.xyzf"), len(sizes), names)[:4]
    rng = np.random.default_rng(7)
    x = 1e-3 * rng.standard_normal(model.ncols) * np.exp(spread * rng.standard_normal(model.ncols))
    frames = cg.Frames.from_arrays(model, nat, types, xyz, cell).independent()
    sess = cg.Session(model, 0)
    sess.md_setup(x)
    F, S = sess.md_force(frames)
    Fo, So = oracle.md_force(fm, nat, types, xyz, cell, x)
    assert np.abs(F - Fo).max() <= 1e-10 * np.abs(Fo).max()
    assert np.all(np.abs(S - So) <= 1e-10 * np.abs(So).max(axis=0, keepdims=True) + 1e-10 * np.abs(So).max(axis=1, keepdims=True))
    # coefficients that are not finite stay visible
    c = model.columns()
    x[c["n2b"] + c["n3b"]: c["n2b"] + c["n3b"] + c["n4b"]] = np.nan
    sess.md_setup(x)
    E = sess.md_force(frames)[1][:, 0]
    assert sess.md_last_counts()["quads"] == 0 or not np.isfinite(E).all()
