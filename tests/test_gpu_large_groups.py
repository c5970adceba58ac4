"""Digit-product rows (csrc/tensor_rows.cu) of an owner with more than 2^16 clusters of one
type: a slab of three atoms of one element 1 A apart, repeated along y and z (7 layers of
images), vacuum along x, 3-body cut-off 6.5 A with the sharp TERSOFF cut-off and no transform,
so that most of an atom's 270,000 incidences are near the group's largest magnitude and their
share sum passes 2^32.  Checked against the CPU oracle and the range form.

Tolerance: FP64 sums of n = 3e5 terms differ by up to n 2^-53 = 3e-11 of the terms'
magnitudes, which add up to a few times the column's largest entry (the neighbours of an
outer atom lie on one side): 1e-9 of it.  An output that overflowed is wrong by its size."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_more_than_65536_clusters_of_a_type(cg, oracle, tmp_path):
    synth = importlib.import_module("chimes_lsq-myllfork_gb300.synth")
    fm = str(tmp_path / "fm_setup.in")
    with open(tmp_path / "traj.xyzf", "w") as f:
        f.write("3\n12.0 1.0 1.0\n")
        for x in (4.0, 5.0, 6.0):
            f.write(f"O {x} 0.5 0.5 0.0 0.0 0.0\n")
    synth.write_fm_setup(fm, str(tmp_path / "traj.xyzf"), 1, ["O"], [16.0], 5, 5, 0, 0.8, 6.5, 1.4, smax3=6.5, nlayers=7)
    text = open(fm).read()
    assert "\tMORSE\n" in text and "\tCUBIC\n" in text
    open(fm, "w").write(text.replace("\tMORSE\n", "\tNONE\n").replace("\tCUBIC\n", "\tTERSOFF 0.02\n"))
    model = cg.Model(fm)
    frames = cg.Frames.read(model)
    sess = cg.Session(model, 0)
    A = sess.assemble(frames, cg.CG_FP64)
    assert sess.last_counts()["triplets"] > 3 * 65536
    sess.tune("force_range", 2)
    B = sess.assemble(frames, cg.CG_FP64)
    O, _ = oracle.assemble(fm, nthreads=8)
    scale = np.abs(O).max(axis=0)[None, :]
    assert np.all(np.abs(A - O) <= 1e-9 * scale)
    assert np.all(np.abs(B - O) <= 1e-9 * scale)
