"""Digit-product rows (csrc/tensor_rows.cu) under the options of the input file, at the orders
that take them (3-body 8, 4-body 4): the smooth cut-off TERSOFF, the transforms INVRSE_R and
NONE, cut-offs of single cluster types (unequal along a cluster's slots), excluded types
with and without the hierarchical exclusion, and the forms below s_min.  FP64 rows against
the CPU oracle, 1e-12 of the entry and of its column's scale as for every other form of them,
and the FP64 forces of the MD contraction at the same orders to 1e-10 of the largest."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RAISE = "\nSPECIAL 3B S_MINIM: ALL 1.3\n\nSPECIAL 4B S_MINIM: ALL 1.3\n\n# FCUTTYP #"
OPTIONS = {
    "tersoff": [("\tCUBIC", "\tTERSOFF 0.5")],
    "tersoff_steep": [("\tCUBIC", "\tTERSOFF 0.05")],
    "invrse_r": [("\tMORSE", "\tINVRSE_R")],
    "no_transform": [("\tMORSE", "\tNONE")],
    "specific": [("SPECIAL 3B S_MAXIM: ALL 4.0",
                  "SPECIAL 3B S_MAXIM: SPECIFIC 2\nCCCCCC CC CC CC 4.2 4.2 4.2\nCCCHCH CC CH CH 3.9 3.6 3.6\n\n"
                  "SPECIAL 3B S_MINIM: SPECIFIC 1\nCHCHHH CH CH HH 1.1 1.1 1.2"),
                 ("SPECIAL 4B S_MAXIM: ALL 3.5",
                  "SPECIAL 4B S_MAXIM: SPECIFIC 2\nCCCCCCCCCCCC CC CC CC CC CC CC 3.6 3.6 3.6 3.6 3.6 3.6\n"
                  "CCCCCHCCCHCH CC CC CH CC CH CH 3.4 3.4 3.1 3.4 3.1 3.1")],
    "exclude": [("# ENDFILE #", "EXCLUDE 3B INTERACTION: 1\nC C H\n\nEXCLUDE 4B INTERACTION: 2\nC C C H\nH H H H\n\n"
                                "# ENDFILE #")],
    "zero_deriv": [("# PAIRTYP #", "# CHEBYFIX #\n\tZERO_DERIV\n# PAIRTYP #"), ("# FCUTTYP #", RAISE)],
    "constant_deriv": [("# PAIRTYP #", "# CHEBYFIX #\n\tCONSTANT_DERIV\n# PAIRTYP #"), ("# FCUTTYP #", RAISE)],
    "smooth": [("# PAIRTYP #", "# CHEBYFIX #\n\tSMOOTH 0.02\n# PAIRTYP #"), ("# FCUTTYP #", RAISE)],
}


def _patched(synth, tmp_path, name):
    sizes = [24, 50] if name == "specific" else [60, 110]   # (its other types reach to 5 A: many quadruplets)
    fm = synth.make_workload("chno-4b", str(tmp_path), nframes=2, seed=91, labels=False, sizes=sizes,
                             triclinic=False, species2=True, order=(6, 8, 4))
    text = open(fm).read()
    for old, new in OPTIONS[name]:
        assert text.count(old) == 1, old
        text = text.replace(old, new)
    open(fm, "w").write(text)
    return fm


@pytest.mark.parametrize("name", sorted(OPTIONS))
def test_rows_match_oracle(cg, oracle, tmp_path, name):
    synth = importlib.import_module("chimes_lsq-myllfork_gb300.synth")
    fm = _patched(synth, tmp_path, name)
    model = cg.Model(fm)
    sess = cg.Session(model, 0)
    A = sess.assemble(cg.Frames.read(model), cg.CG_FP64)
    counts = sess.last_counts()
    assert counts["triplets"] > 0 and counts["quads"] > 0
    O, _ = oracle.assemble(fm, nthreads=8)
    assert A.shape == O.shape
    assert np.all(np.abs(A - O) <= 1e-12 * np.abs(O) + 1e-12 * np.abs(O).max(axis=0)[None, :])


@pytest.mark.parametrize("name", sorted(OPTIONS))
def test_forces_match_oracle(cg, oracle, tmp_path, name):
    synth = importlib.import_module("chimes_lsq-myllfork_gb300.synth")
    fm = _patched(synth, tmp_path, name)
    model = cg.Model(fm)
    nat, types, xyz, cell = synth.frames_arrays(str(tmp_path / "traj.xyzf"), 2, ["C", "H"])[:4]
    x = 1e-3 * np.random.default_rng(5).standard_normal(model.ncols)
    sess = cg.Session(model, 0)
    sess.md_setup(x)
    F, _ = sess.md_force(cg.Frames.from_arrays(model, nat, types, xyz, cell).independent())
    Fo, _ = oracle.md_force(fm, nat, types, xyz, cell, x)
    assert np.abs(F - Fo).max() <= 1e-10 * np.abs(Fo).max()


def test_hierarchical_exclusion(cg, oracle, tmp_path):
    """Water rows without the columns of excluded 1- and 2-body terms."""
    synth = importlib.import_module("chimes_lsq-myllfork_gb300.synth")
    fm = synth.make_workload("water-3b", str(tmp_path), nframes=2, seed=19, nmol=24, L=8.96, order=(8, 8, 0),
                             fitstrs="ALL", fitener=True)
    text = open(fm).read()
    for old, new in (("# NLAYERS #", "# HIERARC #\n\ttrue\n# NLAYERS #"),
                     ("# ENDFILE #", "EXCLUDE 1B INTERACTION: 1\nH\n\nEXCLUDE 2B INTERACTION: 1\nO H\n\n# ENDFILE #")):
        assert text.count(old) == 1
        text = text.replace(old, new)
    open(fm, "w").write(text)
    model = cg.Model(fm)
    sess = cg.Session(model, 0)
    A = sess.assemble(cg.Frames.read(model), cg.CG_FP64)
    O, _ = oracle.assemble(fm, nthreads=8)
    assert A.shape == O.shape
    assert np.all(np.abs(A - O) <= 1e-12 * np.abs(O) + 1e-12 * np.abs(O).max(axis=0)[None, :])


def test_bases_continued_below_s_min_take_the_fp64_form(cg, tmp_path):
    """CONSTANT_DERIV's bases grow without bound below s_min, and digits under a group's largest
    magnitude would hold the other clusters' small columns less accurately: the rows are those
    of the FP64 range form."""
    synth = importlib.import_module("chimes_lsq-myllfork_gb300.synth")
    fm = _patched(synth, tmp_path, "constant_deriv")
    model = cg.Model(fm)
    frames = cg.Frames.read(model)
    sess = cg.Session(model, 0)
    A = sess.assemble(frames, cg.CG_FP64)
    sess.tune("force_range", 2)
    assert np.array_equal(A, sess.assemble(frames, cg.CG_FP64))
