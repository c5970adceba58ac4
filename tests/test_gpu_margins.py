"""Pairs, triplets and quadruplets decided near their cut-offs (csrc/geom.cu): groups of four
atoms whose longest distance is a cut-off plus or minus 1e-9 to 1e-2 A, in cells of 40 to
900 A, where FP32 positions err by 1e-6 to 1e-4 A.  The counts are integer work: equal to
those of FP64 distances."""
import importlib
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CUTS = (5.0, 4.0, 3.5)


@pytest.mark.parametrize("side", [40.0, 250.0, 900.0])
def test_counts(cg, tmp_path, side):
    synth = importlib.import_module("chimes_lsq-myllfork_gb300.synth")
    fm = str(tmp_path / "fm_setup.in")
    synth.write_fm_setup(fm, "traj.xyzf", 1, ["O"], [16.0], 2, 2, 2, 0.8, CUTS[0], 3.0,
                         smax3=CUTS[1], smax4=CUTS[2])
    model = cg.Model(fm)
    rng = np.random.default_rng(int(side))
    cells = list(itertools.product(range(3), repeat=3))
    frames, want = [], np.zeros(3, int)
    for c in CUTS:
        for sign in (-1, 1):
            ds = sign * np.array([1e-9, 1e-8, 1e-7, 1e-6, 3e-6, 1e-5, 1e-4, 1e-3, 1e-2])
            xyz = []
            for k, d in enumerate(ds):
                o = (np.array(cells[k * 3 % 27]) + 0.2 + 0.3 * rng.random(3)) * (side / 3)
                r = c + d
                g = o + np.array([[0, 0, 0], [1.1, 0, 0], [0, 1.1, 0], [r / 3**0.5] * 3])
                dist = {p: np.linalg.norm(g[p[0]] - g[p[1]]) for p in itertools.combinations(range(4), 2)}
                for nb in (2, 3, 4):
                    want[nb - 2] += sum(all(dist[p] < CUTS[nb - 2] for p in itertools.combinations(t, 2))
                                        for t in itertools.combinations(range(4), nb))
                xyz.append(g)
            frames.append(np.concatenate(xyz))
    n = [len(x) for x in frames]
    fr = cg.Frames.from_arrays(model, n, np.zeros(sum(n), int), np.concatenate(frames),
                               np.stack([(np.eye(3) * side).reshape(9)] * len(n))).independent()
    sess = cg.Session(model, 0)
    sess.assemble(fr, cg.CG_FP64)
    got = sess.last_counts()
    assert [got["pairs"], got["triplets"], got["quads"]] == want.tolist()
