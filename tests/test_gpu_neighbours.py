"""Neighbour lists (csrc/geom.cu k_neigh) against a plain FP64 enumeration: the number of
pairs and clusters over frame sizes around the 32-atom chunks, cubic and triclinic
cells, cells shorter than the cut-off (unordered lists, several image layers), and batches
small and large enough for each split of an atom over warps.  Sets are integer work: the
counts are equal."""
import importlib
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pairs(xyz, cell, cut, smin, layers):
    """Pairs (i, image of j) with smin < r < cut; parents i <= j, or all when the cell is
    not longer than the cut-off (the small-cell convention)."""
    n = len(xyz)
    rng = range(-layers, layers + 1)
    shifts = np.array(list(itertools.product(rng, rng, rng)), dtype=float) @ cell
    frac = xyz @ np.linalg.inv(cell)
    x = (frac - np.floor(frac)) @ cell
    small = min(abs(np.diag(cell))) <= cut
    count = 0
    for s in shifts:
        d = np.linalg.norm(x[None, :, :] + s - x[:, None, :], axis=2)
        ok = (d < cut) & (d > smin)
        if not np.any(s):
            np.fill_diagonal(ok, False)
        count += int(ok.sum()) if small else int(np.triu(ok).sum())
    return count


@pytest.mark.parametrize("sizes,side,layers", [((31, 32, 33, 64, 65, 95), None, 1), ((1, 2, 5), 4.0, 2), ((7, 40), 3.2, 4),
                                               ((257, 700), None, 1), ((20,) * 300, None, 1)])
def test_pair_counts(cg, tmp_path, sizes, side, layers):
    synth = importlib.import_module("chimes_lsq-myllfork_gb300.synth")
    fm = str(tmp_path / "fm_setup.in")
    synth.write_fm_setup(fm, "traj.xyzf", len(sizes), ["O", "H"], [16.0, 1.0], 6, 0, 0, 0.8, 5.0, 1.4, nlayers=layers)
    model = cg.Model(fm)
    rng = np.random.default_rng(len(sizes))
    xyz, typ, cells, want = [], [], [], 0
    for k, n in enumerate(sizes):
        L = side or max((n / 0.1) ** (1 / 3), 5.5)
        cell = np.diag([L, L, L])
        if side is None and k % 2:
            cell = cell + np.array([[0, 0, 0], [0.3, 0, 0], [-0.2, 0.4, 0]])
        x = rng.uniform(-0.2, 1.2, (n, 3)) @ cell
        xyz.append(x); typ.append(rng.integers(0, 2, n)); cells.append(cell.reshape(9))
        want += _pairs(x, cell, 5.0, 0.8, layers)
    fr = cg.Frames.from_arrays(model, list(sizes), np.concatenate(typ), np.concatenate(xyz), np.stack(cells)).independent()
    sess = cg.Session(model, 0)
    sess.assemble(fr, cg.CG_FP64)
    assert sess.last_counts()["pairs"] == want
