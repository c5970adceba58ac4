"""FP64 MD steps on kept lists with the tensor-core contraction of triplets and quadruplets
(3-body order 8, 4-body order 4): clusters grouped at the build, filtered each step into
partly filled tiles, lists rebuilt and built ahead as atoms move.  The same trajectory with
lists enumerated every step agrees to 1e-9 A (the force sums' order differs), and the last
step's forces are those of one force call at the last positions, to 1e-10 of the largest."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
MASSES = np.array([12.011, 1.0079, 14.007, 15.9994])


@pytest.mark.parametrize("sizes,speed", [([64, 120, 33], 0.02), ([90], 0.3), ([5, 40, 150], 0.3)])
def test_kept_lists_match_enumeration_every_step(cg, tmp_path, sizes, speed):
    torch = pytest.importorskip("torch")
    synth = importlib.import_module("chimes_lsq-myllfork_gb300.synth")
    fm = synth.make_workload("chno-4b", str(tmp_path), nframes=len(sizes), seed=sum(sizes), order=(8, 8, 4),
                             sizes=list(sizes), triclinic=False, labels=False)
    model = cg.Model(fm)
    nat, types, xyz, cell = synth.frames_arrays(str(tmp_path / "traj.xyzf"), len(sizes), ["C", "H", "N", "O"])[:4]
    rng = np.random.default_rng(8)
    x = 2e-5 * rng.standard_normal(model.ncols)
    n = int(sum(nat))
    v0 = rng.standard_normal((n, 3)) * speed
    out = []
    for skin_milli in (500, 0):
        sess = cg.Session(model, 0)
        sess.md_setup(x)
        sess.tune("md_skin_milli", skin_milli)
        dfr = sess.upload(cg.Frames.from_arrays(model, nat, types, xyz, cell).independent())
        v = torch.from_numpy(v0.reshape(-1).copy()).cuda()
        F = torch.zeros(3 * n, dtype=torch.float64, device="cuda")
        sess.md_nve(dfr, MASSES, 0.5, 40, v.data_ptr(), F.data_ptr())
        torch.cuda.synchronize()
        pos = dfr.read_positions()
        alone = cg.Frames.from_arrays(model, nat, types, np.asarray(pos).reshape(n, 3), cell).independent()
        F1, _ = sess.md_force(alone)
        counts = sess.md_last_counts()
        assert counts["triplets"] > 0 and counts["quads"] > 0
        assert np.abs(F.cpu().numpy().reshape(n, 3) - F1).max() <= 1e-10 * np.abs(F1).max()
        out.append(np.asarray(pos).reshape(n, 3))
    moved = np.abs(out[0] - xyz.reshape(n, 3)).max()
    assert moved > (0.25 if speed > 0.1 else 1e-3)
    assert np.abs(out[0] - out[1]).max() <= 1e-9
