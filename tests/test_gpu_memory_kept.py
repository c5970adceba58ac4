"""Device memory that the library keeps: large frames (lists, arenas, row blocks; more than 256
MiB, csrc/scratch.h POOL_BLOCK) go back to the driver when they are freed, and everything
unused does with cg_session_tune "release_memory".  Free memory is the driver's figure; 64 MiB
allowed for the 2 MiB granules of other allocations and the context."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SLACK = 64 << 20


def test_freed_frames_go_back(cg, tmp_path):
    torch = pytest.importorskip("torch")
    synth = importlib.import_module("chimes_lsq-myllfork_gb300.synth")
    model = cg.Model(synth.make_workload("water-2b", str(tmp_path), nframes=1, seed=3))
    sess = cg.Session(model, 0)
    n, per = 320, 8001                       # 27 images of 40 bytes per atom: 2.77 GB
    cell = np.diag([43.4] * 3).reshape(1, 9)
    xyz = np.random.default_rng(1).uniform(0.0, 43.4, (n * per, 3))
    types = np.tile(np.array([0, 1, 1], dtype=np.int32), n * per // 3)
    frames = cg.Frames.from_arrays(model, [per] * n, types, xyz, np.repeat(cell, n, axis=0))
    sess.tune("release_memory", 1)
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    up = sess.upload(frames)
    held = free0 - torch.cuda.mem_get_info()[0]
    assert held > 27 * 40 * n * per
    del up
    torch.cuda.synchronize()
    assert free0 - torch.cuda.mem_get_info()[0] <= SLACK


def test_scratch_goes_back_on_request(cg, tmp_path):
    torch = pytest.importorskip("torch")
    synth = importlib.import_module("chimes_lsq-myllfork_gb300.synth")
    sess = cg.Session(cg.Model(synth.make_workload("water-2b", str(tmp_path), nframes=1, seed=3)), 0)
    rows, n = 60000, 2000
    A = torch.randn((rows, n), dtype=torch.float32, device="cuda")
    b = torch.randn(rows, dtype=torch.float64, device="cuda")
    G = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    h = torch.zeros(n, dtype=torch.float64, device="cuda")
    sess.gram(cg.CG_FP32, A.data_ptr(), n, 64, n, b.data_ptr(), 1, G.data_ptr(), h.data_ptr())
    sess.tune("release_memory", 1)
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    sess.gram(cg.CG_FP32, A.data_ptr(), n, rows, n, b.data_ptr(), 1, G.data_ptr(), h.data_ptr())
    torch.cuda.synchronize()
    kept = free0 - torch.cuda.mem_get_info()[0]
    assert kept > 2 * SLACK                  # the BF16 planes stay for the next call
    sess.tune("release_memory", 1)
    assert free0 - torch.cuda.mem_get_info()[0] <= SLACK
