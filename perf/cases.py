"""Timed cases of the library's public entry points.

The work a user has the library do: MD forces (one system through host arrays, larger
systems and mixed batches resident on the device, a served batch of short NVE runs),
A-matrix assembly (2-, 3- and 4-body bases, FP64 and FP32, even and uneven frames), the
normal equations in both forms, a batched fit replayed as one graph, and the Cholesky
factorisation and solve that end a fit.

`listed()` gives the cases, `draw(rng)` another of the same ranges, `prepare` the inputs
and handles a program holds before the call, `run` one pass, `work` the bytes and
operations of one pass, and `exact` the outputs in 64 bits from plain torch.
"""
import importlib
import itertools
import math
import os
import tempfile

import numpy as np
import torch

cg = importlib.import_module("chimes_lsq-myllfork_gb300")
synth = importlib.import_module("chimes_lsq-myllfork_gb300.synth")

# order and cut-offs (A) of the 2-, 3- and 4-body terms, species, rows beside the forces
BASES = {
    "water2b": dict(species=("O", "H"), order=(12, 0, 0), cut=(5.0, None, None), extra=False),
    "water3b": dict(species=("O", "H"), order=(16, 8, 0), cut=(5.0, 4.0, None), extra=True),
    "ch4b": dict(species=("C", "H"), order=(16, 8, 4), cut=(5.0, 4.0, 3.5), extra=True),
    "chno4b": dict(species=("C", "H", "N", "O"), order=(16, 8, 4), cut=(5.0, 4.0, 3.5), extra=True),
}
MASS = {"C": 12.011, "H": 1.0079, "N": 14.007, "O": 15.9994}
SMIN, LAMBDA, SMOOTH = 0.8, 1.4, 0.01   # inner cut-off, Morse length, smoothing below the inner cut-off
DENSITY = 0.1                           # atoms per A^3 of the cubic C/H/N/O cells
KB, TFS = 0.0019872067, 48.888          # kcal/mol/K; fs per internal time unit
DT = 0.2                                # MD time step, fs
RIDGE = 1e-6                            # ridge of the solve over the largest diagonal entry
MD_SCALE = 1e-4                         # size of the MD coefficients


def listed():
    return [
        # one chimes_md-like force call on a small system, host arrays in and out: the latency floor
        dict(name="md_host_64_f64", kind="md", basis="chno4b", sizes="64", prec=64, host=True),
        # the FP64 force of an ordinary system resident on the device
        dict(name="md_1000_f64", kind="md", basis="chno4b", sizes="1000", prec=64, host=False),
        # a batch of uneven systems in the FP32 contraction form
        dict(name="md_mixed_f32", kind="md", basis="chno4b", sizes="64 301 1111 2600", prec=32, host=False),
        # continuous-batching service: requests of uneven sizes, NVE steps with resident lists
        dict(name="serve_f32", kind="serve", basis="chno4b", sizes="96 250 700 1024", prec=32, nsteps=40),
        # a whole small fit's A, host frames in and host A out
        dict(name="fit_water2b_host_f64", kind="asm", basis="water2b", sizes=" ".join(["192"] * 10), prec=64, host=True,
             tri=False),
        # the 3-body water workload, FP64 rows on the device
        dict(name="fit_water3b_f64", kind="asm", basis="water3b", sizes=" ".join(["384"] * 32), prec=64, host=False,
             tri=False),
        # the 4-body triclinic workload, FP64 rows: the plain form of the headline assembly
        dict(name="fit_chno4b_f64", kind="asm", basis="chno4b", sizes=" ".join(["256"] * 16), prec=64, host=False,
             tri=True),
        # a block of the batched form's uneven frames, FP32 rows
        dict(name="fit_chno4b_uneven_f32", kind="asm", basis="chno4b", sizes="33 57 120 201 256 410 640 1001", prec=32,
             host=False, tri=False),
        # a batched fit (FP32 assembly and tensor-core Gram of uneven frames) replayed as one graph
        dict(name="batch_fit_ch4b", kind="batch", basis="ch4b", block=8,
             sizes="40 77 130 255 64 311 90 48 190 36 222 101 400 57 83 149 35 270 61 120 45 333 72 98"),
        # mixed form's Gram of an FP32 row block with an odd number of columns
        dict(name="gram_mixed_12000x6007", kind="gram", rows=12000, cols=6007, prec=32, mode=1),
        # plain form's FP64 Gram at the 3-body workload's column count
        dict(name="gram_f64_30001x820", kind="gram", rows=30001, cols=820, prec=64, mode=0),
        # factorisation and solve of the normal equations
        dict(name="cholesky_solve_5000", kind="chol", n=5000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["md", "md", "serve", "asm", "asm", "asm", "batch", "gram", "gram", "chol"])
    if kind == "md":
        prec = rng.choice([64, 32])
        sizes = [_log(rng, 64, 3000) for _ in range(rng.randint(1, 4))]
        if prec == 64:   # within the cost of the largest FP32 batches
            sizes = sizes[:1]
        return dict(kind="md", basis=rng.choice(["chno4b", "ch4b"]), sizes=" ".join(map(str, sizes)), prec=prec,
                    host=rng.random() < 0.3)
    if kind == "serve":
        sizes = [_log(rng, 64, 1100) for _ in range(rng.randint(1, 5))]
        return dict(kind="serve", basis="chno4b", sizes=" ".join(map(str, sizes)), prec=32, nsteps=rng.randint(5, 40))
    if kind == "asm":
        basis = rng.choice(["water2b", "water3b", "chno4b", "ch4b"])
        prec = rng.choice([64, 32])
        if basis.startswith("water"):
            sizes = [3 * _log(rng, 50, 128)] * _log(rng, 1, 40)
            return dict(kind="asm", basis=basis, sizes=" ".join(map(str, sizes)), prec=prec, host=basis == "water2b",
                        tri=False)
        tri = rng.random() < 0.4
        n = rng.randint(1, 10)
        sizes = [256] * n if tri else [_log(rng, 32, 700) for _ in range(min(n, 6))]
        return dict(kind="asm", basis=basis, sizes=" ".join(map(str, sizes)), prec=prec, host=False, tri=tri)
    if kind == "batch":
        return dict(kind="batch", basis="ch4b", block=rng.randint(3, 9),
                    sizes=" ".join(str(_log(rng, 32, 350)) for _ in range(rng.randint(5, 24))))
    if kind == "gram":
        if rng.random() < 0.5:
            return dict(kind="gram", rows=_log(rng, 300, 12000), cols=_log(rng, 500, 6000), prec=rng.choice([32, 64]), mode=1)
        return dict(kind="gram", rows=_log(rng, 300, 30000), cols=_log(rng, 100, 1000), prec=64, mode=0)
    return dict(kind="chol", n=_log(rng, 300, 5000))


# ------------------------------------------------------------------ inputs
DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _place(rng, n, cell, sep):
    """n points uniform in the cell, no two (over periodic images) closer than sep."""
    inv = np.linalg.inv(cell)
    pts = np.empty((0, 3))
    while len(pts) < n:
        for p in rng.uniform(0, 1, size=(2 * n, 3)) @ cell:
            f = (pts - p) @ inv
            f -= np.round(f)
            d = f @ cell
            if len(pts) and np.min(np.einsum("ij,ij->i", d, d)) < sep * sep:
                continue
            pts = np.concatenate([pts, p[None]])
            if len(pts) == n:
                break
    return pts


def _water(rng, nmol):
    """Rigid H2O at random positions and orientations (density of 128 in 15.65 A), jittered by 0.1 A."""
    side = 15.65 * (nmol / 128.0) ** (1.0 / 3.0)
    o = _place(rng, nmol, np.diag([side] * 3), 2.5)
    half = math.radians(104.5 / 2)
    q, _ = np.linalg.qr(rng.normal(size=(nmol, 3, 3)))
    body = 0.96 * np.array([[math.sin(half), 0.0, math.cos(half)], [-math.sin(half), 0.0, math.cos(half)]])
    x = np.concatenate([o[:, None], o[:, None] + np.einsum("kj,mij->mki", body, q)], axis=1).reshape(-1, 3)
    x = (x + rng.normal(scale=0.1, size=x.shape)) % side
    return x, np.tile(np.array([0, 1, 1], dtype=np.int32), nmol), np.diag([side] * 3)


def _triclinic(rng):
    a, b, c = rng.uniform(12.0, 16.0, size=3)
    al, be, ga = np.deg2rad(rng.uniform(80.0, 100.0, size=3))
    cx = c * math.cos(be)
    cy = c * (math.cos(al) - math.cos(be) * math.cos(ga)) / math.sin(ga)
    return np.array([[a, 0, 0], [b * math.cos(ga), b * math.sin(ga), 0], [cx, cy, math.sqrt(c * c - cx * cx - cy * cy)]])


def _frames(case, seed):
    """[(xyz, types, cell rows)] of a case, from the seed alone."""
    rng = np.random.default_rng([seed, 17])
    nt = len(BASES[case["basis"]]["species"])
    out = []
    for n in map(int, case["sizes"].split()):
        if case["basis"].startswith("water"):
            out.append(_water(rng, n // 3))
        else:
            side = (n / DENSITY) ** (1.0 / 3.0)
            cell = _triclinic(rng) if case.get("tri") else np.diag([side] * 3)
            out.append((_place(rng, n, cell, 0.9), rng.integers(0, nt, size=n).astype(np.int32), cell))
    return out


_models = {}


def _model(basis, nframes):
    """The parsed model of a basis (a program parses its fm_setup.in once)."""
    if (basis, nframes) not in _models:
        b = BASES[basis]
        with tempfile.TemporaryDirectory() as tmp:
            p = os.path.join(tmp, "fm_setup.in")
            synth.write_fm_setup(p, "traj.xyzf", nframes, list(b["species"]), [MASS[s] for s in b["species"]], *b["order"],
                                 SMIN, b["cut"][0], LAMBDA, smax3=b["cut"][1], smax4=b["cut"][2],
                                 fitstrs="ALL" if b["extra"] else None, fitener=b["extra"])
            _models[(basis, nframes)] = cg.Model(p)
    return _models[(basis, nframes)]


def _arrays(frames):
    return ([len(x) for x, _, _ in frames], np.concatenate([t for _, t, _ in frames]),
            np.concatenate([x for x, _, _ in frames]), np.stack([c.reshape(9) for _, _, c in frames]))


def _rows(case):
    extra = 12 if BASES[case["basis"]]["extra"] else 0
    return [3 * int(n) + extra for n in case["sizes"].split()]


def _coefs(case, seed, ncols):
    return np.random.default_rng([seed, 5]).standard_normal(ncols) * MD_SCALE


def _velocities(case, seed, frames):
    rng = np.random.default_rng([seed, 6])
    m = np.array([MASS[s] for s in BASES[case["basis"]]["species"]])
    return [rng.standard_normal(x.shape) * np.sqrt(KB * 300.0 / m[t])[:, None] for x, t, _ in frames]


def _labels(case, seed, device):
    g = torch.Generator().manual_seed(seed * 7 + 3)
    return torch.randn(sum(_rows(case)), dtype=torch.float64, generator=g).to(device) * 20.0


def _gram_inputs(case, seed, device):
    """Rows like a fit's: columns of very different size, a third of the entries zero."""
    g = torch.Generator(device=device).manual_seed(seed * 11 + 1)
    rows, cols = case["rows"], case["cols"]
    dt = torch.float64 if case["prec"] == 64 else torch.float32
    scale = torch.exp(torch.randn(cols, dtype=torch.float64, device=device, generator=g))
    a = torch.randn((rows, cols), dtype=dt, device=device, generator=g)
    a *= torch.rand((rows, cols), dtype=torch.float32, device=device, generator=g) > 1.0 / 3.0
    a *= scale.to(dt)
    return a, torch.randn(rows, dtype=torch.float64, device=device, generator=g) * 20.0


def _normal_matrix(case, seed, device):
    """A fit-like G (columns of different size, correlated) and h."""
    g = torch.Generator(device=device).manual_seed(seed * 13 + 2)
    n = case["n"]
    x = torch.randn((n + n // 2, n), dtype=torch.float32, device=device, generator=g)
    x += torch.randn((n + n // 2, 1), dtype=torch.float32, device=device, generator=g)
    x *= torch.exp(torch.randn(n, dtype=torch.float32, device=device, generator=g))
    G = (x.T @ x).double()
    G = 0.5 * (G + G.T) + 1e-4 * torch.diag(torch.diagonal(G))   # symmetric, safely definite
    return G, torch.randn(n, dtype=torch.float64, device=device, generator=g)


def _torch_prec(case):
    return (torch.float64, cg.CG_FP64) if case["prec"] == 64 else (torch.float32, cg.CG_FP32)


def prepare(case, seed):
    s = dict(case=case)
    kind = case["kind"]
    if kind == "gram":
        s["sess"] = cg.Session(_model("water2b", 1), 0)
        s["A"], s["b"] = _gram_inputs(case, seed, "cuda")
        n = case["cols"]
        s["G"] = torch.empty((n, n), dtype=torch.float64, device="cuda")
        s["h"] = torch.empty(n, dtype=torch.float64, device="cuda")
        return s
    if kind == "chol":
        s["sess"] = cg.Session(_model("water2b", 1), 0)
        s["G"], s["h"] = _normal_matrix(case, seed, "cuda")
        s["ridge"] = RIDGE * float(torch.diagonal(s["G"]).max())
        s["L"], s["x"] = torch.empty_like(s["G"]), torch.empty_like(s["h"])
        return s
    frames = _frames(case, seed)
    model = _model(case["basis"], len(frames))
    sess = s["sess"] = cg.Session(model, 0)
    host = cg.Frames.from_arrays(model, *_arrays(frames))
    if kind in ("md", "serve"):
        host.independent()
        sess.md_setup(_coefs(case, seed, model.ncols), precision=_torch_prec(case)[1])
    if kind == "serve":
        v = _velocities(case, seed, frames)
        s["requests"] = [dict(types=t, xyz=x, cell=c.reshape(9), v=w, nsteps=case["nsteps"], arrival=0.0)
                         for (x, t, c), w in zip(frames, v)]
        s["masses"] = [MASS[k] for k in BASES[case["basis"]]["species"]]
    elif kind == "md":
        if case["host"]:
            s["frames"] = host
        else:
            s["dframes"] = sess.upload(host)
            s["F"] = torch.empty((host.natoms_total, 3), dtype=torch.float64, device="cuda")
            s["S"] = torch.empty((len(frames), 11), dtype=torch.float64, device="cuda")
    elif kind == "asm":
        dt, s["prec"] = _torch_prec(case)
        s["ncols"] = model.ncols
        if case["host"]:
            s["frames"] = host
            s["A"] = np.empty((host.nrows, model.ncols), dtype=np.float64 if case["prec"] == 64 else np.float32)
        else:
            s["dframes"] = sess.upload(host)
            s["A"] = torch.empty((host.nrows, model.ncols), dtype=dt, device="cuda")
    else:   # batch: the graph is captured once and replayed
        n, bf = model.ncols, case["block"]
        blocks = [host.slice(f, min(bf, len(frames) - f)) for f in range(0, len(frames), bf)]
        b = s["b"] = _labels(case, seed, "cuda")
        s["A"] = torch.empty((max(k.nrows for k in blocks), n), dtype=torch.float32, device="cuda")
        s["G"] = torch.zeros((n, n), dtype=torch.float64, device="cuda")
        s["h"] = torch.zeros(n, dtype=torch.float64, device="cuda")
        ofs = np.concatenate([[0], np.cumsum([k.nrows for k in blocks])])
        s["blocks"] = [sess.upload(k) for k in blocks]
        s["fit"] = sess.batch_fit(s["blocks"], [b.data_ptr() + 8 * int(o) for o in ofs[:-1]], cg.CG_FP32,
                                  s["A"].data_ptr(), n, s["G"].data_ptr(), s["h"].data_ptr())
    return s


def run(s):
    case, sess = s["case"], s["sess"]
    kind = case["kind"]
    if kind == "md":
        if case["host"]:
            return sess.md_force(s["frames"])
        sess.md_force_device(s["dframes"], s["F"].data_ptr(), s["S"].data_ptr())
        return s["F"], s["S"]
    if kind == "serve":
        xyz, _, _, _ = sess.md_serve(s["requests"], s["masses"], dt_fs=DT, max_batch_atoms=4096, max_batch_frames=64)
        return xyz
    if kind == "asm":
        if case["host"]:
            return sess.assemble(s["frames"], s["prec"], out=s["A"])
        sess.assemble_device(s["dframes"], s["prec"], s["A"].data_ptr(), s["ncols"])
        return s["A"]
    if kind == "chol":
        n = case["n"]
        sess.cholesky(s["G"].data_ptr(), n, s["ridge"], s["L"].data_ptr())
        sess.cholesky_solve(s["L"].data_ptr(), n, s["h"].data_ptr(), s["x"].data_ptr())
        return torch.triu(s["L"]), s["x"]   # the factor is L^T in the upper triangle
    G, h = s["G"].zero_(), s["h"].zero_()
    if kind == "batch":
        s["fit"].launch()
    else:
        prec = _torch_prec(case)[1]
        sess.gram(prec, s["A"].data_ptr(), case["cols"], case["rows"], case["cols"], s["b"].data_ptr(), case["mode"],
                  G.data_ptr(), h.data_ptr())
    sess.gram_finish(G.data_ptr(), G.shape[0])
    return G, h


# ------------------------------------------------------------------ work
def _powers(nt, nb, order):
    """Over the cluster types: (mean allowed powers per cluster, columns)."""
    types = _types(nt, nb)
    tabs = [_columns(t, nb, order) for t in types]
    return float(np.mean([len(t[0]) for t in tabs])), sum(t[2] for t in tabs)


def _columns_total(basis):
    b = BASES[basis]
    nt = len(b["species"])
    n = nt * (nt + 1) // 2 * b["order"][0] + (nt if b["extra"] else 0)
    for nb, order in ((3, b["order"][1]), (4, b["order"][2])):
        if order:
            n += _powers(nt, nb, order)[1]
    return n


def _volume(case, n):
    if case["basis"].startswith("water"):
        return 15.65 ** 3 * n / 384.0
    return 2700.0 if case.get("tri") else n / DENSITY   # mean triclinic cell


def _clusters(case):
    """Expected (pairs, triplets, quadruplets) of uniformly placed atoms: every pair of a
    cluster within the cut-off (15/32 for a pair of neighbours, 0.1587 for three)."""
    cut = BASES[case["basis"]]["cut"]
    out = [0.0, 0.0, 0.0]
    for n in map(int, case["sizes"].split()):
        rho = n / _volume(case, n)
        for k, frac in enumerate((1.0, 15.0 / 32.0, 0.1587)):
            if cut[k]:
                m = rho * 4.0 / 3.0 * math.pi * cut[k] ** 3
                out[k] += n * m ** (k + 1) * frac / math.factorial(k + 2)
    return out


def _md_flops(case):
    o2, o3, o4 = BASES[case["basis"]]["order"]
    p, t, q = _clusters(case)
    return p * 4 * o2 + t * 4 * o3 ** 3 + q * 4 * o4 ** 6   # two multiply-adds per coefficient tensor entry


def _asm_flops(case):
    """3 multiply-adds per member and power for the forces; 13 per power for stress and energy."""
    b = BASES[case["basis"]]
    nt = len(b["species"])
    p, t, q = _clusters(case)
    fl = p * b["order"][0] * 2 * (6 + (7 if b["extra"] else 0))
    for nb, order, n in ((3, b["order"][1], t), (4, b["order"][2], q)):
        if order:
            fl += n * _powers(nt, nb, order)[0] * 2 * (3 * nb + (13 if b["extra"] else 0))
    return fl


def work(case):
    kind = case["kind"]
    if kind == "gram":
        k, n = case["rows"], case["cols"]
        return dict(bytes=k * n * case["prec"] / 8 + 8 * k + 8 * n * n + 8 * n, flops=k * n * (n + 1) + 2 * k * n)
    if kind == "chol":
        n = case["n"]
        return dict(bytes=8 * n * n + 8 * n * (n + 1) // 2 + 16 * n, flops=n ** 3 / 3 + 2 * n * n)
    atoms = sum(map(int, case["sizes"].split()))
    if kind == "md":
        return dict(bytes=atoms * (28 + 24) + 88 * len(case["sizes"].split()), flops=_md_flops(case))
    if kind == "serve":
        return dict(bytes=atoms * (52 + 24), flops=_md_flops(case) * case["nsteps"])
    rows, cols = sum(_rows(case)), _columns_total(case["basis"])
    if kind == "asm":
        return dict(bytes=rows * cols * case["prec"] / 8 + atoms * 28, flops=_asm_flops(case))
    return dict(bytes=8 * cols * cols + 8 * cols + 8 * rows + atoms * 28, flops=_asm_flops(case) + rows * cols * (cols + 1))


# ------------------------------------------------------------------ 64-bit values
EDGES = {3: ((0, 1), (0, 2), (1, 2)), 4: ((0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3))}


def _types(nt, nb):
    return list(itertools.combinations_with_replacement(range(nt), nb))


def _columns(atoms, nb, order):
    """Power tuples of a cluster type with canonical atoms `atoms` (any order with equal
    ones adjacent): (tuples [n, slots] grouped by column, column of each, columns).  Every
    atom takes part; tuples that a permutation of equal atoms turns into one another
    share a column, numbered by the first of them."""
    edges = EDGES[nb]
    slot = {e: k for k, e in enumerate(edges)}
    slot.update({(b, a): k for (a, b), k in list(slot.items())})
    p = np.array(list(itertools.product(range(order), repeat=len(edges))))
    w = order ** np.arange(len(edges))[::-1]
    used = [np.any(p[:, [k for k, e in enumerate(edges) if a in e]] > 0, axis=1) for a in range(nb)]
    p = p[np.all(used, axis=0)]
    code = p @ w
    first = code
    for perm in itertools.permutations(range(nb)):
        if all(atoms[perm[a]] == atoms[a] for a in range(nb)):
            first = np.minimum(first, p[:, [slot[(perm[a], perm[b])] for a, b in edges]] @ w)
    uniq, col = np.unique(first, return_inverse=True)
    o = np.argsort(col, kind="stable")
    return p[o], col[o], len(uniq)


def _basis(r, cut, order, first):
    """g = f T_n and h = dg/dr (n = first .. first + order - 1) of distances r, cubic cut-off."""
    lo, hi = math.exp(-cut / LAMBDA), math.exp(-SMIN / LAMBDA)
    rr = r.clamp(min=SMIN)
    ex = torch.exp(-rr / LAMBDA)
    x = (ex - 0.5 * (lo + hi)) / (0.5 * (hi - lo))
    dx = -ex / LAMBDA / (0.5 * (hi - lo))
    T, U = [torch.ones_like(x), x], [torch.ones_like(x), 2 * x]
    for _ in range(order):
        T.append(2 * x * T[-1] - T[-2])
        U.append(2 * x * U[-1] - U[-2])
    damp = torch.where(r < SMIN, torch.exp((r - SMIN) / SMOOTH), torch.ones_like(r))
    f, fd = (1 - r / cut) ** 3, -3 / cut * (1 - r / cut) ** 2
    g, h = [], []
    for n in range(first, first + order):
        t, d = T[n], (n * dx * U[n - 1] if n else torch.zeros_like(x))
        t = t + SMOOTH * (damp - 1) * d
        g.append(f * t)
        h.append(f * d * damp + fd * t)
    return torch.stack(g, -1), torch.stack(h, -1)


class _System:
    """Pairs and clusters of one frame: members by atom index and position vector."""

    def __init__(self, xyz, cell, device):
        self.x = torch.as_tensor(xyz, dtype=torch.float64, device=device)
        c = torch.as_tensor(cell, dtype=torch.float64, device=device)
        self.vol = abs(float(np.linalg.det(cell)))
        sh = torch.tensor(list(itertools.product((-1, 0, 1), repeat=3)), dtype=torch.float64, device=device) @ c
        n = len(self.x)
        self.g = (sh[:, None] + self.x[None]).reshape(-1, 3)
        self.parent = torch.arange(n, device=device).repeat(len(sh))

    def neighbours(self, cut):
        """Padded lists [n, most] of images of later atoms within cut (-1: none)."""
        ii, jj = [], []
        n = len(self.x)
        for a in range(0, n, 256):
            d = (self.x[a:a + 256, None] - self.g[None]).square().sum(-1)
            k = (d < cut * cut) & (self.parent[None] > torch.arange(a, min(n, a + 256), device=d.device)[:, None])
            i, j = torch.nonzero(k, as_tuple=True)
            ii.append(i + a)
            jj.append(j)
        return torch.cat(ii), torch.cat(jj)

    def clusters(self, nb, cut):
        """[m, nb] images (first member in the home cell), members by rising atom index."""
        n = len(self.x)
        home = 13 * n   # the unshifted images
        i, j = self.neighbours(cut)
        if nb == 2:
            return torch.stack([i + home, j], 1)
        j = j[torch.argsort(i * n + self.parent[j], stable=True)]
        deg = torch.bincount(i, minlength=n)
        start = torch.cumsum(deg, 0) - deg
        most = int(deg.max()) if len(deg) else 0
        combos = torch.combinations(torch.arange(most, device=j.device), nb - 1)
        out = []
        for a in range(0, n, 64):
            hi = deg[a:a + 64]
            ok = combos[None, :, -1] < hi[:, None]
            k, c = torch.nonzero(ok, as_tuple=True)
            m = j[start[a + k][:, None] + combos[c]]
            keep = torch.ones(len(m), dtype=torch.bool, device=m.device)
            for p, q in itertools.combinations(range(nb - 1), 2):
                keep &= (self.g[m[:, p]] - self.g[m[:, q]]).square().sum(-1) < cut * cut
                keep &= self.parent[m[:, p]] != self.parent[m[:, q]]
            out.append(torch.cat([(a + k + home)[keep][:, None], m[keep]], 1))
        return torch.cat(out) if out else torch.empty((0, nb), dtype=torch.long, device=j.device)


def _sorted_by_type(sysm, m, types, species):
    """Members reordered so that their species names ascend; the type multiset's index."""
    rank = torch.as_tensor(np.argsort(np.argsort(np.array(species))), device=m.device)
    t = types[sysm.parent[m]]
    o = torch.argsort(rank[t], dim=1, stable=True)
    m, t = torch.gather(m, 1, o), torch.gather(t, 1, o)
    nt, nb = len(species), m.shape[1]
    key = (torch.sort(t, dim=1).values * (nt ** torch.arange(nb - 1, -1, -1, device=m.device))).sum(1)
    return m, key


def _pair_type(a, b, nt):
    pairs = [(i, i) for i in range(nt)] + [(i, j) for i in range(nt) for j in range(i + 1, nt)]
    table = torch.zeros((nt, nt), dtype=torch.long)
    for k, (i, j) in enumerate(pairs):
        table[i, j] = table[j, i] = k
    return table.to(a.device)[a, b]


def _groups(sysm, types, basis, nb):
    """Per cluster type: (members, atoms in name order)."""
    b = BASES[basis]
    nt = len(b["species"])
    m, key = _sorted_by_type(sysm, sysm.clusters(nb, b["cut"][nb - 2]), types, b["species"])
    for t in _types(nt, nb):
        k = sum(v * nt ** (nb - 1 - q) for q, v in enumerate(t))
        yield sorted(t, key=lambda v: b["species"][v]), m[key == k]


def _geometry(sysm, m):
    e = EDGES[m.shape[1]]
    d = torch.stack([sysm.g[m[:, q]] - sysm.g[m[:, p]] for p, q in e], 1)
    return d, d.norm(dim=-1)


def _exact_rows(frames, basis, device):
    """The A matrix of the frames (forces, then 9 stress and 3 energy rows where fitted)."""
    b = BASES[basis]
    nt, extra = len(b["species"]), b["extra"]
    ncols = _columns_total(basis)
    A = torch.zeros((sum(3 * len(x) + (12 if extra else 0) for x, _, _ in frames), ncols), dtype=torch.float64,
                    device=device)
    tables = {nb: [_columns(t, nb, b["order"][nb - 2]) for t in
                   [sorted(t, key=lambda v: b["species"][v]) for t in _types(nt, nb)]]
              for nb in (3, 4) if b["order"][nb - 2]}
    row = 0

    def add(sysm, m, c0, D, E, d, r):
        """Rows of columns c0 ..: per cluster and slot dE/dr (D [m, slots, cols]) and E [m, cols]."""
        n = len(sysm.x)
        k = D.shape[2]
        blk = torch.zeros((n, 3, k), dtype=torch.float64, device=device)
        W = torch.zeros((3, 3, k), dtype=torch.float64, device=device)
        for s, (p, q) in enumerate(EDGES.get(m.shape[1], ((0, 1),))):
            u = d[:, s] / r[:, s, None]
            f = u[:, :, None] * D[:, s, None]
            blk.index_add_(0, sysm.parent[m[:, p]], f)
            blk.index_add_(0, sysm.parent[m[:, q]], -f)
            W -= torch.einsum("mab,mk->abk", d[:, s, :, None] * u[:, None, :], D[:, s])
        A[row:row + 3 * n, c0:c0 + k] += blk.reshape(3 * n, k)
        if extra:
            A[row + 3 * n:row + 3 * n + 9, c0:c0 + k] += W.reshape(9, k) / sysm.vol
            A[row + 3 * n + 9:row + 3 * n + 12, c0:c0 + k] += E.sum(0)

    for xyz, types, cell in frames:
        sysm = _System(xyz, cell, device)
        t = torch.as_tensor(types, dtype=torch.long, device=device)
        m = sysm.clusters(2, b["cut"][0])
        d, r = _geometry2(sysm, m)
        m, d, r = m[r > SMIN], d[r > SMIN], r[r > SMIN]
        pt = _pair_type(t[sysm.parent[m[:, 0]]], t[sysm.parent[m[:, 1]]], nt)
        for k in range(nt * (nt + 1) // 2):
            w = pt == k
            g, h = _basis(r[w], b["cut"][0], b["order"][0], 1)
            add(sysm, m[w], k * b["order"][0], h[:, None], g, d[w][:, None], r[w][:, None])
        c0 = nt * (nt + 1) // 2 * b["order"][0]
        for nb, tabs in tables.items():
            ns = len(EDGES[nb])
            for (_, mm), (pw, col, k) in zip(_groups(sysm, t, basis, nb), tabs):
                pw, col = torch.as_tensor(pw, device=device), torch.as_tensor(col, device=device)
                for a in range(0, len(mm), 1000):
                    m = mm[a:a + 1000]
                    d, r = _geometry(sysm, m)
                    g, h = _basis(r, b["cut"][nb - 2], b["order"][nb - 2], 0)
                    gp = [g[:, s][:, pw[:, s]] for s in range(ns)]
                    pre, suf = [None] * (ns + 1), [None] * (ns + 1)
                    for s in range(ns):
                        pre[s + 1] = gp[s] if s == 0 else pre[s] * gp[s]
                        suf[ns - 1 - s] = gp[ns - 1 - s] if s == 0 else suf[ns - s] * gp[ns - 1 - s]
                    red = lambda v: torch.zeros((len(m), k), dtype=torch.float64, device=device).index_add_(1, col, v)
                    D = []
                    for s in range(ns):
                        v = h[:, s][:, pw[:, s]]
                        v = v * pre[s] if s else v
                        D.append(red(v * suf[s + 1] if s < ns - 1 else v))
                    add(sysm, m, c0, torch.stack(D, 1), red(pre[ns]), d, r)
                c0 += k
        if extra:
            n = len(xyz)
            A[row + 3 * n + 9:row + 3 * n + 12, c0:c0 + nt] = torch.bincount(t, minlength=nt).double()
        row += 3 * len(xyz) + (12 if extra else 0)
    return A


def _geometry2(sysm, m):
    d = sysm.g[m[:, 1]] - sysm.g[m[:, 0]]
    return d, d.norm(dim=-1)


def _dense(x, basis, device):
    """Coefficients per cluster type as tensors over the slots' powers."""
    b = BASES[basis]
    nt = len(b["species"])
    c0, out = nt * (nt + 1) // 2 * b["order"][0], {}
    for nb in (3, 4):
        o = b["order"][nb - 2]
        out[nb] = []
        for t in _types(nt, nb):
            pw, col, k = _columns(sorted(t, key=lambda v: b["species"][v]), nb, o)
            C = np.zeros(o ** len(EDGES[nb]))
            C[pw @ (o ** np.arange(len(EDGES[nb]))[::-1])] = x[c0 + col]
            c0 += k
            out[nb].append(torch.as_tensor(C, device=device).reshape(o ** (nb - 1), -1))
    return out


def _exact_force(frame, x, dense, basis, device):
    """(forces, the 11 scalars) of one system."""
    b = BASES[basis]
    nt = len(b["species"])
    xyz, types, cell = frame
    sysm = _System(xyz, cell, device)
    t = torch.as_tensor(types, dtype=torch.long, device=device)
    n = len(xyz)
    F = torch.zeros((n, 3), dtype=torch.float64, device=device)
    W = torch.zeros((3, 3), dtype=torch.float64, device=device)
    E = torch.zeros((), dtype=torch.float64, device=device)
    P = torch.zeros((), dtype=torch.float64, device=device)

    def add(m, s, p, q, d, r, de):
        f = (de / r)[:, None] * d
        F.index_add_(0, sysm.parent[m[:, p]], f)
        F.index_add_(0, sysm.parent[m[:, q]], -f)
        return -(f[:, :, None] * d[:, None, :]).sum(0), -(de * r).sum()

    m = sysm.clusters(2, b["cut"][0])
    d, r = _geometry2(sysm, m)
    c2 = torch.as_tensor(x[:nt * (nt + 1) // 2 * b["order"][0]], device=device).reshape(-1, b["order"][0])
    c = c2[_pair_type(t[sysm.parent[m[:, 0]]], t[sysm.parent[m[:, 1]]], nt)]
    g, h = _basis(r, b["cut"][0], b["order"][0], 1)
    pen = (SMIN + 0.01 - r).clamp(min=0)   # cubic penalty just above the inner cut-off
    E = E + (c * g).sum() + 1e4 * pen.pow(3).sum()
    w, p = add(m, 0, 0, 1, d, r, (c * h).sum(1) - 3e4 * pen.square())
    W, P = W + w, P + p
    for nb in (3, 4):
        o = b["order"][nb - 2]
        for (_, m), C in zip(_groups(sysm, t, basis, nb), dense[nb]):
            if not len(m):
                continue
            d, r = _geometry(sysm, m)
            g, h = _basis(r, b["cut"][nb - 2], o, 0)
            u = [g[:, s].detach().requires_grad_(True) for s in range(len(EDGES[nb]))]
            outer = lambda v: v[0] if len(v) == 1 else (v[0][:, :, None] * outer(v[1:])[:, None, :]).reshape(len(m), -1)
            e = ((outer(u[:nb - 1]) @ C) * outer(u[nb - 1:])).sum()
            G = torch.autograd.grad(e, u)
            E = E + e.detach()
            for s, (p_, q_) in enumerate(EDGES[nb]):
                w, p = add(m, s, p_, q_, d[:, s], r[:, s], (G[s] * h[:, s]).sum(1))
                W, P = W + w, P + p
    return F, torch.cat([E.reshape(1), (P / (3.0 * sysm.vol)).reshape(1), W.reshape(9) / sysm.vol])


def exact(case, seed):
    kind = case["kind"]
    if kind == "gram":
        A, b = _gram_inputs(case, seed, DEV)
        A = A.double()
        return A.T @ A, A.T @ b
    if kind == "chol":
        G, h = _normal_matrix(case, seed, DEV)
        G.diagonal().add_(RIDGE * float(torch.diagonal(G).max()))
        L = torch.linalg.cholesky(G)
        return L.T.contiguous(), torch.cholesky_solve(h[:, None], L)[:, 0]
    frames = _frames(case, seed)
    if kind == "asm":
        return _exact_rows(frames, case["basis"], DEV)
    if kind == "batch":
        A, b = _exact_rows(frames, case["basis"], DEV), _labels(case, seed, DEV)
        return A.T @ A, A.T @ b
    x = _coefs(case, seed, _columns_total(case["basis"]))
    dense = _dense(x, case["basis"], DEV)
    if kind == "md":
        out = [_exact_force(f, x, dense, case["basis"], DEV) for f in frames]
        return torch.cat([f for f, _ in out]), torch.stack([s for _, s in out])
    mass = np.array([MASS[s] for s in BASES[case["basis"]]["species"]])
    out = []
    for (xyz, types, cell), v in zip(frames, _velocities(case, seed, frames)):
        pos, a, dt = xyz.copy(), None, DT / TFS
        for step in range(case["nsteps"]):   # the first step only evaluates forces
            if step:
                pos = pos + v * dt + 0.5 * a * dt * dt
                v = v + 0.5 * a * dt
            F, _ = _exact_force((pos, types, cell), x, dense, case["basis"], DEV)
            a = F.cpu().numpy() / mass[types][:, None]
            if step:
                v = v + 0.5 * a * dt
        out.append(pos)
    return out
