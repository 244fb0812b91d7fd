"""The work that programs give this framework, as cases that can be timed.

Energies and forces of high-dimensional neural network potentials through the
public entry points: molecular dynamics on positions that live on the GPU,
one-off predictions of host structures, batches of independent structures,
the neighbor list of an MD engine, and the fitting of a student network.
The potentials are the ones under tests/golden; structures are seeded water
boxes at ambient density or the example structures, repeated and shaken by
thermal noise.

A case is a dict of plain values:
  kind       md | predict | replicas | screen | engine | train
  potential  directory under tests/golden
  precision  fp64 | mixed
  structure  water | example
  mol, a, b, c   molecules of the base water box (or the example's cell) and
             how often it is repeated along each box vector
  count      structures of a batch (replicas, screen)
"""
import ctypes
import math
import os

import numpy as np
import torch

from n2p2_b200 import _capi, synth
from n2p2_b200.mode import Mode, Prediction

GOLDEN = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                      "tests", "golden")
W52 = "potentials/h2o_52"          # 52 symmetry functions, 25-25 tanh
W92 = "potentials/h2o_92"          # 92, 64-64-64 softplus
WTD = "potentials/h2o_wtd"         # element-weighted types 12, 13, 23-25
POLY = "potentials/h2o_poly"       # compact types 20-22
RPBE = "ref_examples/H2O_RPBE-D3"  # 27 / 30, tanh^3 cutoff
CU2S = "ref_examples/Cu2S_PBE"     # narrow and wide angular functions
ANISOLE = "ref_examples/Anisole_SCAN"      # up to 354 compact functions
ETHYLBENZENE = "ref_examples/Ethylbenzene_SCAN"
DMABN = "ref_examples/DMABN_SCAN"  # one open molecule of 21 atoms
STUDENT = "potentials/h2o_92_student"
SIGMA = 0.1                        # thermal noise in bohr (Cu2S: see _noise)


def _case(name, kind, potential, precision="fp64", structure="water", mol=64,
          a=1, b=1, c=1, count=1):
    return dict(name=name, kind=kind, potential=potential,
                precision=precision, structure=structure, mol=mol, a=a, b=b,
                c=c, count=count)


def listed():
    return [
        # A step of molecular dynamics of a small box: launches and latency.
        _case("md_water_192", "md", W52),
        # The largest FP64 box of the benchmark, a step on GPU positions.
        _case("md_water_24576", "md", W52, mol=256, a=4, b=4, c=2),
        # Production size in the mixed form with the wide network.
        _case("md_water_98304_mixed", "md", W92, "mixed", mol=256, a=8, b=4,
              c=4),
        # One structure from host arrays and back: the published water
        # potential on its own example, 1,080 atoms.
        _case("predict_rpbe_1080", "predict", RPBE, structure="example"),
        # One isolated molecule, the smallest call there is.
        _case("predict_dmabn_21", "predict", DMABN, structure="example"),
        # A crystal with narrow and wide angular functions, odd supercell.
        _case("md_cu2s_1728", "md", CU2S, structure="example", a=2, b=3, c=2),
        # A molecular liquid described by compact functions only.
        _case("md_anisole_2048", "md", ANISOLE, structure="example", a=2, b=2,
              c=2),
        # Element-weighted functions, an odd box.
        _case("md_weighted_3537", "md", WTD, mol=131, a=3, b=3),
        # Replicas stepped together by a captured graph, mixed form.
        _case("replicas_384_mixed", "replicas", W52, "mixed", count=384),
        # Energies alone of new structures on every call (screening).
        _case("screen_96", "screen", W92, count=96),
        # The MD engine brings the neighbor list, ghost atoms included.
        _case("engine_10368", "engine", W52, mol=192, a=3, b=3, c=2),
        # One frame of fitting a student network.
        _case("train_6144_mixed", "train", W92, "mixed", mol=256, a=2, b=2,
              c=2),
    ]


def draw(rng):
    kind = rng.choice(["md", "md", "md", "predict", "replicas", "screen",
                       "engine", "train"])
    water = [W52, W52, W92, RPBE]
    mol = rng.randint(24, 256)
    if kind in ("replicas", "screen"):
        count = int(round(math.exp(rng.uniform(math.log(2), math.log(384)))))
        return _plain(kind, rng.choice([W52, W92]),
                      rng.choice(["fp64", "mixed"]), "water", mol, 1, 1, 1,
                      count)
    if kind == "train":
        a, b, c = _tiles(rng, 16)
        return _plain(kind, W92, "mixed", "water", max(mol, 128), a, b, c, 1)
    if kind == "engine":
        a, b, c = _tiles(rng, 32)
        return _plain(kind, rng.choice([W52, W92]),
                      rng.choice(["fp64", "mixed"]), "water", mol, a, b, c, 1)
    if rng.random() < 0.4:
        # The other families, sized so that none costs more than the largest
        # listed case.
        pot = rng.choice([CU2S, ANISOLE, ETHYLBENZENE, POLY, WTD])
        a, b, c = _tiles(rng, 8)
        if pot in (POLY, WTD):
            return _plain(kind, pot, "fp64", "water", mol, a, b, c, 1)
        return _plain(kind, pot, "fp64", "example", 0, a, b, c, 1)
    precision = rng.choice(["fp64", "mixed"])
    a, b, c = _tiles(rng, 96)
    return _plain(kind, rng.choice(water), precision, "water", mol, a, b, c, 1)


def _tiles(rng, most):
    n = int(round(math.exp(rng.uniform(0.0, math.log(most)))))
    a = max(1, int(round(n ** (1 / 3) * math.exp(rng.uniform(-0.4, 0.4)))))
    b = max(1, int(round(math.sqrt(n / a) * math.exp(rng.uniform(-0.3, 0.3)))))
    return a, b, max(1, n // (a * b))


def _plain(kind, potential, precision, structure, mol, a, b, c, count):
    d = _case("", kind, potential, precision, structure, mol, a, b, c, count)
    del d["name"]
    return d


# ---- structures ------------------------------------------------------------

def _read_example(potential):
    """Cell, positions and symbols of an example's input.data."""
    box, pos, sym = [], [], []
    with open(os.path.join(GOLDEN, potential, "input.data")) as fh:
        for line in fh:
            w = line.split()
            if w and w[0] == "lattice":
                box.append([float(x) for x in w[1:4]])
            elif w and w[0] == "atom":
                pos.append([float(x) for x in w[1:4]])
                sym.append(w[4])
            elif w and w[0] == "end":
                break
    return (np.array(box) if box else None), np.array(pos), sym


def _repeat(box, pos, elem, a, b, c):
    if box is None or a * b * c == 1:
        return box, pos, elem
    shift = np.array([[i, j, k] for i in range(a) for j in range(b)
                      for k in range(c)], dtype=np.float64) @ box
    pos = (pos[None, :, :] + shift[:, None, :]).reshape(-1, 3)
    return (box * np.array([[a], [b], [c]], dtype=np.float64), pos,
            np.tile(elem, a * b * c))


def _noise(case):
    """Displacement width: 0.1 bohr, in the units of the structure (the
    Cu2S example is in Angstrom) and half as much for the examples, which are
    thermal frames already."""
    if case["potential"] == CU2S:
        return 0.03
    return SIGMA if case["structure"] == "water" else 0.5 * SIGMA


def _structure(case, seed):
    """(box or None, positions, element indices) of one structure."""
    rng = np.random.default_rng(seed)
    if case["structure"] == "water":
        box, pos, elem = synth.water_box(case["mol"], seed)
    else:
        box, pos, sym = _read_example(case["potential"])
        order = sorted(set(_settings(case["potential"])["elements"][0]
                           .split()), key=_SYMBOLS.index)
        elem = np.array([order.index(s) for s in sym], dtype=np.int32)
    box, pos, elem = _repeat(box, pos, elem, case["a"], case["b"], case["c"])
    return box, pos + rng.normal(0.0, _noise(case), pos.shape), elem


def _batch(case, seed):
    """`count` water boxes of 11 to 171 molecules: shaken copies of up to 16
    boxes.  The sizes are those of the data set, the seed makes the atoms."""
    rng = np.random.default_rng(seed)
    kinds = min(16, case["count"])
    sizes = np.random.default_rng(case["count"]).integers(11, 172, size=kinds)
    base = [synth.water_box(int(m), seed * 16 + k)
            for k, m in enumerate(sizes)]
    out = []
    for s in range(case["count"]):
        box, pos, elem = base[s % kinds]
        out.append((box, pos + rng.normal(0.0, SIGMA, pos.shape), elem))
    return out


def _prediction(case):
    p = Prediction(os.path.join(GOLDEN, case["potential"]))
    p.setup()
    # No warning lines: noise takes single atoms out of the small training
    # sets' ranges.
    p.setup_symmetry_function_statistics(False, False, False, False)
    if case["precision"] != "fp64":
        p.set_precision(case["precision"])
    return p


# ---- prepare and run ---------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    p = _prediction(case)
    s = {"kind": kind, "mixed": case["precision"] != "fp64", "p": p}
    if kind in ("replicas", "screen"):
        batch = _batch(case, seed)
        s["batch"] = batch
        if kind == "replicas":
            p.set_structures(batch)
            p.evaluate_nnp(True)
            p.capture_graph(True)
            pos = np.concatenate([x[1] for x in batch])
            s["pos"] = torch.tensor(pos, dtype=torch.float64, device="cuda")
            s["forces"] = torch.zeros_like(s["pos"])
        return s
    box, pos, elem = _structure(case, seed)
    s.update(box=box, elem=elem)
    if kind == "predict":
        s["pos"] = pos
    elif kind == "engine":
        i, t, dr, elem_t, _ = _pair_list(box, pos, elem, _max_rc(case))
        s["counts"] = np.bincount(i, minlength=len(elem)).astype(np.int64)
        s["index"] = t.astype(np.int64)
        s["nbr_elem"] = elem_t[t].astype(np.int32)
        s["dr"] = np.ascontiguousarray(dr)
        s["targets"] = _targets(case, len(elem_t))
        s["forces"] = np.zeros((s["targets"], 3))
    else:
        p.set_structure(pos, elem, box)
        s["pos"] = torch.tensor(pos, dtype=torch.float64, device="cuda")
        s["forces"] = torch.zeros_like(s["pos"])
        if kind == "train":
            teacher = _prediction({**case, "precision": "fp64"})
            teacher.set_structure(pos, elem, box)
            teacher.evaluate_nnp(True)
            s["label_e"] = torch.tensor(teacher.atomic_energies(),
                                        device="cuda")
            s["label_f"] = torch.tensor(teacher.forces(), device="cuda")
            teacher.close()
            p.setup_student(os.path.join(GOLDEN, STUDENT))
            g = torch.Generator(device="cuda")
            g.manual_seed(int(seed))
            perm = torch.randperm(len(elem), generator=g,
                                  device="cuda").to(torch.int32)
            s["batches"] = [x.contiguous() for x in perm.split(4096)]
    return s


def _targets(case, used):
    """Length of the engine's per-atom arrays: atoms and ghosts with room to
    spare, whatever the frame."""
    n = 3 * case["mol"] * case["a"] * case["b"] * case["c"]
    side = synth.box_length(case["mol"])
    rc = _max_rc(case)
    full = n * math.prod(1.0 + 2.0 * rc / (side * case[k]) for k in "abc")
    room = int(1.1 * full) + 256
    if used > room:
        raise ValueError("more ghost atoms than room")
    return room


def run(s):
    p, kind = s["p"], s["kind"]
    if kind == "md":
        p.set_positions(s["pos"])
        p.evaluate_nnp(True)
        return _result(s, p.energy, p.forces(s["forces"]))
    if kind == "predict":
        return _result(s, *p.predict(s["pos"], s["elem"], s["box"]))
    if kind == "replicas":
        p.set_positions(s["pos"])
        p.launch_graph()
        p.finish()
        return _result(s, p.structure_energies(), p.forces(s["forces"]))
    if kind == "screen":
        p.set_structures(s["batch"])
        p.evaluate_nnp(False)
        return _result(s, p.structure_energies(), None)
    if kind == "engine":
        L, h = p._L, p._h
        ptr = lambda x, t: x.ctypes.data_as(ctypes.POINTER(t))  # noqa: E731
        p._check(L.n2p2b_set_neighbor_list(
            h, len(s["elem"]), ptr(s["elem"], ctypes.c_int32),
            ptr(s["counts"], ctypes.c_int64), ptr(s["index"], ctypes.c_int64),
            ptr(s["nbr_elem"], ctypes.c_int32), ptr(s["dr"], ctypes.c_double),
            s["targets"]))
        p.evaluate_nnp(True)
        p._check(L.n2p2b_get_target_forces(
            h, ptr(s["forces"], ctypes.c_double)))
        return _result(s, p.energy, s["forces"])
    # train: the symmetry functions of a frame, then its minibatches at the
    # rate at which a fit ends.
    p.set_positions(s["pos"])
    p.calculate_neighbor_list()
    p.calculate_symmetry_function_groups(True)
    for k, idx in enumerate(s["batches"]):
        loss = p.student_train_step(s["label_e"], s["label_f"], idx, 1.0, 1.0,
                                    1e-5, want_loss=k + 1 == len(s["batches"]))
    return {"loss": list(loss), "weights": _single(p.student_weights()),
            "gradient": _single(p.student_gradient())}


def _single(x):
    return torch.as_tensor(x).float()


def _result(s, energy, forces):
    """Energies and forces as the program keeps them: in the mixed form,
    whose symmetry functions are 32-bit, as 32-bit values."""
    if s["mixed"]:
        energy = _single(energy)
        forces = None if forces is None else _single(forces)
    return {"energy": energy} if forces is None else {"energy": energy,
                                                      "forces": forces}


# ---- what a pass cannot do without -------------------------------------------

def work(case):
    """Positions and elements in, energies and forces out; operations: per
    pair and radial function 15, per valid triplet 60 and per triplet and
    angular function 4 for the values, and with forces about three times as
    many (the derivative of a sum of products costs two more passes)."""
    sfs, rc = _functions(case["potential"])
    conv = _units(case["potential"])[2]
    if case["kind"] in ("replicas", "screen"):
        atoms, density = 3 * 91 * case["count"], 0.0148438
    elif case["structure"] == "water":
        atoms = 3 * case["mol"] * case["a"] * case["b"] * case["c"]
        density = 0.0148438
    else:
        box, pos, _ = _read_example(case["potential"])
        atoms = len(pos) * case["a"] * case["b"] * case["c"]
        density = (len(pos) / abs(np.linalg.det(box)) if box is not None
                   else None)
    if density is None:
        atoms, n = len(pos), len(pos) - 1
    else:
        n = density * 4.0 / 3.0 * math.pi * (rc / conv) ** 3
    ne = len(sfs)
    pairs = ne * (ne + 1) / 2
    flops = 0.0
    for e in range(ne):
        rad = sum(1 for s in sfs[e] if s["radial"])
        rad /= 1 if any(s["type"] in (12, 23) for s in sfs[e]) else ne
        ang = [s for s in sfs[e] if not s["radial"]]
        wide = any(s["type"] in (9, 22, 25) for s in ang)
        per = len(ang) / (1 if any(s["weighted"] for s in ang) else pairs)
        trip = 0.5 * n * n * (1.0 if wide else 15.0 / 32.0)
        flops += atoms / ne * (15.0 * n * rad + trip * (60.0 + 4.0 * per))
    if case["kind"] == "screen":
        return {"bytes": 28.0 * atoms, "flops": flops}
    byte = 52.0 * atoms
    if case["kind"] == "engine":
        byte = atoms * (28.0 + 36.0 * n)
    if case["kind"] == "train":
        byte += 32.0 * atoms
    return {"bytes": byte, "flops": 3.0 * flops}


# ---- the same values in plain 64-bit torch -------------------------------------

_SYMBOLS = (
    "H He Li Be B C N O F Ne Na Mg Al Si P S Cl Ar K Ca Sc Ti V Cr Mn Fe Co "
    "Ni Cu Zn").split()
_TYPES_RADIAL = (2, 12, 20, 23)
_parsed: dict = {}


def _settings(potential):
    if potential not in _parsed:
        out: dict = {}
        with open(os.path.join(GOLDEN, potential, "input.nn")) as fh:
            for line in fh:
                w = line.split("#")[0].split()
                if w:
                    out.setdefault(w[0], []).append(" ".join(w[1:]))
        _parsed[potential] = out
    return _parsed[potential]


def _units(potential):
    st = _settings(potential)
    if "conv_length" not in st:
        return 0.0, 1.0, 1.0
    return tuple(float(st[k][0])
                 for k in ("mean_energy", "conv_energy", "conv_length"))


def _functions(potential):
    """Per element the symmetry functions in the order of the network's
    inputs, in internal length units, and the largest cutoff radius."""
    st = _settings(potential)
    order = sorted(st["elements"][0].split(), key=_SYMBOLS.index)
    conv = _units(potential)[2]
    sfs = [[] for _ in order]
    for v in st["symfunction_short"]:
        a = v.split()
        t = int(a[1])
        s = {"type": t, "radial": t in _TYPES_RADIAL,
             "weighted": t in (12, 13, 23, 24, 25), "e1": -1, "e2": -1}
        x = a[2:]
        if not s["weighted"]:
            k = 1 if s["radial"] else 2
            e = sorted(order.index(y) for y in x[:k])
            s["e1"], s["e2"] = e[0], (e[1] if k == 2 else -1)
            x = x[k:]
        if t >= 20:
            s["rl"], s["rc"] = float(x[0]) * conv, float(x[1]) * conv
            s["left"], s["right"] = ((0.0, 0.0) if s["radial"] else
                                     (float(x[2]), float(x[3])))
            s["sub"] = x[-1]
            s["key"] = ((t, s["sub"], s["e1"], s["rc"], s["rl"])
                        if s["radial"] else
                        (t, s["sub"], s["e1"], s["e2"], s["rc"], s["rl"],
                         s["left"], s["right"]))
        else:
            s["eta"] = float(x[0]) / conv ** 2
            if s["radial"]:
                s["rs"], s["rc"] = float(x[1]) * conv, float(x[2]) * conv
                s["key"] = (t, s["rc"], s["eta"], s["rs"], s["e1"])
            else:
                if t == 13:
                    rs, lam, zeta, rc = x[1:5]
                else:
                    lam, zeta, rc = x[1:4]
                    rs = x[4] if len(x) > 4 else 0.0
                s["rs"], s["rc"] = float(rs) * conv, float(rc) * conv
                s["lam"], s["zeta"] = float(lam), float(zeta)
                s["key"] = (t, s["rc"], s["eta"], s["rs"], s["zeta"],
                            s["lam"], s["e1"], s["e2"])
        sfs[order.index(a[0])].append(s)
    for e in sfs:
        e.sort(key=lambda s: s["key"])
    return sfs, max(s["rc"] for e in sfs for s in e)


def _max_rc(case):
    return _functions(case["potential"])[1] / _units(case["potential"])[2]


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _ghosts(box, pos, elem, rc):
    """Atoms wrapped into the cell, followed by their images within rc of it:
    positions, elements and the atom that each one copies."""
    n = len(pos)
    if box is None:
        return pos, elem, np.arange(n)
    inv = np.linalg.inv(box)
    frac = pos @ inv
    frac = frac - np.floor(frac)
    # Distance between the faces of the cell, per box vector.
    margin = rc * np.linalg.norm(inv, axis=0) + 1e-9
    most = np.ceil(margin).astype(int)
    out_f, out_o = [frac], [np.arange(n)]
    for i in range(-most[0], most[0] + 1):
        for j in range(-most[1], most[1] + 1):
            for k in range(-most[2], most[2] + 1):
                if i == j == k == 0:
                    continue
                f = frac + np.array([i, j, k], dtype=np.float64)
                near = np.all((f >= -margin) & (f <= 1.0 + margin), axis=1)
                out_f.append(f[near])
                out_o.append(np.nonzero(near)[0])
    own = np.concatenate(out_o)
    return np.concatenate(out_f) @ box, elem[own], own


def _windows(box, pos, elem, rc, most):
    """For chunks of centers (sorted along x): centers, candidates, the
    vectors r_center - r_candidate and which of them are neighbors."""
    dev = _device()
    gp, ge, own = _ghosts(box, pos, elem, rc)
    n = len(pos)
    x = torch.tensor(gp, dtype=torch.float64, device=dev)
    order = torch.argsort(x[:, 0])
    xs = x[order, 0].contiguous()
    for e in sorted(set(int(v) for v in elem)):
        idx = torch.tensor(np.nonzero(elem == e)[0], device=dev)
        idx = idx[torch.argsort(x[idx, 0])]
        for at in range(0, len(idx), most):
            c = idx[at:at + most]
            lo = int(torch.searchsorted(xs, x[c[0], 0] - rc))
            hi = int(torch.searchsorted(xs, x[c[-1], 0] + rc, right=True))
            cand = order[lo:hi]
            vec = x[c][:, None, :] - x[cand][None, :, :]
            near = ((vec * vec).sum(-1) <= rc * rc) & (c[:, None] != cand)
            yield e, c, cand, vec, near
    return


def _pair_list(box, pos, elem, rc):
    """Full neighbor list on local and ghost atoms, by center."""
    gp, ge, own = _ghosts(box, pos, elem, rc)
    i, t, d = [], [], []
    for _, c, cand, vec, near in _windows(box, pos, elem, rc, 1024):
        a, b = torch.nonzero(near, as_tuple=True)
        i.append(c[a])
        t.append(cand[b])
        d.append(vec[a, b])
    i, t, d = torch.cat(i), torch.cat(t), torch.cat(d)
    order = torch.argsort(i, stable=True)
    return (i[order].cpu().numpy(), t[order].cpu().numpy(),
            d[order].cpu().numpy(), ge, own)


def _cutoff(st, r, rc):
    kind = int(st["cutoff_type"][0].split()[0])
    if kind == 1:
        return 0.5 * (torch.cos(math.pi * r / rc) + 1.0)
    if kind == 2:
        return torch.tanh(1.0 - r / rc) ** 3
    if kind == 6:
        x = r / rc
        return ((15.0 - 6.0 * x) * x - 10.0) * x ** 3 + 1.0
    raise ValueError("cutoff type %d" % kind)


def _core(sub, x):
    if sub.endswith("a"):
        x, sub = (2.0 - x) * x, sub[:-1]
    if sub == "e":
        return math.e * torch.exp(1.0 / (x * x - 1.0))
    if sub == "p1":
        return (2.0 * x - 3.0) * x ** 2 + 1.0
    if sub == "p2":
        return ((15.0 - 6.0 * x) * x - 10.0) * x ** 3 + 1.0
    if sub == "p3":
        return (x * (x * (20.0 * x - 70.0) + 84.0) - 35.0) * x ** 4 + 1.0
    return (x * (x * ((315.0 - 70.0 * x) * x - 540.0) + 420.0)
            - 126.0) * x ** 5 + 1.0


def _compact(sub, left, right, r):
    """The compact function and where it is not zero."""
    inside = (r > left) & (r < right)
    u = torch.where(inside, (r - 0.5 * (left + right))
                    * (2.0 / (right - left)), torch.full_like(r, 0.5))
    return torch.where(inside, _core(sub, u.abs()), torch.zeros_like(r))


class _Exact:
    def __init__(self, potential):
        self.st = st = _settings(potential)
        self.order = sorted(st["elements"][0].split(), key=_SYMBOLS.index)
        self.z = [_SYMBOLS.index(s) + 1 for s in self.order]
        self.sfs, self.rc = _functions(potential)
        self.mean, self.conv_e, self.conv_l = _units(potential)
        offsets = {v.split()[0]: float(v.split()[1])
                   for v in st.get("atom_energy", [])}
        self.offset = [offsets.get(s, 0.0) for s in self.order]
        dev = _device()
        rows = []
        with open(os.path.join(GOLDEN, potential, "scaling.data")) as fh:
            for line in fh:
                if not line.startswith("#") and line.split():
                    rows.append([float(v) for v in line.split()])
        center, scale = ("center_symmetry_functions" in st,
                         "scale_symmetry_functions" in st)
        sigma = "scale_symmetry_functions_sigma" in st and not scale
        smin = float(st.get("scale_min_short", ["0.0"])[0])
        smax = float(st.get("scale_max_short", ["1.0"])[0])
        self.scaling, at = [], 0
        for e in self.sfs:
            v = np.array([x[2:6] for x in rows[at:at + len(e)]])
            at += len(e)
            one = np.ones(len(e))
            if scale:
                f, m, lo = ((smax - smin) / (v[:, 1] - v[:, 0]),
                            v[:, 2] if center else v[:, 0], smin)
            elif sigma:
                f, m, lo = (smax - smin) / v[:, 3], v[:, 2], smin
            else:
                f, m, lo = one, (v[:, 2] if center else 0.0 * one), 0.0
            self.scaling.append((torch.tensor(f, device=dev),
                                 torch.tensor(m, device=dev), lo))
        nodes = [int(v) for v in st["global_nodes_short"][0].split()]
        self.act = st["global_activation_short"][0].split()
        self.net = []
        for e, z in zip(self.sfs, self.z):
            w = []
            path = os.path.join(GOLDEN, potential, "weights.%03d.data" % z)
            with open(path) as fh:
                for line in fh:
                    if line.split() and not line.startswith("#"):
                        w.append(float(line.split()[0]))
            w, at, layers = np.array(w), 0, []
            width = [len(e)] + nodes + [1]
            for i, o in zip(width[:-1], width[1:]):
                layers.append((torch.tensor(w[at:at + i * o].reshape(i, o),
                                            device=dev),
                               torch.tensor(w[at + i * o:at + i * o + o],
                                            device=dev)))
                at += i * o + o
            self.net.append(layers)

    def energies(self, e, R, M):
        """Atomic energies of centers of element e from the padded neighbor
        vectors R[f] and their masks M[f]."""
        st, ne = self.st, len(R)
        r2 = [(v * v).sum(-1) for v in R]
        r = [v.sqrt() for v in r2]
        B = R[0].shape[0]
        zero = torch.zeros(B, dtype=torch.float64, device=R[0].device)
        G = [zero] * len(self.sfs[e])
        fc = {}

        def cut(f, rc):
            if (f, rc) not in fc:
                fc[f, rc] = torch.where(M[f] & (r[f] < rc),
                                        _cutoff(st, r[f], rc),
                                        torch.zeros_like(r[f]))
            return fc[f, rc]

        for s_at, s in enumerate(self.sfs[e]):
            if not s["radial"]:
                continue
            for f in range(ne):
                if s["e1"] not in (-1, f):
                    continue
                w = float(self.z[f]) if s["weighted"] else 1.0
                if s["type"] < 20:
                    v = torch.exp(-s["eta"] * (r[f] - s["rs"]) ** 2) \
                        * cut(f, s["rc"])
                else:
                    v = torch.where(M[f], _compact(s["sub"], s["rl"], s["rc"],
                                                   r[f]), zero[:, None])
                G[s_at] = G[s_at] + w * v.sum(-1)
        for f1 in range(ne):
            for f2 in range(f1, ne):
                todo = [(k, s) for k, s in enumerate(self.sfs[e])
                        if not s["radial"] and (s["weighted"] or
                                                (s["e1"], s["e2"]) == (f1, f2))]
                if todo and R[f1].shape[1] and R[f2].shape[1]:
                    self._angular(todo, f1, f2, R, M, r, r2, cut, G)
        f, m, lo = self.scaling[e]
        x = lo + f * (torch.stack(G, -1) - m)
        for (w, b), a in zip(self.net[e], self.act):
            x = x @ w + b
            x = (torch.tanh(x) if a == "t" else
                 torch.nn.functional.softplus(x, threshold=1e9)
                 if a == "p" else x)
        return x[:, 0]

    def _angular(self, todo, f1, f2, R, M, r, r2, cut, G):
        n1, n2 = R[f1].shape[1], R[f2].shape[1]
        both = M[f1][:, :, None] & M[f2][:, None, :]
        dot = R[f1] @ R[f2].transpose(1, 2)
        s3 = r2[f1][:, :, None] + r2[f2][:, None, :] - 2.0 * dot
        if f1 == f2:
            both = both & torch.ones(n1, n2, dtype=torch.bool,
                                     device=both.device).triu(1)
        d = R[f1][:, :, None, :] - R[f2][:, None, :, :]
        s3 = torch.where(both, (d * d).sum(-1), torch.ones_like(s3))
        r3 = s3.sqrt()
        cos = torch.where(both, dot / (r[f1][:, :, None] * r[f2][:, None, :]),
                          torch.zeros_like(dot))
        nil = torch.zeros((), dtype=torch.float64, device=cos.device)
        memo: dict = {}

        def once(key, make):
            if key not in memo:
                memo[key] = make()
            return memo[key]

        zz = float(self.z[f1] * self.z[f2])
        for k, s in todo:
            rc, narrow = s["rc"], s["type"] in (3, 13, 21, 24)
            if s["type"] < 20:
                def weight():
                    w = cut(f1, rc)[:, :, None] * cut(f2, rc)[:, None, :]
                    q = ((r[f1][:, :, None] - s["rs"]) ** 2
                         + (r[f2][:, None, :] - s["rs"]) ** 2)
                    if narrow:
                        w = w * torch.where(both & (r3 < rc),
                                            _cutoff(self.st, r3, rc), nil)
                        q = q + (r3 - s["rs"]) ** 2
                    return torch.where(both, w * torch.exp(-s["eta"] * q), nil)

                v = once(("w", narrow, rc, s["eta"], s["rs"]), weight)
                c = once(("c", s["lam"], s["zeta"]),
                         lambda: (1.0 + s["lam"] * cos) ** int(s["zeta"])
                         * 2.0 ** (1.0 - s["zeta"]))
                if s["zeta"] != int(s["zeta"]):
                    raise ValueError("zeta that is no whole number")
                v = v * c
            else:
                def radial():
                    p = (s["sub"], s["rl"], rc)
                    v = (_compact(*p, r[f1])[:, :, None]
                         * _compact(*p, r[f2])[:, None, :])
                    if narrow:
                        v = v * _compact(*p, r3)
                    return torch.where(both, v, nil)

                v = once(("r", narrow, s["sub"], s["rl"], rc), radial)
                sub = s["sub"][:-1] if s["sub"].endswith("a") else s["sub"]
                theta = once("theta", lambda: torch.acos(cos.clamp(-1, 1)))
                v = v * once(("a", sub, s["left"], s["right"]),
                             lambda: _compact(sub, math.radians(s["left"]),
                                              math.radians(s["right"]),
                                              theta))
            v = v.sum((1, 2))
            G[k] = G[k] + (zz * v if s["weighted"] else v)

    def evaluate(self, box, pos, elem, forces=True):
        """(energy, forces on atoms and ghosts, the ghosts' atoms), physical
        units."""
        L = self.conv_l
        box = None if box is None else box * L
        pos = pos * L
        gp, ge, own = _ghosts(box, pos, elem, self.rc)
        dev = _device()
        ge_t = torch.tensor(ge, device=dev)
        F = torch.zeros((len(gp), 3), dtype=torch.float64, device=dev)
        ang = max(sum(1 for s in e if not s["radial"]) for e in self.sfs)
        most = self._centers(box, pos, ang)
        total = 0.0
        for e, c, cand, vec, near in _windows(box, pos, elem, self.rc, most):
            R, M, where = [], [], []
            for f in range(len(self.order)):
                nf = near & (ge_t[cand] == f)[None, :]
                n = int(nf.sum(1).max()) if nf.numel() else 0
                a, b = torch.nonzero(nf, as_tuple=True)
                col = (nf.cumsum(1) - 1)[a, b]
                # Empty places: far away, no two in the same place.
                v = torch.zeros((len(c), n, 3), dtype=torch.float64,
                                device=dev)
                v[..., 0] = (3.0 + f) * self.rc
                v[..., 1] = torch.arange(n, device=dev) * 0.37 + 0.1
                m = torch.zeros((len(c), n), dtype=torch.bool, device=dev)
                m[a, col] = True
                v[a, col] = vec[a, b]
                R.append(v.requires_grad_(forces))
                M.append(m)
                where.append((a, col, cand[b]))
            with torch.set_grad_enabled(forces):
                E = self.energies(e, R, M).sum()
            total += float(E.detach())
            if not forces:
                continue
            grads = torch.autograd.grad(E, R, allow_unused=True)
            for g, (a, col, t) in zip(grads, where):
                if g is None:
                    continue
                v = g[a, col]
                F.index_add_(0, c[a], -v)   # R = r_center - r_neighbor
                F.index_add_(0, t, v)
        n = len(elem)
        energy = (total / self.conv_e + n * self.mean
                  + sum(self.offset[int(x)] for x in elem))
        return energy, F * (L / self.conv_e), own

    def _centers(self, box, pos, ang):
        """Centers per chunk: some 20 GB of intermediates on a GPU."""
        if box is None:
            n = len(pos)
        else:
            n = (len(pos) / abs(np.linalg.det(box)) * 4.19 * self.rc ** 3)
        room = (6.0e8 if _device().type == "cuda" else 4.0e6) / (ang + 10.0)
        return max(1, min(1024, int(room / max(1.0, n * n))))


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return None  # an optimizer's state after several steps
    x = _Exact(case["potential"])
    if kind in ("replicas", "screen"):
        E, F = [], []
        for box, pos, elem in _batch(case, seed):
            e, f, own = x.evaluate(box, pos, elem, kind == "replicas")
            E.append(e)
            F.append(_onto_atoms(f, own, len(elem)))
        E = torch.tensor(E, dtype=torch.float64)
        return {"energy": E} if kind == "screen" else {"energy": E,
                                                       "forces": torch.cat(F)}
    box, pos, elem = _structure(case, seed)
    e, f, own = x.evaluate(box, pos, elem)
    if kind == "engine":
        f = torch.nn.functional.pad(f, (0, 0, 0,
                                        _targets(case, len(f)) - len(f)))
    else:
        f = _onto_atoms(f, own, len(elem))
    return {"energy": e, "forces": f}


def _onto_atoms(f, own, n):
    return torch.zeros((n, 3), dtype=f.dtype, device=f.device).index_add_(
        0, torch.tensor(own, device=f.device), f)
