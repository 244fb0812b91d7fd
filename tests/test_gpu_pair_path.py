"""The two-pass symmetry-function path (values, then forces with dE/dG
contracted inside the triplets) against the kernels that form dG/dr
(N2P2B_SF_VARIANT asks for those) and, where it covers the functions, against
the restated oracle.

Systems at the edges of the path's tiles: one to three atoms, neighbor counts
around the 32-bit mask words, every unit kind (powers of two, other integer
zeta, shifted Gaussians, non-integer zeta and |lambda| != 1, compact, element-
weighted), narrow and wide, several cutoff radii.  Tolerances as for the
other kernels: G 1e-12 of the array's scale, energy 1e-10 relative, forces
1e-10 max(|F|, rms F).
"""
import os

import numpy as np
import pytest

from n2p2_b200 import synth

pytestmark = pytest.mark.gpu

GOLD = os.path.join(os.path.dirname(__file__), "golden")
POTS = ["potentials/h2o_52", "potentials/h2o_92", "potentials/h2o_wtd",
        "ref_examples/H2O_RPBE-D3", "ref_examples/Cu2S_PBE",
        "ref_examples/Ethylbenzene_SCAN"]


@pytest.fixture(scope="module")
def gpu():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _prediction(d, general, monkeypatch, precision="fp64"):
    from n2p2_b200.mode import Prediction
    if general:
        monkeypatch.setenv("N2P2B_SF_VARIANT", "6")
    else:
        monkeypatch.delenv("N2P2B_SF_VARIANT", raising=False)
    p = Prediction(d)
    p.setup()
    p.setup_symmetry_function_statistics(False, False, False, False)
    if precision != "fp64":
        p.set_precision(precision)
    return p


def _cluster(n, ne, seed, spacing):
    """n atoms on a jittered lattice (no two closer than 0.7 spacing)."""
    rng = np.random.default_rng(seed)
    m = int(np.ceil(n ** (1 / 3)))
    g = np.array([[i, j, k] for i in range(m) for j in range(m)
                  for k in range(m)], dtype=float)[:n]
    pos = spacing * (g + rng.uniform(-0.15, 0.15, g.shape))
    return pos, rng.integers(0, ne, size=n).astype(np.int32)


def _compare(d, pos, elem, box, monkeypatch):
    a = _prediction(d, True, monkeypatch)
    b = _prediction(d, False, monkeypatch)
    e0, f0 = a.predict(pos, elem, box)
    e1, f1 = b.predict(pos, elem, box)
    G0, G1 = a.symmetry_functions(), b.symmetry_functions()
    assert np.abs(G0 - G1).max() <= 1e-12 * max(1.0, np.abs(G0).max())
    assert abs(e1 - e0) <= 1e-10 * abs(e0)
    scale = np.maximum(np.abs(f0), np.sqrt(np.mean(f0 ** 2)))
    assert np.all(np.abs(f1 - f0) <= 1e-10 * scale)
    return e1, f1, b


@pytest.mark.parametrize("n", [1, 2, 3, 32, 33, 34, 65, 97])
@pytest.mark.parametrize("pot", POTS)
def test_clusters(gpu, monkeypatch, pot, n):
    d = os.path.join(GOLD, pot)
    # All atoms of the smaller clusters are neighbors of each other.
    spacing = 1.8 if "Cu2S" in pot else 3.0
    pos, elem = _cluster(n, 2, n, spacing)
    _compare(d, pos, elem, None, monkeypatch)


@pytest.mark.parametrize("pot", ["potentials/h2o_52", "potentials/h2o_wtd"])
def test_water_box(gpu, monkeypatch, pot):
    """A periodic box; dG/dr on request after an evaluation without it, and
    the same energy and forces from a second evaluation, step by step and
    from a captured graph."""
    d = os.path.join(GOLD, pot)
    box, pos, elem = synth.water_box(64, 3)
    e, f, p = _compare(d, pos, elem, box, monkeypatch)
    p.evaluate_nnp(True)
    assert p.energy == e and np.array_equal(p.forces(), f)
    g = p.symmetry_functions()
    s, _ = p.dGdr()
    q = _prediction(d, True, monkeypatch)
    q.predict(pos, elem, box)
    s0, _ = q.dGdr()
    assert np.abs(s - s0).max() <= 1e-12 * np.abs(s0).max()
    assert np.array_equal(g, p.symmetry_functions())
    p.capture_graph(True)
    p.launch_graph()
    p.finish()
    assert p.energy == e and np.array_equal(p.forces(), f)
    p.calculate_neighbor_list()
    p.calculate_symmetry_function_groups(True)
    p.calculate_atomic_neural_networks(True)
    p.calculate_energy()
    p.calculate_forces()
    scale = np.maximum(np.abs(f), np.sqrt(np.mean(f ** 2)))
    assert np.all(np.abs(p.forces() - f) <= 1e-10 * scale)


def _write_general(d, out):
    """h2o_52 with functions that need the general units: shifted narrow and
    wide Gaussians, zeta 2.5 and 3, lambda 0.5, a second cutoff radius."""
    keep, nets = [], []
    with open(os.path.join(d, "input.nn")) as fh:
        for line in fh:
            w = line.split()
            if w[:1] == ["symfunction_short"]:
                continue
            keep.append(line)
    sf = []
    for c in "HO":
        for e in "HO":
            sf.append(f"{c} 2 {e} 0.02 1.5 12.0")
            sf.append(f"{c} 2 {e} 0.3 0.0 7.0")
        for a, b in (("H", "H"), ("H", "O"), ("O", "O")):
            sf += [f"{c} 3 {a} {b} 0.02 1.0 1.0 12.0 1.5",
                   f"{c} 3 {a} {b} 0.01 -1.0 2.5 12.0",
                   f"{c} 3 {a} {b} 0.01 0.5 2.0 12.0",
                   f"{c} 3 {a} {b} 0.03 1.0 3.0 8.0",
                   f"{c} 3 {a} {b} 0.03 -1.0 3.0 8.0",
                   f"{c} 3 {a} {b} 0.1 1.0 16.0 8.0",
                   f"{c} 9 {a} {b} 0.02 1.0 3.0 12.0 2.0",
                   f"{c} 9 {a} {b} 0.02 -1.0 6.0 8.0"]
    with open(os.path.join(out, "input.nn"), "w") as fh:
        fh.writelines(keep)
        fh.writelines(f"symfunction_short {s}\n" for s in sf)
    per = len(sf) // 2
    rng = np.random.default_rng(4)
    with open(os.path.join(out, "scaling.data"), "w") as fh:
        for e in (1, 2):
            for k in range(per):
                fh.write(f"{e} {k + 1} 0.0 10.0 1.0 1.0\n")
    widths = [per, 25, 25, 1]
    count = sum(i * o + o for i, o in zip(widths[:-1], widths[1:]))
    for z in (1, 8):
        with open(os.path.join(out, f"weights.{z:03d}.data"), "w") as fh:
            fh.writelines(f"{v:.16e}\n"
                          for v in rng.uniform(-0.3, 0.3, count))


@pytest.mark.parametrize("n", [3, 33, 97])
def test_general_units(gpu, monkeypatch, tmp_path, n):
    _write_general(os.path.join(GOLD, "potentials/h2o_52"), str(tmp_path))
    pos, elem = _cluster(n, 2, 7, 3.0)
    e, f, _ = _compare(str(tmp_path), pos, elem, None, monkeypatch)
    from oracle import restated
    e0, f0 = restated.predict(str(tmp_path), pos, elem, None)
    assert abs(e - e0) <= 1e-10 * abs(e0)
    scale = np.maximum(np.abs(f0), np.sqrt(np.mean(f0 ** 2)))
    assert np.all(np.abs(f - f0) <= 1e-10 * scale)


@pytest.mark.parametrize("pot", ["potentials/h2o_52", "potentials/h2o_92",
                                 "ref_examples/Ethylbenzene_SCAN"])
def test_mixed(gpu, monkeypatch, pot):
    """The mixed form keeps its accuracy targets, E/atom 1e-4 and force RMSE
    5e-3, against the FP64 form."""
    d = os.path.join(GOLD, pot)
    if "Ethyl" in pot:
        pos, elem = _cluster(97, 2, 5, 3.0)
        box = None
    else:
        box, pos, elem = synth.water_box(64, 5)
    e0, f0 = _prediction(d, True, monkeypatch).predict(pos, elem, box)
    e1, f1 = _prediction(d, False, monkeypatch, "mixed").predict(pos, elem,
                                                                 box)
    assert abs(e1 - e0) / len(elem) <= 1e-4
    assert np.sqrt(np.mean((f1 - f0) ** 2)) <= 5e-3


@pytest.mark.parametrize("mol", [394, 395, 592, 593, 769, 770])
def test_team_sizes(gpu, monkeypatch, mol):
    """Atom counts on both sides of the values pass's rules (two thirds of a
    wave, one wave, 1.3 waves of 148 x 12 warps) against one and four warps
    per atom asked for."""
    box, pos, elem = synth.water_box(mol, 4)
    out = []
    for wpa in (None, "1", "4"):
        if wpa is None:
            monkeypatch.delenv("N2P2B_PAIR_WPA", raising=False)
        else:
            monkeypatch.setenv("N2P2B_PAIR_WPA", wpa)
        p = _prediction(os.path.join(GOLD, POTS[0]), False, monkeypatch)
        p.set_structure(pos, elem, box)
        p.evaluate_nnp(True)
        out.append((p.symmetry_functions(), p.forces()))
    for G, F in out[1:]:
        assert np.abs(out[0][0] - G).max() <= 1e-12 * np.abs(G).max()
        assert np.abs(out[0][1] - F).max() <= 1e-10 * np.abs(F).max()


def test_two_threads(gpu, monkeypatch):
    """Two host threads whose launches of the same kernels take different
    amounts of shared memory: results as alone."""
    import threading
    work = []
    for mol, scale in ((64, 1.0), (64, 0.85)):
        box, pos, elem = synth.water_box(mol, 6)
        p = _prediction(os.path.join(GOLD, POTS[0]), False, monkeypatch)
        p.set_structure(pos * scale, elem, box * scale)
        p.evaluate_nnp(True)
        work.append((p, p.forces()))
    wrong = []

    def run(p, f0):
        try:
            for _ in range(50):
                p.evaluate_nnp(True)
                if not np.array_equal(p.forces(), f0):
                    wrong.append("forces")
        except Exception as e:        # noqa: BLE001
            wrong.append(repr(e))
    threads = [threading.Thread(target=run, args=w) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
