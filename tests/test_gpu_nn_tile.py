"""Networks of many atoms (nnTileKernel: several atoms of one element per
warp) on both sides of the rule that takes it, atoms of an element no
multiple of the tile, against a float64 evaluation from the weight files.

Tolerance: a running error bound of the same sweeps.  A sum of m products
has an error of (m + 4) u sum |w x| (accumulation, bias, rounded weights and
inputs), an activation function one of 16 u, all slopes are at most 1 and
their own slopes too."""
import os
import shutil

import numpy as np
import pytest

from n2p2_b200 import synth

pytestmark = pytest.mark.gpu

POTS = os.path.join(os.path.dirname(__file__), "golden", "potentials")


@pytest.fixture(scope="module")
def gpu():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _layers(d, z, nin):
    """[(W, b, activation)] of n2p2's weights.*.data."""
    with open(os.path.join(d, "input.nn")) as f:
        words = [w for w in (line.split("#")[0].split() for line in f) if w]
    key = {w[0]: w[1:] for w in words}
    width = [nin] + [int(v) for v in key["global_nodes_short"]] + [1]
    act = key["global_activation_short"]
    v = np.loadtxt(os.path.join(d, f"weights.{z:03d}.data"), usecols=0)
    out, o = [], 0
    for k, (a, b) in enumerate(zip(width[:-1], width[1:])):
        w = v[o:o + a * b].reshape(a, b).T
        o += a * b
        out.append((w, v[o:o + b], act[k]))
        o += b
    assert o == len(v)
    return out


def _activate(a, z):
    if a == "t":
        t = np.tanh(z)
        return t, 1.0 - t * t
    if a == "p":
        s = 1.0 / (1.0 + np.exp(-z))
        return np.logaddexp(0.0, z), s
    return z, np.ones_like(z)


def _network(layers, g, norm, u):
    """Energies, dE/dG and the error bounds of both."""
    x, ex, kept = g, u * np.abs(g), []
    for w, b, a in layers:
        m = w.shape[1]
        s = 1.0 / m if norm else 1.0
        ez = s * (ex @ np.abs(w).T
                  + (m + 4) * u * (np.abs(x) @ np.abs(w).T + np.abs(b)))
        z = s * (x @ w.T + b)
        x, f = _activate(a, z)
        ex = ez + 16 * u * np.maximum(1.0, np.abs(x))
        ef = (0.0 if a == "l" else 1.0) * ez + (a != "l") * 16 * u
        kept.append((w, f, ef, s))
    e, ee = x[:, 0], ex[:, 0]
    d, ed = np.ones_like(x), np.zeros_like(x)
    for w, f, ef, s in reversed(kept):
        ed = s * (ed * np.abs(f) + (np.abs(d) + ed) * ef
                  + 4 * u * np.abs(d * f))
        d = s * d * f
        m = w.shape[0]
        ed = ed @ np.abs(w) + (m + 4) * u * (np.abs(d) @ np.abs(w))
        d = d @ w
    return e, d, ee, ed


@pytest.mark.parametrize("mol", [3157, 3158, 3161])
@pytest.mark.parametrize("name,precision,norm",
                         [("h2o_52", "fp64", False), ("h2o_92", "fp64", False),
                          ("h2o_92", "fp64", True),
                          ("h2o_92_student", "fp32", False)])
def test_networks(gpu, tmp_path, name, precision, norm, mol):
    from n2p2_b200.mode import Prediction
    d = str(tmp_path / "pot")
    shutil.copytree(os.path.join(POTS, name), d)
    if norm:
        with open(os.path.join(d, "input.nn"), "a") as f:
            f.write("\nnormalize_nodes\n")
    fp64 = precision == "fp64"
    p = Prediction(d if fp64 else os.path.join(POTS, "h2o_92"))
    p.setup()
    p.setup_symmetry_function_statistics(False, False, False, False)
    if not fp64:
        p.set_precision("mixed")
        p.setup_student(d)
        p.set_student_mode("only")
    box, pos, elem = synth.water_box(mol, 3)
    p.set_structure(pos, elem, box)
    p.evaluate_nnp(True)
    G, E, D = p.symmetry_functions(), p.atomic_energies(), p.dEdG()
    u = 2.0 ** -53 if fp64 else 2.0 ** -24
    for e, z in enumerate((1, 8)):
        nsf = p.num_symmetry_functions(e)
        a = np.flatnonzero(np.asarray(elem) == e)
        en, de, ee, ed = _network(_layers(d, z, nsf), G[a, :nsf], norm, u)
        assert np.all(np.abs(E[a] - en) <= ee)
        assert np.all(np.abs(D[a, :nsf] - de) <= ed)


@pytest.mark.parametrize("mol", [11, 43, 1500])
@pytest.mark.parametrize("name", ["h2o_52", "h2o_92", "h2o_wtd"])
def test_tensor_core_networks(gpu, name, mol):
    """Rows shared by four warps (tensor cores): less than a tile, a tile
    and one atom, many; 16-byte and single stores of dE/dG.  Operands are
    pairs of BF16: a product errs by less than 2^-16 of itself."""
    from n2p2_b200.mode import Prediction
    d = os.path.join(POTS, name)
    p = Prediction(d)
    p.setup()
    p.setup_symmetry_function_statistics(False, False, False, False)
    p.set_precision("mixed")
    box, pos, elem = synth.water_box(mol, 3)
    p.set_structure(pos, elem, box)
    p.evaluate_nnp(True)
    G, E, D = p.symmetry_functions(), p.atomic_energies(), p.dEdG()
    for e, z in enumerate((1, 8)):
        nsf = p.num_symmetry_functions(e)
        a = np.flatnonzero(np.asarray(elem) == e)
        en, de, ee, ed = _network(_layers(d, z, nsf), G[a, :nsf], False,
                                  2.0 ** -16)
        assert np.all(np.abs(E[a] - en) <= ee)
        assert np.all(np.abs(D[a, :nsf] - de) <= ed)
