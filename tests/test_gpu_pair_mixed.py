"""FP32 two-pass kernels against FP64, no less accurate than the storing ones.

The networks are linear with weights that BF16 holds exactly, so that dE/dG
is exact and the forces' error is that of the symmetry-function stages alone:
the evaluation (two passes) and the separate steps (dG/dr in FP32, contracted
in FP64) are compared with the same FP64 evaluation.  Forces must not be
further off than the steps', with 2 % for the scatter of an rms over the
water structures' 15,000 components and 25 % where single FP32 roundings of
the same inputs make up the error (other potentials: one structure); the
symmetry functions, whose sums are FP32 in both, within 25 %."""
import os

import numpy as np
import pytest

from conftest import ref_example
from n2p2_b200 import synth
from test_gpu_pair_path import GOLD, gpu  # noqa: F401

pytestmark = pytest.mark.gpu

Z = {"H": 1, "C": 6, "N": 7, "O": 8, "S": 16, "Cu": 29}


def _linear(src, out):
    """The potential in `src` with one hidden layer and linear activations;
    dE/dG are multiples of 1/256 between 1/2 and 1 in size."""
    count = {}
    with open(os.path.join(src, "input.nn")) as fh, \
            open(os.path.join(out, "input.nn"), "w") as to:
        for line in fh:
            w = line.split()
            if w[:1] == ["symfunction_short"]:
                count[w[1]] = count.get(w[1], 0) + 1
            new = {"global_hidden_layers_short": "1",
                   "global_nodes_short": "16",
                   "global_activation_short": "l l"}.get(w[0] if w else "")
            to.write(line if new is None else f"{w[0]} {new}\n")
    with open(os.path.join(src, "scaling.data")) as fh, \
            open(os.path.join(out, "scaling.data"), "w") as to:
        to.write(fh.read())
    rng = np.random.default_rng(11)
    for s in sorted(count, key=Z.get):
        n = count[s]
        w = np.zeros((n, 16))
        w[:, 0] = rng.choice([-1, 1], n) * rng.integers(128, 256, n) / 256.0
        one = np.zeros(16)
        one[0] = 1.0
        np.savetxt(os.path.join(out, f"weights.{Z[s]:03d}.data"),
                   np.concatenate([w.ravel(), np.zeros(16), one, [0.0]]),
                   fmt="%.16e")
    return str(out)


def _water():
    for k in range(12):
        box, pos, elem = synth.water_box(64 + 16 * k, k + 20)
        pos = pos + np.random.default_rng(k).normal(0.0, 0.1, pos.shape)
        scale = 1.0 + 0.01 * (k - 6)
        yield pos * scale, elem, box * scale


def _example(name):
    d, box, pos, sym, _, _ = ref_example(name)
    order = sorted(set(sym), key=Z.get)
    elem = np.array([order.index(s) for s in sym], dtype=np.int32)
    pos = np.asarray(pos) + np.random.default_rng(7).normal(0.0, 0.05,
                                                            np.shape(pos))
    yield pos, elem, box


def _prediction(d, precision):
    from n2p2_b200.mode import Prediction
    p = Prediction(d)
    p.setup()
    p.setup_symmetry_function_statistics(False, False, False, False)
    p.set_precision(precision)
    return p


def _steps(p):
    p.calculate_neighbor_list()
    p.calculate_symmetry_function_groups(True)
    p.calculate_atomic_neural_networks(True)
    p.calculate_energy()
    p.calculate_forces()
    return p.symmetry_functions(), p.forces()


def _rms(parts):
    return np.sqrt(np.mean([np.mean(p ** 2) for p in parts]))


@pytest.mark.parametrize("pot,most", [
    ("potentials/h2o_52", 1.02), ("potentials/h2o_92", 1.02),
    ("ref_examples/H2O_RPBE-D3", 1.02), ("potentials/h2o_wtd", 1.25),
    ("ref_examples/Cu2S_PBE", 1.25),
    ("ref_examples/Ethylbenzene_SCAN", 1.25)])
def test_error_of_two_passes(gpu, monkeypatch, tmp_path, pot, most):
    monkeypatch.delenv("N2P2B_SF_VARIANT", raising=False)
    d = _linear(os.path.join(GOLD, pot), str(tmp_path))
    exact, mixed = _prediction(d, "fp64"), _prediction(d, "mixed")
    err = {"two": ([], []), "steps": ([], [])}
    water = "Cu2S" not in pot and "Ethyl" not in pot
    for pos, elem, box in (_water() if water
                           else _example(os.path.basename(pot))):
        exact.predict(pos, elem, box)
        G, F = exact.symmetry_functions(), exact.forces()
        mixed.predict(pos, elem, box)
        assert np.array_equal(mixed.dEdG(), exact.dEdG())
        two = (mixed.symmetry_functions(), mixed.forces())
        for name, got in (("two", two), ("steps", _steps(mixed))):
            for k, (x, x0) in enumerate(zip(got, (G, F))):
                err[name][k].append((x - x0) / np.sqrt(np.mean(x0 ** 2)))
    g2, f2 = (_rms(v) for v in err["two"])
    gs, fs = (_rms(v) for v in err["steps"])
    print(f"{pot}: G {g2:.3e} / {gs:.3e}, F {f2:.3e} / {fs:.3e}")
    assert 0.0 < g2 <= 1.25 * gs
    assert 0.0 < f2 <= most * fs
