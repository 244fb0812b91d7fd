"""Two-pass symmetry-function kernels on potentials that no committed one
stands for, against the kernels that form dG/dr: symmetry functions of h2o_52
replaced, random networks.  Tolerances as in test_gpu_pair_path.py."""
import os

import numpy as np
import pytest

from n2p2_b200 import synth
from test_gpu_pair_path import (GOLD, _cluster, _compare,  # noqa: F401
                                _prediction, gpu)

pytestmark = pytest.mark.gpu

BASE = os.path.join(GOLD, "potentials/h2o_52")
PAIRS = (("H", "H"), ("H", "O"), ("O", "O"))


def _write(out, functions, cutoff="1 0.0"):
    """A potential directory: `functions` ("type neighbors parameters") for
    both elements, networks with weights of a fixed seed."""
    with open(os.path.join(BASE, "input.nn")) as fh:
        keep = [x for x in fh if x.split()[:1] not in (["symfunction_short"],
                                                       ["cutoff_type"])]
    with open(os.path.join(out, "input.nn"), "w") as fh:
        fh.writelines(keep)
        fh.write(f"cutoff_type {cutoff}\n")
        fh.writelines(f"symfunction_short {c} {s}\n" for c in "HO"
                      for s in functions)
    per = len(functions)
    with open(os.path.join(out, "scaling.data"), "w") as fh:
        for e in (1, 2):
            for k in range(per):
                fh.write(f"{e} {k + 1} 0.0 10.0 1.0 1.0\n")
    widths = [per, 25, 25, 1]
    count = sum(i * o + o for i, o in zip(widths[:-1], widths[1:]))
    rng = np.random.default_rng(4)
    for z in (1, 8):
        with open(os.path.join(out, f"weights.{z:03d}.data"), "w") as fh:
            fh.writelines(f"{v:.16e}\n"
                          for v in rng.uniform(-0.3, 0.3, count))
    return str(out)


def _pow2(pairs, zetas, runs, rc=12.0):
    return [f"3 {a} {b} {0.01 * (r + 1)} {lam} {z} {rc}" for a, b in pairs
            for r in range(runs) for z in zetas for lam in ("-1", "1")]


@pytest.mark.parametrize("n", [3, 33, 97])
@pytest.mark.parametrize("other", ["3 H H 0.02 1.0 3.0 12.0",
                                   "3 H H 0.02 1.0 2.5 12.0",
                                   "3 H H 0.02 1.0 1.0 12.0 1.5"])
def test_few_cells_behind_powers_of_two(gpu, monkeypatch, tmp_path, other, n):
    """Powers of two up to 4 in a kernel with slots up to 16, one radial
    function per neighbor element behind the last unit."""
    sf = ["2 H 0.02 0.0 12.0", "2 O 0.05 0.0 12.0", other]
    d = _write(tmp_path, sf + _pow2(PAIRS[1:], (1, 4), 4))
    pos, elem = _cluster(n, 2, n, 3.0)
    _compare(d, pos, elem, None, monkeypatch)


def test_one_warp_per_atom_asked_for(gpu, monkeypatch):
    """327 neighbors and weighted functions: in the forces pass four atoms do
    not fit a block, so asking for one warp per atom is not followed there
    (the values pass follows: sums in another order)."""
    box, pos, elem = synth.water_box(64, 9)
    out = []
    for wpa in (None, "1"):
        if wpa:
            monkeypatch.setenv("N2P2B_PAIR_WPA", wpa)
        else:
            monkeypatch.delenv("N2P2B_PAIR_WPA", raising=False)
        p = _prediction(os.path.join(GOLD, "potentials/h2o_wtd"), False,
                        monkeypatch)
        e, f = p.predict(0.7 * pos, elem, 0.7 * box)
        assert p.neighbor_counts().max() > 300
        out.append((e, f))
    (e0, f0), (e1, f1) = out
    assert abs(e1 - e0) <= 1e-10 * abs(e0)
    assert np.abs(f1 - f0).max() <= 1e-10 * np.abs(f0).max()


# Hard, exponential, polynomial and tanh cutoffs, the cosine with an inner
# radius: the kernels of powers of two compiled for tanh^3 and polynomial 2
# and for any cutoff, with slots up to 4 and up to 16.
CUTOFFS = ["0", "2", "3", "4", "5", "6", "7", "8", "1 0.2", "6 0.3"]


def _pow2_potential(out, cutoff, zetas):
    sf = [f"2 {e} {eta} 0.0 12.0" for e in "HO" for eta in (0.01, 0.2, 1.0)]
    out.mkdir()
    return _write(out, sf + _pow2(PAIRS, zetas, 3), cutoff)


@pytest.mark.parametrize("n", [3, 33, 97])
@pytest.mark.parametrize("zetas", [(1, 2, 4), (1, 4), (1, 16), (2, 8)])
@pytest.mark.parametrize("cutoff", CUTOFFS)
def test_powers_of_two_by_cutoff(gpu, monkeypatch, tmp_path, cutoff, zetas, n):
    d = _pow2_potential(tmp_path / "p", cutoff, zetas)
    pos, elem = _cluster(n, 2, n, 3.0)
    _compare(d, pos, elem, None, monkeypatch)


@pytest.mark.parametrize("zetas", [(1, 2, 4), (1, 2, 4, 16)])
@pytest.mark.parametrize("cutoff", CUTOFFS + ["1 0.0"])
def test_powers_of_two_by_cutoff_mixed(gpu, monkeypatch, tmp_path, cutoff,
                                       zetas):
    """Errors against FP64 no larger than the storing kernels' by more than a
    quarter (one box of 64 molecules; exact dE/dG)."""
    from test_gpu_pair_mixed import _linear, _rms, _steps
    monkeypatch.delenv("N2P2B_SF_VARIANT", raising=False)
    src = _pow2_potential(tmp_path / "p", cutoff, zetas)
    (tmp_path / "q").mkdir()
    d = _linear(src, str(tmp_path / "q"))
    exact = _prediction(d, False, monkeypatch)
    mixed = _prediction(d, False, monkeypatch, "mixed")
    box, pos, elem = synth.water_box(64, 8)
    pos = pos + np.random.default_rng(1).normal(0.0, 0.1, pos.shape)
    exact.predict(pos, elem, box)
    want = exact.symmetry_functions(), exact.forces()
    mixed.predict(pos, elem, box)
    two = mixed.symmetry_functions(), mixed.forces()
    for name, x, y, x0 in zip("GF", two, _steps(mixed), want):
        e, s = _rms([x - x0]), _rms([y - x0])
        print(f"{cutoff} {zetas}: {name} {e:.3e} / {s:.3e}")
        assert 0.0 < e <= 1.25 * s


@pytest.mark.parametrize("pot", ["potentials/h2o_wtd", "potentials/h2o_52"])
def test_storing_kernels_with_global_tables(gpu, monkeypatch, pot):
    """Group tables in global memory are read by the kernels that form dG/dr,
    which an evaluation on the two-pass path does not launch."""
    d = os.path.join(GOLD, pot)
    box, pos, elem = synth.water_box(64, 17)
    out = []
    for tables in (False, True):
        if tables:
            monkeypatch.setenv("N2P2B_SF_GLOBAL_TABLES", "1")
        p = _prediction(d, True, monkeypatch)
        e, f = p.predict(pos, elem, box)
        out.append((np.array([e]), f, p.symmetry_functions(), p.dGdr()[0]))
    for a, b in zip(*out):
        assert np.abs(a - b).max() <= 1e-12 * np.abs(a).max()
