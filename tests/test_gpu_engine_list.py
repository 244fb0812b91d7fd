"""Neighbor lists supplied by an MD engine (n2p2b_set_neighbor_list): entries
regrouped and reverse-indexed on the device.  The list of a regular
evaluation, its entries shuffled inside each atom, must give that
evaluation's energy and forces (sums in another order: 1e-10), at sizes below
and above the staged upload's chunk, with atoms without neighbors and targets
that nothing points at; entries out of range are refused."""
import ctypes as C
import os

import numpy as np
import pytest

from n2p2_b200 import synth

pytestmark = pytest.mark.gpu

POT = os.path.join(os.path.dirname(__file__), "golden", "potentials",
                   "h2o_52")


@pytest.fixture(scope="module")
def gpu():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _prediction():
    from n2p2_b200.mode import Prediction
    p = Prediction(POT)
    p.setup()
    p.setup_symmetry_function_statistics(False, False, False, False)
    return p


def _set(p, elem, counts, index, nelem, dr, targets):
    ptr = lambda x, t: x.ctypes.data_as(C.POINTER(t))  # noqa: E731
    p._check(p._L.n2p2b_set_neighbor_list(
        p._h, len(elem), ptr(elem, C.c_int32), ptr(counts, C.c_int64),
        ptr(index, C.c_int64), ptr(nelem, C.c_int32), ptr(dr, C.c_double),
        targets))


def _target_forces(p, targets):
    f = np.zeros((targets, 3))
    p._check(p._L.n2p2b_get_target_forces(
        p._h, f.ctypes.data_as(C.POINTER(C.c_double))))
    return f


def _shuffled(p, rng):
    counts, index, dr, _ = p.neighbor_list()
    start = np.concatenate([[0], np.cumsum(counts)])
    order = np.concatenate([start[i] + rng.permutation(int(c))
                            for i, c in enumerate(counts)]).astype(np.int64)
    return counts, index[order].copy(), np.ascontiguousarray(dr[order])


@pytest.mark.parametrize("mol", [11, 64, 300])
def test_same_as_regular_list(gpu, mol):
    box, pos, elem = synth.water_box(mol, mol)
    # One atom far from all others has no neighbors.
    if mol == 11:
        box = None
        pos = np.concatenate([pos, [[500.0, 0.0, 0.0]]])
        elem = np.concatenate([elem, [1]]).astype(np.int32)
    p = _prediction()
    e0, f0 = p.predict(pos, elem, box)
    counts, index, dr = _shuffled(p, np.random.default_rng(1))
    q = _prediction()
    targets = len(elem) + 7
    for _ in range(2):
        _set(q, elem, counts, index, elem[index].astype(np.int32), dr,
             targets)
        q.evaluate_nnp(True)
        f = _target_forces(q, targets)
        assert abs(q.energy - e0) <= 1e-10 * abs(e0)
        scale = np.maximum(np.abs(f0), np.sqrt(np.mean(f0 ** 2)))
        assert np.all(np.abs(f[:len(elem)] - f0) <= 1e-10 * scale)
        assert np.all(f[len(elem):] == 0.0)
    again = _target_forces(q, targets)
    _set(q, elem, counts, index, elem[index].astype(np.int32), dr, targets)
    q.evaluate_nnp(True)
    assert np.array_equal(again, _target_forces(q, targets))


@pytest.mark.parametrize("what", ["index", "negative", "element"])
def test_bad_entry(gpu, what):
    box, pos, elem = synth.water_box(64, 2)
    p = _prediction()
    p.predict(pos, elem, box)
    counts, index, dr = _shuffled(p, np.random.default_rng(1))
    nelem = elem[index].astype(np.int32)
    if what == "index":
        index[5] = len(elem)
    elif what == "negative":
        index[-1] = -1
    else:
        nelem[77] = 2
    with pytest.raises(ValueError):
        _set(p, elem, counts, index, nelem, dr, len(elem))
