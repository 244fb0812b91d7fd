"""A neighbor list that is refused (n2p2b_set_neighbor_list, entries out of
range) leaves what was there before: nothing, a structure or another list."""
import numpy as np
import pytest

from n2p2_b200 import synth
from test_gpu_engine_list import (_prediction, _set, _shuffled,
                                  _target_forces, gpu)  # noqa: F401

pytestmark = pytest.mark.gpu


def _lists(mol):
    box, pos, elem = synth.water_box(mol, 2)
    p = _prediction()
    p.predict(pos, elem, box)
    counts, index, dr = _shuffled(p, np.random.default_rng(1))
    nelem = elem[index].astype(np.int32)
    good = (elem, counts, index, nelem, dr, len(elem))
    bad = []
    for k, (i, e) in enumerate(((len(elem), None), (-1, None), (None, 2),
                                (None, -1))):
        x, y = index.copy(), nelem.copy()
        at = (3, len(x) - 1, len(x) // 2, 0)[k]
        if i is not None:
            x[at] = i
        if e is not None:
            y[at] = e
        bad.append((elem, counts, x, y, dr, len(elem)))
    return (box, pos, elem), good, bad


# 64 molecules: below the staged upload's size, 300: above it.
@pytest.mark.parametrize("mol", [64, 300])
@pytest.mark.parametrize("before", ["nothing", "structure", "list"])
def test_refused_list(gpu, mol, before):
    from n2p2_b200.mode import StateError
    (box, pos, elem), good, bad = _lists(mol)
    _, other, _ = _lists(33)
    q = _prediction()
    if before == "structure":
        q.set_structure(pos, elem, box)
    elif before == "list":
        _set(q, *other)
    if before != "nothing":
        q.evaluate_nnp(True)
        e0 = q.energy
        f0 = q.forces() if before == "structure" else _target_forces(q, 99)
    for b in bad:
        with pytest.raises(ValueError):
            _set(q, *b)
        if before == "nothing":
            with pytest.raises(StateError):
                q.evaluate_nnp(True)
            continue
        q.evaluate_nnp(True)
        assert q.energy == e0
        f = q.forces() if before == "structure" else _target_forces(q, 99)
        assert np.array_equal(f, f0)
    _set(q, *good)
    q.evaluate_nnp(True)
    p = _prediction()
    _set(p, *good)
    p.evaluate_nnp(True)
    assert q.energy == p.energy
    assert np.array_equal(_target_forces(q, len(elem)),
                          _target_forces(p, len(elem)))
