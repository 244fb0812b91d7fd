"""Neighbor lists of batches and small structures (nlbLaneKernel: only the
images in reach are walked) against a numpy enumeration of all images in the
reference's operation order: indices, displacements and distances bit for
bit, in the reference's order."""
import os

import numpy as np
import pytest

from n2p2_b200 import synth

pytestmark = pytest.mark.gpu

POT = os.path.join(os.path.dirname(__file__), "golden", "potentials",
                   "h2o_52")
RC = 12.0


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


def _expected(box, pos):
    """Counts, indices, displacements and distances, all images."""
    n = len(pos)
    shifts = [np.zeros(3)]
    if box is not None:
        vol = abs(np.linalg.det(box))
        most = []
        for k in range(3):
            c = np.cross(box[(k + 1) % 3], box[(k + 2) % 3])
            most.append(int(np.ceil(RC / (vol / np.linalg.norm(c)))))
        shifts = [(i, j, k) for i in range(-most[0], most[0] + 1)
                  for j in range(-most[1], most[1] + 1)
                  for k in range(-most[2], most[2] + 1)]
    idx, dr, d, counts = [], [], [], []
    for i in range(n):
        rows = []
        for b in shifts:
            v = pos[i] - pos
            if box is not None:
                v = v + float(b[0]) * box[0]
                v = v + float(b[1]) * box[1]
                v = v + float(b[2]) * box[2]
            rows.append(v)
        v = np.stack(rows, axis=1)                     # [j][image][3]
        n2 = v[..., 0] * v[..., 0] + v[..., 1] * v[..., 1]
        n2 = n2 + v[..., 2] * v[..., 2]
        zero = next(k for k, b in enumerate(shifts) if not np.any(b))
        hit = n2 <= RC * RC
        hit[i, zero] = False
        jj, _ = np.nonzero(hit)
        counts.append(len(jj))
        idx.append(jj)
        dr.append(v[hit])
        d.append(np.sqrt(n2[hit]))
    return (np.array(counts), np.concatenate(idx), np.concatenate(dr),
            np.concatenate(d))


CASES = {
    "cubic-11": (11, None, 0.0),
    "cubic-64": (64, None, 0.0),
    "skewed": (64, [[1.0, 0.0, 0.0], [0.45, 1.0, 0.0], [-0.4, 0.35, 1.0]],
               0.0),
    "slab": (40, [[1.6, 0.0, 0.0], [0.0, 1.6, 0.0], [0.0, 0.0, 0.390625]],
             0.0),
    "outside": (40, None, 0.7),
    "open": (30, "open", 0.0),
}


@pytest.mark.parametrize("name", list(CASES))
def test_small_structure(gpu, name):
    mol, shape, out = CASES[name]
    box, pos, elem = synth.water_box(mol, 5)
    if shape == "open":
        box = None
    elif shape is not None:
        m = np.array(shape)
        frac = pos @ np.linalg.inv(box)
        box = m * box[0, 0]
        pos = frac @ box
    if out:                 # atoms outside the cell, not remapped
        rng = np.random.default_rng(1)
        pos = pos + rng.integers(-1, 2, pos.shape) * out * box[0, 0]
    else:
        frac = None
    p = _prediction()
    p.set_structure(pos, elem, box, remap=False)
    p.calculate_neighbor_list()
    got = p.neighbor_list()
    for a, b in zip(got, _expected(box, pos)):
        assert np.array_equal(a, b)


def test_batch_equals_single(gpu):
    """A batch's list is each structure's own."""
    batch = [synth.water_box(m, m) for m in (11, 23, 64)]
    p = _prediction()
    p.set_structures(batch, remap=False)
    p.calculate_neighbor_list()
    cnt, idx, dr, d = p.neighbor_list()
    a0 = e0 = 0
    for box, pos, elem in batch:
        c, j, r, q = _expected(box, pos)
        n, m = len(pos), len(j)
        assert np.array_equal(cnt[a0:a0 + n], c)
        assert np.array_equal(idx[e0:e0 + m], j + a0)
        assert np.array_equal(dr[e0:e0 + m], r)
        assert np.array_equal(d[e0:e0 + m], q)
        a0 += n
        e0 += m


@pytest.mark.parametrize("mol", [213, 214, 512, 513])
def test_both_sides_of_the_rule(gpu, mol):
    """639 and 642 atoms: one structure on the lane path, one on the cell
    path (1,536 and 1,539 too); all as the same structure in a batch of one."""
    box, pos, elem = synth.water_box(mol, 3)
    p, q = _prediction(), _prediction()
    p.set_structure(pos, elem, box)
    p.calculate_neighbor_list()
    q.set_structures([(box, pos, elem)])
    q.calculate_neighbor_list()
    for a, b in zip(p.neighbor_list(), q.neighbor_list()):
        assert np.array_equal(a, b)
