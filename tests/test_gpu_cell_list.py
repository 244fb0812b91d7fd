"""Neighbor lists of larger periodic structures (nlCellKernel: cells as runs
of sorted FP32 positions, hits ranked in shared memory) against the same
structure in a batch of one (no cells): indices, displacements and distances
bit for bit; the forces need every entry's mirror entry, hence the key order.
One and two cells along a side, skewed cells, atoms on the cell's faces, more
neighbors than the shared ranks hold, atoms outside the cell."""
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


CUBE = np.eye(3)
CASES = {
    # name: (molecules, shape in units of the cube's side, scale, remap)
    "cube": (1100, CUBE, 1.0, True),
    "one-cell-high": (600, np.diag([2.0, 2.0, 0.25]), 1.0, True),
    "one-cell-wide": (600, np.diag([0.25, 2.0, 2.0]), 1.0, True),
    "two-cells-high": (700, np.diag([1.4, 1.4, 0.5102]), 1.0, True),
    "skewed": (800, np.array([[1.0, 0.0, 0.0], [0.3, 1.0, 0.0],
                              [-0.25, 0.35, 1.0]]), 1.0, True),
    "dense": (2000, CUBE, 0.7, True),
    "outside": (600, CUBE, 1.0, False),
}


@pytest.mark.parametrize("name", list(CASES))
def test_cells(gpu, name):
    from n2p2_b200.mode import Prediction
    mol, shape, scale, remap = CASES[name]
    cube, pos, elem = synth.water_box(mol, 7)
    frac = pos @ np.linalg.inv(cube)
    frac[:40, 0] = 0.0
    frac[20:60, 2] = 0.0
    box = shape * cube[0, 0] * scale
    pos = frac @ box
    if not remap:
        pos[:9] += box[1]
    p, q = Prediction(POT), Prediction(POT)
    for o in (p, q):
        o.setup()
        o.setup_symmetry_function_statistics(False, False, False, False)
        if name == "dense":     # FP64 stages no more than 256 neighbors
            o.set_precision("mixed")
    p.set_structure(pos, elem, box, remap=remap)
    q.set_structures([(box, pos, elem)], remap=remap)
    for o in (p, q):
        o.calculate_neighbor_list()
    a, b = p.neighbor_list(), q.neighbor_list()
    assert (a[0].max() > 256) == (name == "dense")
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
