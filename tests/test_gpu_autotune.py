"""What the autotuner times, by the kernels it launches: the neighbor list's
settings of a batch for every potential, and the variants of the kernels that
form dG/dr where the context uses them."""
import os

import numpy as np
import pytest

from n2p2_b200 import synth
from test_gpu_pair_path import GOLD, _prediction, gpu  # noqa: F401

pytestmark = pytest.mark.gpu

REPS = 2


def _launches(call):
    from n2p2_b200 import _capi
    lib = _capi.load()
    before = lib.n2p2b_kernel_launch_count()
    call()
    return lib.n2p2b_kernel_launch_count() - before


@pytest.mark.parametrize("dgdr", [False, True])
@pytest.mark.parametrize("pot", ["potentials/h2o_52", "potentials/h2o_92"])
def test_times_every_setting(gpu, monkeypatch, pot, dgdr):
    p = _prediction(os.path.join(GOLD, pot), False, monkeypatch)
    p.set_structures(synth.batch_structures(6, 13, lo=11, hi=40))
    p.evaluate_nnp(True)
    if dgdr:
        p.calculate_neighbor_list()
        p.calculate_symmetry_function_groups(True)
        p.evaluate_nnp(True)
    per = _launches(lambda: p.evaluate_nnp(True))
    f = p.forces()
    out = []
    n = _launches(lambda: out.append(p.autotune(True, REPS)))
    assert out[0].startswith("bucket ")
    # The start and three numbers of warps per block; with dG/dr also the
    # start and 6 x 4 + 2 variants and orders of one kernel.
    assert n == (1 + REPS) * (4 * per + (27 if dgdr else 0))
    p.evaluate_nnp(True)
    scale = np.maximum(np.abs(f), np.sqrt(np.mean(f ** 2)))
    assert np.all(np.abs(p.forces() - f) <= 1e-10 * scale)
