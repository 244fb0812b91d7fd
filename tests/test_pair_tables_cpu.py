"""Host tables of the two-pass symmetry-function path (CPU).

tests/pair_tables/main.cpp, linked with the table builder alone, prints the
tables of a list of symmetry-function groups.
"""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "n2p2_b200", "csrc")
POW2, LADDER, GENERAL = 0, 1, 2


@pytest.fixture(scope="module")
def tables(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(nvcc)))
    exe = str(tmp_path_factory.mktemp("tables") / "main")
    r = subprocess.run(
        ["g++", "-std=c++17", "-O1", "-Wall", "-I" + CSRC,
         "-I" + os.path.join(cuda, "include"),
         os.path.join(ROOT, "tests", "pair_tables", "main.cpp"),
         os.path.join(CSRC, "sf_pair_tables.cpp"), "-o", exe],
        capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def run(elements, groups):
        text = [str(elements)]
        for g in groups:
            text.append(" ".join(str(v) for v in g[:-1])
                        + f" {len(g[-1])}")
            text += [" ".join(repr(float(v)) for v in m) for m in g[-1]]
        out = subprocess.run([exe], input="\n".join(text) + "\n",
                             capture_output=True, text=True, check=True)
        return [line.split() for line in out.stdout.splitlines()]
    return run


def _angular(zetas, runs, rc, shift=0.0):
    return [(0.01 * (a + 1), shift, lam, z) for a in range(runs)
            for z in zetas for lam in (-1.0, 1.0)]


@pytest.mark.parametrize("other", [(3, 0.0), (2.5, 0.0), (3, 1.5)])
@pytest.mark.parametrize("zetas", [(1,), (1, 4), (1, 2, 4), (1, 16)])
@pytest.mark.parametrize("runs", [1, 4, 5])
@pytest.mark.parametrize("radials", [1, 8])
def test_cells_of_units(tables, zetas, runs, radials, other):
    """Every unit adds its sums to its own cells: those lie one after another,
    the radial members' behind them, none beyond the element's.  Units of
    powers of two beside another kind are the case in which a kernel has more
    slots than the unit."""
    zeta, shift = other
    groups = []
    for e in (0, 1):
        groups += [(e, 3, 0, 0, 12.0, _angular(zetas, runs, 12.0)),
                   (e, 3, 0, 1, 12.0, _angular((zeta,), 1, 12.0, shift)),
                   (e, 3, 1, 1, 12.0, _angular(zetas, runs, 12.0)),
                   (e, 2, 0, -1, 12.0,
                    [(0.01 * k, 0.0, 0.0, 0.0) for k in range(radials)])]
    out = tables(2, groups)
    assert out[0][0] == "ok"
    slots, kinds = int(out[0][1]), int(out[0][2])
    assert slots == (5 if 16 in zetas else 3)
    assert kinds & (1 << POW2) and kinds & ~(1 << POW2)
    for e in "01":
        at = 0
        for line in out[1:]:
            if line[1] != e:
                continue
            if line[0] == "unit":
                assert int(line[3]) == at
                at += int(line[4])
            elif line[0] == "radial":
                assert int(line[2]) == at
                at += 1
            else:
                assert int(line[2]) == at


@pytest.mark.parametrize("zeta", [1.0, 3.0, 2.5])
@pytest.mark.parametrize("radial,eta,rs,served", [
    (r, eta, rs, ok) for r in (True, False) for eta, rs, ok in (
        (0.0, 0.0, True), (4.0, 0.0, True), (4.0, 1.5, True),
        (100.0, 8.0, True), (-1e-4, 0.0, False), (-0.6, 0.0, False),
        (-0.6, 2.0, False), (5.0, 1100.0, False), (50000.0, 0.0, False))
] + [(False, 2870.0, 0.0, True), (False, 2885.0, 0.0, False),
     (True, 40200.0, 0.0, True), (True, 40400.0, 0.0, False)])
def test_exponents(tables, zeta, radial, eta, rs, served):
    """-eta (sum of squares) has to stay between 0 and -5.8e6 (2^31 ln 2 /
    256) for every partner that the kernels form it for, the far one of idle
    lanes included (14 rc^2; radial: rc^2); other potentials are left to the
    storing kernels.  The function's own cutoff (6) is not the largest (12)."""
    member, plain = (eta, rs, 1.0, zeta), (0.01, 0.0, 1.0, zeta)
    groups = [(0, 3, 0, 0, 6.0, [plain if radial else member]),
              (0, 2, 0, -1, 6.0, [member if radial else plain]),
              (0, 2, 0, -1, 12.0, [(0.01, 0.0, 0.0, 0.0)])]
    out = tables(1, groups)
    assert (out[0][0] == "ok") == served
