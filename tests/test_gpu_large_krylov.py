"""Dot products of the Krylov solver on both sides of the size from which a
launch of its own sums their partials (2,048 partials, 524,288 cells)."""
import os
import tempfile

import numpy as np
import pytest

import ccfd_b200 as cc
from ccfd_b200 import meshgen
from oracle import restated

pytestmark = pytest.mark.gpu


def _case(ni, nj):
    with tempfile.TemporaryDirectory() as tmp:
        meshgen.naca_ogrid(0.0, 0.0, 0.12, ni, nj, h0=2e-3, wall_code=101).write_gmsh(os.path.join(tmp, "m.msh"))
        ini = meshgen.airfoil_ini("m", mach=0.5, alpha=1.0, cfl=2.0, precond=False)
        return cc.CaseData.from_text(ini.replace("epsNewton = 0.001", "epsNewton = 0.5"), tmp)


# 2,048 and 2,052 partials; beside a small member, whose partials stay with
# the kernels that need them
@pytest.mark.parametrize("nj", [512, 513])
def test_step_matches_the_oracle(nj):
    case = _case(1024, nj)
    s, small = cc.Solver(case), cc.Solver(_case(64, 16))
    rep = s.run(1)
    state = s.get_state()
    want, info, _ = restated.run_implicit(case, 1)
    assert (rep["newton_iterations"], rep["gmres_iterations"]) == (info["newton_iterations"], info["gmres_iterations"])
    assert rep["gmres_iterations"] > 2
    assert np.abs(state - want).max() <= 1e-8 * np.abs(want).max()
    small.run(1)
    alone = small.get_state()
    b = cc.Batch(0)
    for k in (s, small):
        k.time = 0.0
        k.set_state(k.case.prim0())
        b.add(k, 1)
    b.step(1)
    b.close()
    assert np.array_equal(s.get_state(), state) and np.array_equal(small.get_state(), alone)
    s.close()
    small.close()
