"""Periodic meshes two cells wide, where two cells face each other across two
sides: the preconditioner does not depend on what its memory held before."""
import os
import tempfile

import numpy as np
import pytest

import ccfd_b200 as cc
from ccfd_b200 import meshgen

pytestmark = pytest.mark.gpu


def _two_wide(precision):
    ini = meshgen.sinewave_ini(None, n=8, periodic=True, implicit=True, source=False, limiter=2, cfl=2.0)
    ini = ini.replace("nElemsY = 8", "nElemsY = 2").replace("epsNewton = 0.001", "epsNewton = 0.1")
    return cc.CaseData.from_text(ini + f"precision = {precision}\n")


def _run(solver):
    solver.time = 0.0
    solver.set_state(solver.case.prim0())
    rep = solver.run(2)
    return rep["newton_iterations"], rep["gmres_iterations"], solver.get_state()


@pytest.mark.parametrize("precision", [0, 1])
def test_steps_do_not_depend_on_recycled_memory(precision):
    case = _two_wide(precision)
    first = cc.Solver(case)
    want = _run(first)
    # Krylov vectors of another solver fill the memory that the next ones get
    with tempfile.TemporaryDirectory() as tmp:
        meshgen.naca_ogrid(0.0, 0.0, 0.12, 64, 32, r_far=5.0, h0=1e-2, wall_code=101).write_gmsh(
            os.path.join(tmp, "m.msh"))
        ini = meshgen.airfoil_ini("m", mach=0.4, alpha=2.0, n_kdim=60, cfl=20.0, precond=False)
        other = cc.Solver(cc.CaseData.from_text(ini, tmp))
    other.run(2)
    other.close()
    solvers = [cc.Solver(case) for _ in range(24)]
    for s in solvers:
        got = _run(s)
        assert got[:2] == want[:2]
        assert np.array_equal(got[2], want[2])
    for s in [first] + solvers:
        s.close()
