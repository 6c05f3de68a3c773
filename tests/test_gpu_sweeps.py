"""LU-SGS sweeps against the oracle: by clusters on meshes where the warps'
cell ranges are empty, partly filled or ragged, and by one CTA on a numbering
that needs more mailboxes than the cluster has."""
import os
import tempfile

import numpy as np
import pytest

import ccfd_b200 as cc
from ccfd_b200 import meshgen
from oracle import restated

pytestmark = pytest.mark.gpu


def _case(kind, a, b):
    with tempfile.TemporaryDirectory() as tmp:
        path = os.path.join(tmp, "m.msh")
        if kind == "quad":
            meshgen.naca_ogrid(0.0, 0.0, 0.12, a, b, r_far=5.0, h0=1e-2, wall_code=101).write_gmsh(path)
        elif kind == "shuffled":
            mesh = meshgen.naca_ogrid(0.0, 0.0, 0.12, a, b, r_far=5.0, h0=1e-2, wall_code=101)
            mesh.quad = mesh.quad[np.random.Generator(np.random.PCG64(5)).permutation(len(mesh.quad))]
            mesh.write_gmsh(path)
        else:
            meshgen.cylinder_mesh(a, b, wall_code=101).write_gmsh(path)
        ini = meshgen.airfoil_ini("m", mach=0.4, alpha=2.0, n_kdim=10, cfl=5.0)
        return cc.CaseData.from_text(ini, tmp)


# 16 cells: most of the 32 ranges empty; rows of 31 and 33 cells: ranges that
# cut rows; 70 x 40: levels of several chunks; 12,800 cells in random order:
# about 3,000 values between the ranges of a CTA
@pytest.mark.parametrize("kind,a,b", [("quad", 8, 2), ("quad", 31, 5), ("quad", 33, 32), ("quad", 70, 40),
                                      ("tri", 12, 3), ("tri", 48, 11), ("shuffled", 128, 100)])
def test_sweep_matches_the_oracle(kind, a, b):
    case = _case(kind, a, b)
    rng = np.random.Generator(np.random.PCG64(a * 100 + b))
    s = cc.Solver(case)
    s.set_state(case.prim0() * (1.0 + 0.02 * rng.uniform(-1.0, 1.0, (case.n_cells, 4))))
    _, Di, O = s.build_matrix(0.0, s.calc_time_step())
    rhs = rng.standard_normal((case.n_cells, 4))
    x = s.lusgs(rhs)
    s.close()
    want = restated.lusgs(case, Di, O, rhs)
    # the same operations in the same order; 1e-13 allows for the oracle's compiler
    assert np.abs(x - want).max() <= 1e-13 * np.abs(want).max()
