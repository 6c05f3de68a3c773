"""Periodic meshes one cell wide, where a cell is its own neighbour across two
of its sides: the sweeps leave such a side out, as the reference's loops over
lower and higher cell numbers do, and the residual takes it as any other."""
import numpy as np
import pytest

import ccfd_b200 as cc
from ccfd_b200 import meshgen
from oracle import restated
from tests.helpers import rel_max_err

pytestmark = pytest.mark.gpu


def _case(nx, ny, precision=0, implicit=True):
    ini = meshgen.sinewave_ini(None, n=8, periodic=True, implicit=implicit, source=False, limiter=2)
    ini = ini.replace("nElemsX = 8", f"nElemsX = {nx}").replace("nElemsY = 8", f"nElemsY = {ny}")
    case = cc.CaseData.from_text(ini + f"precision = {precision}\n")
    m = case.mesh()
    assert (m["face_cells"][:, 0] == m["face_cells"][:, 1]).any()  # the mesh is one cell wide
    return case


def _state(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    return case.prim0() * (1.0 + 0.05 * rng.uniform(-1.0, 1.0, (case.n_cells, 4)))


@pytest.mark.parametrize("nx,ny", [(3, 1), (37, 1), (1, 8), (1, 1)])
def test_residual_matches_the_oracle(nx, ny):
    case = _case(nx, ny, implicit=False)
    prim = _state(case, 7)
    s = cc.Solver(case)
    s.set_state(prim)
    ut = s.fv_time_derivative(0.0)
    s.close()
    assert rel_max_err(ut, restated.residual(case, prim, 0.0)) <= 1e-12


# widths of three or more along the mesh: no pair of cells shares two faces
@pytest.mark.parametrize("nx,ny", [(3, 1), (37, 1), (400, 1), (1, 8), (1, 1)])
@pytest.mark.parametrize("precision", [0, 1])
def test_sweep_leaves_the_cell_itself_out(nx, ny, precision):
    case = _case(nx, ny, precision)
    s = cc.Solver(case)
    s.set_state(_state(case, 11))
    _, Di, O = s.build_matrix(0.0, 0.036 / max(nx, ny, 36))
    rng = np.random.Generator(np.random.PCG64(13))
    rhs = rng.standard_normal((case.n_cells, 4)).astype(np.float32).astype(np.float64)
    out = [s.lusgs(rhs) for _ in range(2)]
    s.close()
    want = restated.lusgs(case, Di, O, rhs)
    # FP64: the same operations in the same order.  FP32 sweeps round some 40
    # operations a row, and a row passes its error on to the rows after it by
    # the factor |D^-1 O| < 1/2 of these blocks: two sweeps stay below
    # 2 * 2 * 40 * 2^-24 < 1e-5
    m = case.mesh()
    own = np.repeat(np.arange(case.n_cells), np.diff(m["hs_offset"]))
    across = np.abs(O[m["hs_nb"] != own]).sum(axis=2).max(initial=0.0)
    assert across * np.abs(Di).sum(axis=2).max() < 0.5
    tol = 1e-13 if precision == 0 else 1e-5
    for x in out:
        assert np.abs(x - want).max() <= tol * np.abs(want).max()
    assert np.array_equal(*out)
