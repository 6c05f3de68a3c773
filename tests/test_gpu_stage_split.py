"""Edges of the gradient / flux kernel pair and of the batched Jacobian columns:
tile and CTA sizes that leave remainders, wing sums longer than one pass, and
column scratch that does not fit the idle Krylov vectors."""
import os
import tempfile

import numpy as np
import pytest

import ccfd_b200 as cc
from ccfd_b200 import meshgen
from tests.golden import cases as CASES

pytestmark = pytest.mark.gpu


# 32: the smallest tile; 40: threads beyond the tile's cells; 2048: one tile
# with several passes per thread; 384: the largest CTA
@pytest.mark.parametrize("tile,threads", [(32, 32), (40, 96), (128, 384), (2048, 128)])
@pytest.mark.parametrize("key", ["dmr_f05_vk", "dmr_f02_bj", "dmr_f03_o1", "zoo_ns_vk", "sine_periodic_vk"])
def test_tile_and_cta_sizes_give_identical_results(ref_small, key, tile, threads, monkeypatch):
    spec = CASES.residual_cases()[key]
    with tempfile.TemporaryDirectory() as tmp:
        case, _, _ = CASES.load_case(spec, tmp)
    prim = ref_small[f"{key}/prim"].reshape(-1, 4)
    base = cc.Solver(case)
    monkeypatch.setenv("CCFD_TILE_CELLS", str(tile))
    monkeypatch.setenv("CCFD_STAGE_THREADS", str(threads))
    other = cc.Solver(case)
    for s in (base, other):
        s.set_state(prim)
    (ua, ga), (ub, gb) = (s.fv_time_derivative(spec["time"], with_grad=True) for s in (base, other))
    assert np.array_equal(ua, ub) and np.array_equal(ga, gb)
    for s in (base, other):
        s.set_state(case.prim0())
        s.run(3)
    assert np.array_equal(base.get_state(), other.get_state())
    base.close()
    other.close()


# around one and two passes of 256 wall faces
@pytest.mark.parametrize("ni", [255, 256, 257, 513])
def test_wing_sums_of_a_step_equal_the_sequential_sum(ni):
    with tempfile.TemporaryDirectory() as tmp:
        meshgen.naca_ogrid(0.0, 0.0, 0.12, ni, 4, r_far=5.0, h0=5e-2, wall_code=101).write_gmsh(
            os.path.join(tmp, "m.msh"))
        case = cc.CaseData.from_text(meshgen.airfoil_ini("m", mach=0.4, alpha=2.0, implicit=False, precond=False,
                                                         cfl=0.5), tmp)
    s = cc.Solver(case)
    rep = s.run(2)
    # the host sums the same wall pressures one after the other
    assert (rep["cl"], rep["cd"]) == s.clcd()
    s.close()


# two Krylov vectors hold none of the columns' scratch, thirty hold all of it
@pytest.mark.parametrize("ns", [False, True])
@pytest.mark.parametrize("precision", [0, 1])
def test_jacobian_blocks_do_not_depend_on_the_krylov_dimension(ns, precision):
    out = []
    for kdim in (2, 30):
        with tempfile.TemporaryDirectory() as tmp:
            meshgen.naca_ogrid(0.0, 0.0, 0.12, 37, 9, r_far=5.0, h0=1e-2, wall_code=201 if ns else 101).write_gmsh(
                os.path.join(tmp, "m.msh"))
            case = cc.CaseData.from_text(meshgen.airfoil_ini("m", mach=0.4, alpha=2.0, navier_stokes=ns,
                                                             reynolds=500.0, n_kdim=kdim, cfl=5.0,
                                                             precision=precision), tmp)
        s = cc.Solver(case)
        out.append(s.build_matrix(0.0, 1e-3))
        s.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
