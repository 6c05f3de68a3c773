"""Device-memory estimate of implicit requests (ccfd_estimate_device_bytes):
not above what admitted them while the sweeps needed no records of their own,
and never below what a context takes."""
import os
import tempfile

import numpy as np
import pytest

import ccfd_b200 as cc
from ccfd_b200 import meshgen


def _case(ni, nj, kdim=30, precision=0, ns=False, tri=False, shuffled=False, precond=True):
    with tempfile.TemporaryDirectory() as tmp:
        wall = 201 if ns else 101
        if tri:
            mesh = meshgen.cylinder_mesh(ni, nj, wall_code=wall)
        else:
            mesh = meshgen.naca_ogrid(0.0, 0.0, 0.12, ni, nj, h0=2e-3, wall_code=wall)
        if shuffled:
            mesh.quad = mesh.quad[np.random.Generator(np.random.PCG64(5)).permutation(len(mesh.quad))]
        mesh.write_gmsh(os.path.join(tmp, "m.msh"))
        ini = meshgen.airfoil_ini("m", navier_stokes=ns, n_kdim=kdim, precision=precision, precond=precond)
        return cc.CaseData.from_text(ini, tmp)


# bytes estimated for these airfoils before the cluster sweeps
@pytest.mark.parametrize("kw,before", [(dict(ni=256, nj=128), 155_340_032),
                                       (dict(ni=256, nj=128, ns=True), 155_340_032),
                                       (dict(ni=256, nj=128, precision=1), 155_340_032),
                                       (dict(ni=512, nj=256), 617_388_544)])
def test_a_budget_that_held_still_holds(kw, before):
    assert cc.estimate_device_bytes(_case(**kw)) <= before


@pytest.mark.gpu
@pytest.mark.parametrize("kw", [dict(ni=200, nj=80, kdim=1), dict(ni=200, nj=80, kdim=11), dict(ni=203, nj=81, kdim=30),
                                dict(ni=200, nj=80, kdim=7, precision=1), dict(ni=200, nj=80, kdim=5, ns=True),
                                dict(ni=201, nj=80, kdim=13, ns=True, precision=1),
                                dict(ni=120, nj=40, kdim=9, tri=True), dict(ni=160, nj=80, shuffled=True),
                                dict(ni=200, nj=80, precond=False), dict(ni=16, nj=3, kdim=3)])
def test_estimate_covers_the_context(kw):
    case = _case(**kw)
    s = cc.Solver(case)
    actual = s.device_bytes()
    s.close()
    assert actual <= cc.estimate_device_bytes(case) <= 1.25 * actual + (2 << 20)
