"""LU-SGS in lockstep sets whose members differ: a member without
preconditioner or with a numbering that the cluster kernel does not take leaves
the others their route and their results, and both sweep kernels give the same
results in both precisions."""
import os
import tempfile

import numpy as np
import pytest

import ccfd_b200 as cc
from ccfd_b200 import meshgen

pytestmark = pytest.mark.gpu


def _airfoil(ni, nj, kind="fits", precision=0):
    with tempfile.TemporaryDirectory() as tmp:
        mesh = meshgen.naca_ogrid(0.0, 0.0, 0.12, ni, nj, h0=2e-3, wall_code=101)
        if kind == "shuffled":  # needs more mailboxes than a cluster has
            mesh.quad = mesh.quad[np.random.Generator(np.random.PCG64(5)).permutation(len(mesh.quad))]
        mesh.write_gmsh(os.path.join(tmp, "m.msh"))
        ini = meshgen.airfoil_ini("m", mach=0.5, alpha=1.0, cfl=1.0, precond=kind != "plain", precision=precision)
        return cc.CaseData.from_text(ini.replace("epsNewton = 0.001", "epsNewton = 0.1"), tmp)


def _alone(case, steps):
    s = cc.Solver(case)
    s.run(steps)
    out = s.get_state()
    s.close()
    return out


def _batch(solvers, steps):
    """states and device milliseconds of a batch of fresh states"""
    b = cc.Batch(0)
    for s in solvers:
        s.time = 0.0
        s.set_state(s.case.prim0())
        b.add(s, steps)
    b.step(steps)
    ms = b.report(solvers[0])["device_ms"]
    b.close()
    return [s.get_state() for s in solvers], ms


# one set: every member sweeps by single CTAs; several sets: each by its route
@pytest.mark.parametrize("sets", [1, 2, 8])
@pytest.mark.parametrize("precision", [0, 1])
def test_members_equal_alone_whatever_the_route(sets, precision, monkeypatch):
    monkeypatch.setenv("CCFD_IMPLICIT_SETS", str(sets))
    kinds = ["fits", "plain", "shuffled", "fits", "fits", "shuffled"]
    cases = [_airfoil(128 + 9 * k, 96, kind, precision) for k, kind in enumerate(kinds)]
    want = [_alone(c, 2) for c in cases]
    solvers = [cc.Solver(c) for c in cases]
    got, _ = _batch(solvers, 2)
    for s in solvers:
        s.close()
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


# by clusters a step of these airfoils takes half the time of single CTAs; one
# other member costs a few percent
@pytest.mark.parametrize("kind", ["plain", "shuffled"])
def test_one_other_member_leaves_the_clusters_to_the_rest(kind):
    def best(first):
        solvers = [cc.Solver(_airfoil(128, 64, first))] + [cc.Solver(_airfoil(128 + 17 * k, 64)) for k in range(1, 8)]
        ms = min(_batch(solvers, 3)[1] for _ in range(4))
        for s in solvers:
            s.close()
        return ms

    assert best(kind) <= 1.4 * best("fits")


# NaN and infinity travel through the sweeps as through the reference's loops;
# a NaN of all ones is the pattern that marks a value as not arrived
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("bits", [0xFFFFFFFFFFFFFFFF, 0x7FF8000000000000, 0x7FF0000000000000])
def test_not_finite_values_arrive(precision, bits):
    case = _airfoil(64, 24, precision=precision)
    s = cc.Solver(case)
    _, Di, O = s.build_matrix(0.0, s.calc_time_step())
    rhs = np.random.Generator(np.random.PCG64(3)).standard_normal((case.n_cells, 4))
    rhs[700, 2] = np.array([bits], dtype=np.uint64).view(np.float64)[0]
    x = s.lusgs(rhs)
    s.close()
    from oracle import restated
    want = restated.lusgs(case, Di, O, rhs)
    assert np.array_equal(np.isnan(x), np.isnan(want))
    assert np.isnan(x).any()


# levels of several chunks and ranges that cut rows, in FP32 by clusters, and by
# one CTA on the shuffled numbering
@pytest.mark.parametrize("ni,nj,kind", [(70, 40, "fits"), (33, 32, "fits"), (128, 100, "shuffled")])
def test_fp32_sweep_matches_the_oracle(ni, nj, kind):
    from oracle import restated
    case = _airfoil(ni, nj, kind, precision=1)
    s = cc.Solver(case)
    _, Di, O = s.build_matrix(0.0, 0.05 * s.calc_time_step())
    rhs = np.random.Generator(np.random.PCG64(17)).standard_normal((case.n_cells, 4))
    rhs = rhs.astype(np.float32).astype(np.float64)
    x = s.lusgs(rhs)
    s.close()
    # some 60 rounded operations a row; a row passes its error on by the factor
    # |D^-1 O| summed over its sides, below 1/2 at this time step: two sweeps
    # stay below 2 * 2 * 60 * 2^-24 < 1.5e-5
    off = case.mesh()["hs_offset"][:-1]
    across = np.add.reduceat(np.abs(O).sum(axis=2).max(axis=1), off)
    assert (across * np.abs(Di).sum(axis=2).max(axis=1)).max() < 0.5
    want = restated.lusgs(case, Di, O, rhs)
    assert np.abs(x - want).max() <= 1.5e-5 * np.abs(want).max()
