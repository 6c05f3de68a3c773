"""A mesh whose cells have other than three or four sides is refused before
anything is written by it: the per-cell records hold four."""
import ctypes as C

import numpy as np
import pytest

import ccfd_b200 as cc
from ccfd_b200 import _native as N
from ccfd_b200 import meshgen

pytestmark = pytest.mark.gpu

ERR_ARG = 1  # CCFD_ERR_ARG


# five sides at the first cell or at the last but one (then the last has three),
# two at the last cell
@pytest.mark.parametrize("where,by", [(1, 1), (-2, 1), (-2, 2)])
def test_other_cells_are_refused(where, by):
    case = cc.CaseData.from_text(meshgen.sod_ini(20, 2))
    c = case.c
    off = np.array(case.mesh()["hs_offset"])
    off[where] += by
    sides = np.diff(off)
    assert sides.min() < 3 or sides.max() > 4
    mesh = N.Mesh()
    C.memmove(C.byref(mesh), C.byref(c.mesh), C.sizeof(mesh))
    mesh.hs_offset = off.ctypes.data_as(C.POINTER(C.c_long))
    ctx = C.c_void_p()
    assert N.lib.ccfd_create(C.byref(c.params), C.byref(ctx)) == 0
    try:
        st = N.lib.ccfd_upload_case(ctx, C.byref(mesh), c.bc_table, c.n_bc_table, C.byref(c.exact), 1)
        assert st == ERR_ARG
        # the context stays usable
        assert N.lib.ccfd_upload_case(ctx, C.byref(c.mesh), c.bc_table, c.n_bc_table, C.byref(c.exact), 1) == 0
    finally:
        N.lib.ccfd_destroy(ctx)
