"""ccfd_errors refuses a state between whose cells the Godunov flux finds a
vacuum, as the residual of that state does."""
import numpy as np
import pytest

import ccfd_b200 as cc
from ccfd_b200 import meshgen

pytestmark = pytest.mark.gpu

VACUUM = 7  # CCFD_ERR_VACUUM


@pytest.mark.parametrize("precision", [0, 1])
def test_vacuum_between_cells_is_refused(precision):
    case = cc.CaseData.from_text(meshgen.sinewave_ini(None, n=8, periodic=True, source=False, flux=1)
                                 + f"precision = {precision}\n")
    x = case.mesh()["cell_bary"][:, 0]
    apart = np.stack([np.ones_like(x), np.where(x < 0.0, -20.0, 20.0), 0.0 * x, np.ones_like(x)], axis=1)
    s = cc.Solver(case)
    good = s.errors()
    assert np.isfinite(good["L1"]).all()
    for call in (lambda: s.fv_time_derivative(0.0), s.errors):
        s.set_state(apart)
        with pytest.raises(cc.CcfdError) as e:
            call()
        assert e.value.status == VACUUM
        s.set_state(case.prim0())
        again = s.errors()
        assert all(np.array_equal(again[k], good[k]) for k in good)
    s.close()
