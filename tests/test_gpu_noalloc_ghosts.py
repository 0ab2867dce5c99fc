"""fx_adesolver_noalloc on a caller's arrays whose ghost cells hold any depth. It
enters the dispersion and the limit of the last row's and column's fluxes
(ADEsolver_calc.cpp:187-194), where a NaN loses every comparison. Against the
oracle on the same arrays, to the 1e-10 of the other tests of this entry
point."""
import numpy as np
import pytest

import fluxos_cpp_b200 as fx
import test_zz_no_alloc as Z

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr,nc,dxy", [(2, 2, 2), (31, 40, 3), (65, 33, 2), (90, 7, 10)])
@pytest.mark.parametrize("depth", [np.nan, np.inf, 0.0, 3.0])
def test_ghost_depths(depth, nr, nc, dxy):
    import torch
    g = Z._random_presweep(nr, nc, seed=nr)
    ghost = np.ones(g["h"].shape, dtype=bool)
    ghost[1:-1, 1:-1] = False
    g["h"][ghost] = depth
    # below 0 a concentration draws a flux from a ghost cell, which the limit is for
    g["conc"][~ghost] -= 1.0
    want = Z._oracle_sweep(g, nr, nc, dxy, 0.5, 0.3)
    got = Z._call_presweep(fx.lib(), torch, g, nr, nc, dxy, 0.3, 0.5)
    assert np.array_equal(np.isnan(want[1:-1, 1:-1]), np.isnan(got[1:-1, 1:-1]))
    assert np.isfinite(want[1:-1, 1:-1]).all()
    Z._check(want, got)
