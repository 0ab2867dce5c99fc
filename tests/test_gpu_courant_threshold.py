"""The Courant scan takes every cell whose depth, 0 at least, is above the dry
threshold (main.cpp:303-320). A threshold below 0 takes a cell that its neighbours have
overdrawn too, whose discharge over a depth of 0 makes the next step 0; one of
0 and more does not. The FP32 state takes the cells that the FP64 state takes."""
import numpy as np
import pytest

from fluxos_cpp_b200 import scenarios as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tma", [1, 0])
@pytest.mark.parametrize("ks", [0.001, 0.0, -1.0])
def test_fp32_takes_the_cells_that_fp64_takes(ks, tma):
    nr, nc, at = 31, 40, (15, 20)
    sc = S.plane_scenario(nr, nc, seed=6)
    sc.horizon, sc.ade, sc.ks = 1e5, False, ks
    sc.dem = np.full((nr, nc), 100.0)
    sc.meteo = ((0.0, 0.0, 0.0), (1e5, 0.0, 0.0))
    sc.init_h, sc.init_qx = np.full((nr, nc), 0.05), np.zeros((nr, nc))
    sc.init_h[at] = 0.04
    # one neighbour draws on the shallow one with what the limit on the
    # shallow cell's own faces does not see
    sc.init_qx[at[0] - 1:at[0] + 2, at[1]] = (-0.2, -0.2, 0.4)
    dts = []
    for precision in ("fp64", "fp32"):
        d = S.make_domain(sc, precision=precision)
        d.set_option("tma", tma)
        dts.append([d.step(1)["dtfl"] for _ in range(2)])
        assert d.download("h")[1:-1, 1:-1].min() == 0.0
        d.close()
    a, b = np.array(dts)
    assert a[0] > 0.0 and (a[1] == 0.0) == (ks < 0)
    assert np.allclose(a, b, rtol=1e-4, atol=0.0)  # FP32 depths and discharges, one step of 2^-23 each
