"""fe_2, fe_3, fn_2 and fn_3 are stored for every cell that does not end a step
above the dry threshold, whether or not "store_all_fluxes" asks for the
others: dry cells, and cells whose depth is no number."""
import numpy as np
import pytest

from fluxos_cpp_b200 import scenarios as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("tma", [1, 0])
def test_fluxes_of_cells_that_are_not_wet(tma, precision):
    nr, nc = 62, 75
    rng = np.random.default_rng(4)
    sc = S.plane_scenario(nr, nc, seed=4)
    sc.horizon = 1e5
    sc.init_h = np.where(rng.random((nr, nc)) < 0.7, rng.uniform(0, 0.05, (nr, nc)), 0.0)
    sc.init_h[rng.random((nr, nc)) < 0.01] = np.nan
    out = []
    for store_all in (1, 0):
        d = S.make_domain(sc, precision=precision)
        d.set_option("tma", tma)
        d.set_option("store_all_fluxes", store_all)
        d.step(1)
        out.append({k: d.download(k)[1:-1, 1:-1] for k in ("h", "fe_2", "fe_3", "fn_2", "fn_3")})
        d.close()
    a, b = out
    rest = ~(a["h"] > 0.5 * sc.ks)  # a depth that is no number reads as 0
    # in FP64 a cell whose level is no number is dry from the first step on
    assert np.isnan(a["fe_2"][rest]).any() == (precision == "fp32")
    for k in a:
        assert np.array_equal(a[k][rest], b[k][rest], equal_nan=True), k
