"""Concentrations that are no numbers, infinite, or so large that their masses
overflow: the two kernels of the solute sweep give the same bits (NaN in the
same cells), in both precisions, as they evaluate the same expressions.
Evaporation that dries cells brings such values about by itself
(common.cpp:226-234 divides by the depth that is left)."""
import numpy as np
import pytest

from fluxos_cpp_b200 import scenarios as S

pytestmark = pytest.mark.gpu
VALUES = {"nan": (np.nan,), "inf": (np.inf,), "mixed": (np.nan, np.inf, -np.inf, -0.0, -1.0), "overflow": (3e37, -3e37)}


def _run(sc, precision, kernel, in_flight):
    d = S.make_domain(sc, precision=precision, steps_in_flight=in_flight)
    d.set_option("ade_kernel", kernel)
    out = []
    for n in (1, 1, 12):
        d.step(n)
        out.append([d.download(k) for k in ("conc", "conc1")])
    d.close()
    return out


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("odd", [*VALUES, "evaporation"])
@pytest.mark.parametrize("nr,nc,dxy,in_flight", [(95, 64, 2, 1), (47, 90, 3, 8)])
def test_both_kernels_agree(nr, nc, dxy, in_flight, odd, precision):
    rng = np.random.default_rng(nr)
    sc = S.plane_scenario(nr, nc, seed=nr)
    sc.dxy, sc.horizon, sc.d_coefs = dxy, 1e5, [0.01, 0.5]
    thin = rng.random((nr, nc)) < 0.2
    sc.init_h = np.where(thin, rng.uniform(0, 6e-5, (nr, nc)), rng.uniform(0, 0.05, (nr, nc)))
    sc.init_conc = [rng.uniform(0, 2, (nr, nc)) * (rng.random((nr, nc)) < 0.7) for _ in range(2)]
    if odd == "evaporation":
        sc.ks = 1e-6
        sc.meteo = ((0.0, -2000.0, 0.0), (1e5, -2000.0, 0.0))
    else:
        for c in sc.init_conc:
            at = rng.random((nr, nc)) < 0.01
            c[at] = rng.choice(VALUES[odd], at.sum())
    a, b = (_run(sc, precision, k, in_flight) for k in (1, 2))
    for i, (x, y) in enumerate(zip(a, b)):
        for k in range(2):
            assert np.array_equal(x[k], y[k], equal_nan=True), (i, k)
