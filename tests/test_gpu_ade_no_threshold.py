"""A dry threshold (ROUGNESS_HEIGHT) of 0: a cell at its bed counts as wet, so
the sweep re-scales its concentration by a depth of 0 (ADEsolver_calc.cpp:64-72:
0 / 0), bounds what follows by the neighbours, and hands fluxes on. FP64 against the
oracle, to the 1e-10 of the other parity tests, and the two kernels of the
sweep against one another, bit for bit, in both precisions."""
import numpy as np
import pytest

import gpu_pairs as GP
import pyoracle as P
from fluxos_cpp_b200 import scenarios as S

pytestmark = pytest.mark.gpu


def _scenario(nr, nc, dxy):
    rng = np.random.default_rng(nr)
    sc = S.plane_scenario(nr, nc, seed=nr)
    sc.dxy, sc.horizon, sc.ks = dxy, 1e5, 0.0
    sc.meteo = ((0.0, 0.0, 0.0), (1e5, 0.0, 0.0))
    sc.init_h = np.where(rng.random((nr, nc)) < 0.6, rng.uniform(0.001, 0.05, (nr, nc)), 0.0)
    sc.init_conc = [rng.uniform(0, 2, (nr, nc)) * (rng.random((nr, nc)) < 0.7)]
    return sc


@pytest.mark.parametrize("kernel", [1, 2])
@pytest.mark.parametrize("nr,nc,dxy", [(62, 75, 2), (31, 40, 3)])
def test_against_the_oracle(nr, nc, dxy, kernel, tmp_path):
    sc = _scenario(nr, nc, dxy)
    sc.write(str(tmp_path))
    ora = P.OracleRun(str(tmp_path), sc, 1)
    ora.apply_wet_start(sc.init_h, None, None, sc.init_conc)
    d = GP.domain_from_oracle(ora, sc, 1)
    d.set_option("ade_kernel", kernel)
    for n in (1, 1):
        GP.advance_oracle(ora, n)
        GP.advance_domain(d, n)
        a, b = ora.interior("conc"), d.download("conc")[1:-1, 1:-1]
        assert np.array_equal(np.isnan(a), np.isnan(b))
        assert GP.rel_err(a, b, 1e-6 * np.nanmax(np.abs(a))) <= 1e-10
    d.close()


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("nr,nc,dxy,in_flight", [(62, 75, 2, 5), (31, 40, 3, 1)])
def test_both_kernels_agree(nr, nc, dxy, in_flight, precision):
    sc = _scenario(nr, nc, dxy)
    out = []
    for kernel in (1, 2):
        d = S.make_domain(sc, precision=precision, steps_in_flight=in_flight)
        d.set_option("ade_kernel", kernel)
        for n in (2, 8):
            d.step(n)
            out.append((kernel, d.download("conc")))
        d.close()
    for (_, a), (_, b) in zip(out[:2], out[2:]):
        assert np.array_equal(a, b, equal_nan=True)
