"""Evaporation (a negative rate of the meteo file) can take a cell's last water
within a step. The reference then divides the diluted mass by a depth of 0
(common.cpp:226-234): NaN where there is no solute in the cell and the forcing,
else infinite, and what the sweep makes of its neighbours follows from that.
The same here, to the bounds of the other parity tests (1e-10), with the cells
that are no numbers in the same places (the FP32 state's quotient, a * (1 / b)
corrected, is NaN for any a / 0)."""
import numpy as np
import pytest

import gpu_pairs as GP
import pyoracle as P
from fluxos_cpp_b200 import scenarios as S

pytestmark = pytest.mark.gpu
RATE = -2000.0  # mm/day: about 0.05 mm a step of these grids


def _scenario(nr, nc, dxy, conc):
    sc = S.plane_scenario(nr, nc, seed=nr)
    sc.dxy, sc.horizon, sc.ks = dxy, 1e5, 1e-6
    sc.meteo = ((0.0, RATE, conc), (1e5, RATE, conc))
    rng = np.random.default_rng(nr + nc)
    thin = rng.random((nr, nc)) < 0.3
    sc.init_h = np.where(thin, rng.uniform(2e-6, 6e-5, (nr, nc)), rng.uniform(0.001, 0.05, (nr, nc)))
    sc.init_conc = [np.where(thin, 0.0, rng.uniform(0, 2, (nr, nc)))]
    return sc


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("nr,nc,dxy,conc", [(62, 75, 2, 0.0), (31, 40, 3, 0.0), (31, 40, 3, 1.0)])
def test_a_cell_that_loses_its_last_water(nr, nc, dxy, conc, precision, tmp_path):
    sc = _scenario(nr, nc, dxy, conc)
    sc.write(str(tmp_path))
    ora = P.OracleRun(str(tmp_path), sc, 1)
    ora.apply_wet_start(sc.init_h, None, None, sc.init_conc)
    d = GP.domain_from_oracle(ora, sc, 1) if precision == "fp64" else S.make_domain(sc, precision="fp32")
    GP.advance_oracle(ora, 1)  # no sweep in the first step: the dilution alone
    GP.advance_domain(d, 1)
    want, got = (a[1:-1, 1:-1] for a in (ora.grid("conc"), d.download("conc")))
    assert np.isnan(want).any() == (conc == 0.0) and np.isinf(want).any() == (conc != 0.0)
    assert np.array_equal(np.isfinite(want), np.isfinite(got))
    for n in (1, 20) if precision == "fp64" else ():
        GP.advance_oracle(ora, n)
        GP.advance_domain(d, n)
        _, bad = GP.compare(ora, d, sc)
        assert not bad, (n, bad)
        want, got = (a[1:-1, 1:-1] for a in (ora.grid("conc"), d.download("conc")))
        assert np.array_equal(np.isnan(want), np.isnan(got)) and np.array_equal(np.isinf(want), np.isinf(got)), n
    d.close()


@pytest.mark.parametrize("nr,nc,dxy", [(31, 40, 3), (62, 33, 2)])
def test_subnormal_depths_in_fp32(nr, nc, dxy):
    """The FP32 state's reciprocal of a subnormal depth is infinite, so a mass
    of 0 diluted over one is NaN: from both kernels of the sweep."""
    rng = np.random.default_rng(nr)
    sc = _scenario(nr, nc, dxy, 1.0)
    sc.meteo = ((0.0, 0.0, 0.0), (1e5, 0.0, 0.0))
    sc.dem = np.full((nr, nc), 1e-50)  # a level of 1e-40 is a depth of 1e-40
    sc.init_h = np.where(rng.random((nr, nc)) < 0.5, 1e-40, rng.uniform(0.001, 0.05, (nr, nc)))
    sc.init_conc = [rng.uniform(0, 2, (nr, nc)) * (rng.random((nr, nc)) < 0.5)]
    out = []
    for kernel in (1, 2):
        d = S.make_domain(sc, precision="fp32")
        d.set_option("ade_kernel", kernel)
        for n in (1, 4):
            d.step(n)
            out.append(d.download("conc"))
        d.close()
    assert np.isnan(out[0]).any()
    for a, b in zip(out[:2], out[2:]):
        assert np.array_equal(a, b, equal_nan=True)
