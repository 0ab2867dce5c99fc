"""Both kernels of the solute sweep on the same small grids, chosen by the
option "ade_kernel" (1: a warp per unit, fx_ade.cu; 2: a block per unit,
fx_ade_chain.cu). Where none is chosen the units at work decide, and grids
this small never take the first.

* Each against the oracle (FP64), to the 1e-10 of the other parity tests: walls
  and NODATA cells, point inflow, soil release, a melt field, cell sizes that
  are and are not powers of two, a dry start, the edges of strips.
* The two against one another in both precisions: the same IEEE expressions on
  the same operands, so the same bits.
* The bounded waits of each give up, are reported, and leave the device usable."""
import numpy as np
import pytest

import fluxos_cpp_b200 as fx
import gpu_pairs as GP
import pyoracle as P
from fluxos_cpp_b200 import scenarios as S

pytestmark = pytest.mark.gpu
KERNELS = (1, 2)


def _everything(nr, nc, dxy, nchem, seed):
    """Walls, NODATA, wet and dry cells, inflow, soil release, melt field, friction."""
    rng = np.random.default_rng(seed)
    sc = S.plane_scenario(nr, nc, seed=seed)
    sc.dxy, sc.horizon = dxy, 1e5
    sc.d_coefs = [0.01 * (k + 1) for k in range(nchem)]
    for _ in range(nr * nc // 200):
        sc.dem[rng.integers(0, nr), rng.integers(0, nc)] = -9999.0 if rng.random() < 0.5 else 0.0
    irow, icol = nr // 2, nc // 3
    sc.dem[nr - irow, icol - 1] = 100.3  # not a wall
    sc.inflow = ((0.0, 0.05, 4.0), (30.0, 0.0, 0.0), (60.0, 0.02, 1.0), (1e4, 0.05, 2.0))
    sc.inflow_xy = (icol * dxy, irow * dxy)
    sc.wintra, sc.soil_release_rate = True, 2.0
    sc.init_soil = rng.uniform(0, 100.0, (nr, nc)) * (rng.random((nr, nc)) < 0.8)
    sc.melt_mult = rng.uniform(0.25, 2.0, (nr, nc))
    sc.manning = rng.uniform(0.03, 0.15, (nr, nc))
    sc.init_h = np.where(rng.random((nr, nc)) < 0.6, rng.uniform(0, 0.03, (nr, nc)), 0.0)
    sc.init_conc = [np.where(sc.init_h > 0.01, 1.0 + k, 0.0) for k in range(nchem)]
    return sc


def _pair(sc, folder, kernel, in_flight):
    sc.write(folder)
    ora = P.OracleRun(folder, sc, 0)
    if sc.init_h is not None:
        ora.apply_wet_start(sc.init_h, None, None, sc.init_conc)
    if sc.init_soil is not None:
        ora.interior("soil_mass")[...] = sc.init_soil.T
    d = GP.domain_from_oracle(ora, sc, 0, steps_in_flight=in_flight)
    d.set_option("ade_kernel", kernel)
    return ora, d


def _compare(ora, d, sc, steps):
    for n in steps:
        GP.advance_oracle(ora, n)
        GP.advance_domain(d, n)
        _, bad = GP.compare(ora, d, sc)
        assert not bad, (n, bad)
    d.close()


@pytest.mark.parametrize("kernel", KERNELS)
@pytest.mark.parametrize("nr,nc,dxy,nchem,in_flight", [(95, 70, 3, 2, 7), (95, 70, 2, 1, 31), (70, 150, 10, 3, 1)])
def test_everything_against_the_oracle(nr, nc, dxy, nchem, in_flight, kernel, tmp_path):
    sc = _everything(nr, nc, dxy, nchem, seed=nr + dxy)
    ora, d = _pair(sc, str(tmp_path), kernel, in_flight)
    soil = ora.grid("soil_mass").sum()
    _compare(ora, d, sc, (1, 20, 150))
    assert ora.grid("soil_mass").sum() < 0.999 * soil  # the release happened


@pytest.mark.parametrize("kernel", KERNELS)
@pytest.mark.parametrize("in_flight", [1, 8])
def test_dry_start(in_flight, kernel, tmp_path):
    sc = S.plane_scenario(48, 40, seed=3)
    sc.meteo = ((0.0, 80.0, 1.0), (3000.0, 80.0, 1.0))
    sc.horizon = 3000.0
    ora, d = _pair(sc, str(tmp_path), kernel, in_flight)
    _compare(ora, d, sc, (1, 2, 3, 50, 400))


@pytest.mark.parametrize("nr,nc,dxy,nchem,in_flight", [
    (2, 2, 2, 1, 3), (2, 41, 3, 2, 7), (29, 3, 2, 1, 5), (30, 5, 1, 1, 5), (31, 64, 3, 1, 7), (60, 4, 2, 3, 9),
    (61, 33, 10, 1, 31), (89, 2, 2, 1, 5), (121, 70, 3, 2, 31)])
def test_strip_edges_of_the_warp_per_unit_kernel(nr, nc, dxy, nchem, in_flight, tmp_path):
    rng = np.random.default_rng(nr * 1000 + nc)
    sc = S.plane_scenario(nr, nc, seed=nr)
    sc.dxy, sc.horizon = dxy, 1e5
    sc.d_coefs = [0.01 * (k + 1) for k in range(nchem)]
    sc.init_h = np.where(rng.random((nr, nc)) < 0.8, rng.uniform(0, 0.05, (nr, nc)), 0.0)
    sc.init_conc = [rng.uniform(0, 2, (nr, nc)) * (sc.init_h > 0.02) for _ in range(nchem)]
    ora, d = _pair(sc, str(tmp_path), 1, in_flight)
    _compare(ora, d, sc, (1, 2, 40))


def _both(sc, precision, in_flight, steps):
    out = []
    for kernel in KERNELS:
        d = S.make_domain(sc, precision=precision, steps_in_flight=in_flight)
        d.set_option("ade_kernel", kernel)
        d.step(steps)
        out.append({k: d.download(k) for k in ["h", "soil_mass", "conc"] + [f"conc{k}" for k in range(1, sc.nchem)]})
        d.close()
    return out


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("nr,nc,dxy,nchem,in_flight", [(95, 70, 3, 2, 7), (121, 300, 2, 3, 31), (2, 41, 10, 1, 5)])
def test_both_kernels_agree(nr, nc, dxy, nchem, in_flight, precision):
    a, b = _both(_everything(nr, nc, dxy, nchem, seed=nr + dxy), precision, in_flight, 70)
    for k in a:
        assert np.isfinite(a[k]).all() and np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_both_kernels_agree_on_a_large_grid(precision):
    sc = S.fractal_scenario(1024, seed=3)
    sc.d_coefs = [0.01, 0.05, 0.2]
    S.wet_start(sc, depth=0.005)
    a, b = _both(sc, precision, 31, 31)
    for k in a:
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("kernel", KERNELS)
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_bounded_waits(precision, kernel):
    sc = S.plane_scenario(120, 90, seed=61)
    sc.horizon = 1e5
    S.wet_start(sc, depth=0.01)

    def domain():
        d = S.make_domain(sc, precision=precision, steps_in_flight=8)
        d.set_option("ade_kernel", kernel)
        return d

    d = domain()
    d.set_option("fail_ade_waits", 1)
    with pytest.raises(fx.FluxosError) as e:
        d.step(8)
    assert e.value.code == -5 and d.status()["device_error"] == 1
    with pytest.raises(fx.FluxosError):
        d.step(1)
    d.close()
    d = domain()
    assert d.step(8)["device_error"] == 0
    d.close()


def test_unknown_kernels_are_refused():
    d = fx.Domain(8, 8, 2)
    for v in (-1, 3):
        with pytest.raises(fx.FluxosError):
            d.set_option("ade_kernel", v)
    d.close()
