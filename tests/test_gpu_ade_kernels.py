"""The two kernels of the solute sweep (fx_ade.cu, fx_ade_chain.cu). Launches
with few units in flight take the chain kernel, others the sweep kernel; a
context's results do not depend on which.

* The chain kernel against the oracle at the edges of its work split: strips
  of 30 rows with 1, 29, 30 rows left over, fewer columns than a round of
  warp steps, cell sizes that are and are not powers of two (divisions by
  dxy), one to three solutes. Both sides evaluate the same IEEE expressions,
  so the bound is the one of the other parity tests, 1e-10.
* The same domain through both kernels (31 steps in flight put more units to
  work than the chain kernel takes, 4 do not): identical bits."""
import numpy as np
import pytest

import gpu_pairs as GP
import pyoracle as P
from fluxos_cpp_b200 import scenarios as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr,nc,dxy,nchem,in_flight", [
    (2, 2, 2, 1, 3), (2, 41, 3, 2, 7), (29, 3, 2, 1, 5), (30, 5, 1, 1, 5), (31, 64, 3, 1, 7), (60, 4, 2, 3, 9),
    (61, 33, 10, 1, 31), (89, 2, 2, 1, 5), (121, 70, 3, 2, 31)])
def test_chain_kernel_edges(nr, nc, dxy, nchem, in_flight, tmp_path):
    rng = np.random.default_rng(nr * 1000 + nc)
    sc = S.plane_scenario(nr, nc, seed=nr)
    sc.dxy, sc.horizon = dxy, 1e5
    if nchem > 1:
        sc.d_coefs = [0.01 * (k + 1) for k in range(nchem)]
    if nr > 8 and nc > 8:
        sc.dem[3:5, 4:7] = -9999.0
    sc.write(str(tmp_path))
    ora = P.OracleRun(str(tmp_path), sc, 0)
    h = np.where(rng.random((nr, nc)) < 0.8, rng.uniform(0, 0.05, (nr, nc)), 0.0)
    ora.apply_wet_start(h, None, None, [rng.uniform(0, 2, (nr, nc)) * (h > 0.02) for _ in range(nchem)])
    d = GP.domain_from_oracle(ora, sc, 0, steps_in_flight=in_flight)
    for n in (1, 2, 40):
        GP.advance_oracle(ora, n)
        GP.advance_domain(d, n)
        _, bad = GP.compare(ora, d, sc)
        assert not bad, (n, bad)
    d.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_chain_and_sweep_kernels_agree(precision):
    sc = S.fractal_scenario(1024, seed=3)
    sc.d_coefs = [0.01, 0.05, 0.2]
    S.wet_start(sc, depth=0.005)
    got = []
    for in_flight in (31, 4):
        d = S.make_domain(sc, precision=precision, steps_in_flight=in_flight)
        d.step(31)
        got.append({k: d.download(k) for k in ("h", "qx", "conc", "conc1", "conc2")})
        d.close()
    for k, a in got[0].items():
        assert np.array_equal(a, got[1][k]), k
