"""The FP64 step's quotients over shared reciprocals (fx_hydro.cu: Over,
over). They are the correctly rounded a / b, so the step gives the oracle's
bits whatever the numerators: zeros of both signs, ordinary ones, and ones so
small (down to subnormal) that the corrections' residuals would not be exact
and the division itself runs. Every tile height, cell sizes that are no power
of two, melt multipliers and friction; the closed edge mode, so that no edge
weir's pow takes part."""
import numpy as np
import pytest

import gpu_pairs as GP
import pyoracle as P
from fluxos_cpp_b200 import scenarios as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile_rows", [4, 8, 16])
@pytest.mark.parametrize("nr,nc,dxy", [(65, 23, 3), (30, 40, 10), (31, 7, 2)])
def test_quotients_give_the_oracles_bits(nr, nc, dxy, tile_rows, tmp_path):
    rng = np.random.default_rng(nr + dxy)
    sc = S.plane_scenario(nr, nc, seed=nr)
    sc.dxy, sc.horizon = dxy, 1e5
    sc.manning = np.where(rng.random((nr, nc)) < 0.8, rng.uniform(0.01, 0.2, (nr, nc)), 0.0)
    sc.melt_mult = rng.uniform(0, 2, (nr, nc))
    sc.write(str(tmp_path))
    ora = P.OracleRun(str(tmp_path), sc, 1)
    h = np.where(rng.random((nr, nc)) < 0.8, rng.uniform(0, 0.05, (nr, nc)), 0.0)
    q = [rng.choice([0.0, -0.0, 1.0, -1.0], (nr, nc)) * rng.choice([1e-3, 1e-100, 1e-215, 1e-300, 1e-320], (nr, nc)) *
         (h > 0) for _ in range(2)]
    ora.apply_wet_start(h, q[0], q[1], [np.where(h > 0.02, 1.0, 0.0)])
    d = GP.domain_from_oracle(ora, sc, 1)
    d.set_option("tile_rows", tile_rows)
    for n in (1, 2, 20):
        GP.advance_oracle(ora, n)
        GP.advance_domain(d, n)
        _, bad = GP.compare(ora, d, sc, rtol=0.0)
        bad.pop("conc", None)  # the solute sweep has tests of its own
        assert not bad, (n, bad)
    d.close()
