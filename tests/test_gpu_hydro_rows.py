"""The tile height that the grid's size decides (fx_default_tile_rows) against
a set one: the same bits, alone and in a batch, on each side of the lines (all
tiles of 4 rows resident at once or not; ten tiles of 16 rows a block or not,
FP32; fewer columns than a staged tile of 16 rows). Each cell's step is the
same expressions on the same operands in every tile shape, so the comparison
is exact."""
import numpy as np
import pytest

import fluxos_cpp_b200 as fx
from fluxos_cpp_b200 import scenarios as S

pytestmark = pytest.mark.gpu
FIELDS = ("z", "h", "qx", "qy", "fe_1", "fn_1", "twet", "conc")


def _run(sizes, precision, rows, steps=6):
    doms = []
    for nr, nc in sizes:
        sc = S.plane_scenario(nr, nc, seed=nr + nc)
        sc.horizon = 1e5
        S.wet_start(sc, depth=0.01)
        doms.append(S.make_domain(sc, precision=precision, steps_in_flight=steps))
    if len(doms) == 1:
        if rows:
            doms[0].set_option("tile_rows", rows)
        doms[0].step(steps)
    else:
        b = fx.Batch()
        if rows:
            b.set_option("tile_rows", rows)
        for d in doms:
            b.add(d)
        b.step(steps)
    return [{k: d.download(k) for k in FIELDS} for d in doms]


@pytest.mark.parametrize("sizes,precision", [
    ([(217, 300)], "fp64"), ([(217, 330)], "fp64"), ([(1300, 1300)], "fp32"), ([(1100, 1000)], "fp32"),
    ([(95, 14), (200, 90)], "fp64"), ([(1400, 1300), (61, 15)], "fp32"), ([(1400, 1300), (61, 80)], "fp32")])
def test_default_tile_height_gives_the_same_bits(sizes, precision):
    for a, b in zip(_run(sizes, precision, 0), _run(sizes, precision, 8)):
        for k in FIELDS:
            assert np.array_equal(a[k], b[k]), k
