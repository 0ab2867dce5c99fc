"""The solute sweep's units in the order of their starts: a launch with more
units than the GPU holds (steps x solutes x strips) gives the bits of launches
of one step, through the sweep kernel (many units at work) and the chain kernel
(few), and a batch of domains of very different sizes, whose units are merged
by the time they are needed, the bits of each domain alone. The same IEEE
expressions on the same operands in every order the dependencies allow, so the
comparison is exact."""
import numpy as np
import pytest

import fluxos_cpp_b200 as fx
from fluxos_cpp_b200 import scenarios as S

pytestmark = pytest.mark.gpu
FIELDS = ("h", "qx", "conc", "conc1")


def _domain(n, precision, in_flight, nchem=2):
    sc = S.fractal_scenario(n, seed=n)
    sc.d_coefs = [0.01 * (k + 1) for k in range(nchem)]
    S.wet_start(sc, depth=0.005)
    return S.make_domain(sc, precision=precision, steps_in_flight=in_flight)


def _fields(d):
    return {k: d.download(k) for k in FIELDS}


@pytest.mark.parametrize("n,nchem,in_flight", [(1024, 4, 63), (512, 2, 63), (130, 2, 7)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_many_steps_in_flight_equal_one_by_one(n, nchem, in_flight, precision):
    got = []
    for k in (in_flight, 1):
        d = _domain(n, precision, k, nchem)
        d.step(in_flight)
        got.append(_fields(d))
        d.close()
    for k, a in got[0].items():
        assert np.array_equal(a, got[1][k]), k


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_a_batch_of_unequal_domains_equals_each_alone(precision):
    sizes, steps = (64, 700, 131, 301), 20
    b = fx.Batch()
    doms = [_domain(n, precision, steps) for n in sizes]
    for d in doms:
        b.add(d)
    b.set_option("steps_in_flight", steps)
    b.step(steps)
    for n, d in zip(sizes, doms):
        alone = _domain(n, precision, steps)
        alone.step(steps)
        for k, a in _fields(alone).items():
            assert np.array_equal(a, d.download(k)), (n, k)
        alone.close()
