"""A batch's solute sweep through each of its two kernels (option
"ade_kernel"; where none is chosen only large ensembles take the one with a
warp per unit): every member's bits are those of the member alone, through the
other kernel. Members of very different sizes, whose units are merged by the
time they are needed, with their own number of solutes, forcing, walls,
inflow and soil release, one without solutes, and one that joins later; more
units than the GPU holds of either kernel, and fewer."""
import numpy as np
import pytest

import fluxos_cpp_b200 as fx
from fluxos_cpp_b200 import scenarios as S
from test_gpu_ade_forced import KERNELS, _everything

pytestmark = pytest.mark.gpu


def _scenarios(large):
    scs = [_everything(95, 70, 3, 2, seed=1), _everything(31, 140, 2, 1, seed=2), _everything(200, 61, 10, 3, seed=3)]
    dry = S.plane_scenario(64, 70, seed=9)
    dry.horizon, dry.ade = 1e5, False
    scs.append(dry)
    if large:
        big = S.fractal_scenario(700, seed=5)
        big.d_coefs = [0.01 * (k + 1) for k in range(6)]
        S.wet_start(big, depth=0.005)
        scs.insert(1, big)
    return scs


def _fields(d):
    return {k: d.download(k) for k in ["h", "soil_mass", "conc"] + [f"conc{k}" for k in range(1, d.nchem)]}


@pytest.mark.parametrize("kernel", KERNELS)
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("large,in_flight", [(False, 5), (True, 31)])
def test_members_of_a_batch_through_each_kernel(large, in_flight, precision, kernel):
    scs = _scenarios(large)
    steps, late = 2 * in_flight + 1, in_flight + 2
    doms = [S.make_domain(sc, precision=precision, steps_in_flight=in_flight) for sc in scs]
    b = fx.Batch()
    b.set_option("ade_kernel", kernel)
    for d in doms[1:]:
        b.add(d)
    b.step(steps - late)
    b.add(doms[0])
    b.step(late)
    for i, (sc, d) in enumerate(zip(scs, doms)):
        alone = S.make_domain(sc, precision=precision, steps_in_flight=in_flight)
        alone.set_option("ade_kernel", 3 - kernel)
        alone.step(steps if i else late)
        for k, a in _fields(alone).items():
            assert np.array_equal(a, d.download(k)), (i, k)
        alone.close()
    b.close()
    for d in doms:
        d.close()


def test_unknown_kernels_are_refused():
    b = fx.Batch()
    for v in (-1, 3):
        with pytest.raises(fx.FluxosError):
            b.set_option("ade_kernel", v)
    b.close()
