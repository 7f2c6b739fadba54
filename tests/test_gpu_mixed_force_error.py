"""The mixed path's rounding error of the forces, as a mean over nine kinds of systems (waters,
chains, ions, an ALSD replica; FP64 path as reference).  The bound is what a kernel with one i
atom a lane and at most 16 terms to an FP32 sum gives on the same systems: the packed kernel's
sums must not be coarser.  The mixed path is reproducible, so the figure is one number.
"""
import numpy as np
import pytest

from j_presto_b200 import abi, systems
from tests._util import rms_rel

pytestmark = pytest.mark.gpu
BOUND = 1.0184e-6     # one i atom a lane, 27 systems (three seeds of each kind)


@pytest.fixture(scope="module")
def eng_mod(engine_lib):
    from j_presto_b200 import engine
    return engine


def kinds(s):
    yield systems.water_box(2000, 40.0, seed=4 + s), {}
    yield systems.water_box(1000, 31.1, seed=1 + s), {}
    yield systems.water_box(700, 27.7, seed=31 + s), {}
    yield systems.water_box(5000, 53.5, seed=41 + s), {}
    yield systems.solvated_polymer(20, 5000, seed=7 + s), {}
    yield systems.solvated_polymer(12, 3000, seed=5000 + s), {}
    yield systems.solvated_polymer(6, 700, seed=11 + s), {}
    yield systems.solvated_polymer(0, 3000, nion_pairs=30, seed=13 + s), {}
    yield (systems.alsd_replica(systems.solvated_polymer(12, 3000, seed=5000 + s), seed=s),
           dict(method=abi.JP_METHOD_GE, alsd=abi.JP_ALSD_LMD, lambda0=0.8, scale_terms=abi.JP_SCALE_TORS))


def test_mean_force_error(eng_mod):
    err = []
    for s in range(3):
        for top, kw in kinds(s):
            kw = dict(dict(method=abi.JP_METHOD_CANO), **kw)
            g = []
            for prec in (abi.JP_PREC_MIXED, abi.JP_PREC_FP64):
                with eng_mod.Engine(top, precision=prec, **kw) as e:
                    g.append(e.energy_grad()[1])
            err.append(rms_rel(g[0], g[1]))
    assert np.mean(err) <= BOUND, np.mean(err)
