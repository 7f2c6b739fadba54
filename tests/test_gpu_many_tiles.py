"""i-blocks with more tiles than the list build keeps in shared memory and than its 16-bit
entry list takes: a free droplet of 9,300 atoms in a cut-off that spans it (every later block
is a tile of the first ones: above 256), against the oracle at the suite's tolerances.
"""
import numpy as np
import pytest

import oracle
from j_presto_b200 import abi, systems
from tests._util import rms_rel

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng_mod(engine_lib):
    from j_presto_b200 import engine
    return engine


def test_cutoff_over_the_whole_system(eng_mod):
    top = systems.droplet(8, 3050, seed=3)
    assert top["natom"] > 32 * 270
    kw = dict(method=abi.JP_METHOD_CANO, bounda=abi.JP_BOUND_NONE, cutoff=90.0)
    o = oracle.Oracle(top, **kw)
    eo, go = o.energy_grad()
    for prec, gtol, rtol, atol in ((abi.JP_PREC_FP64, 1e-12, 1e-8, 1e-7), (abi.JP_PREC_MIXED, 1e-5, 1e-5, 1e-2)):
        with eng_mod.Engine(top, precision=prec, **kw) as e:
            ene, g = e.energy_grad()
            assert e.pair_count() == o.npairs_cut
            assert e.list_stats()[1] == o.npairs_listed
        assert rms_rel(g, go) < gtol
        np.testing.assert_allclose(ene, eo, rtol=rtol, atol=atol)
