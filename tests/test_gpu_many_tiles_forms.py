"""The list build's other forms on i-blocks with more tiles than its shared-memory cache and its
16-bit entry list hold (a droplet of 9,300 atoms inside its cut-off): ALSD's two record
sequences with the 32-bit entry windows, and the H-bond list from tiles in global memory.
Against the oracle at the suite's tolerances.
"""
import numpy as np
import pytest

import oracle
from j_presto_b200 import abi, systems
from tests._util import rms_rel

pytestmark = pytest.mark.gpu
FP64, MIXED = abi.JP_PREC_FP64, abi.JP_PREC_MIXED
KW = dict(bounda=abi.JP_BOUND_NONE, cutoff=90.0)


@pytest.fixture(scope="module")
def eng_mod(engine_lib):
    from j_presto_b200 import engine
    return engine


@pytest.fixture(scope="module")
def drop():
    top = systems.droplet(8, 3050, seed=3)
    assert top["natom"] > 32 * 270
    return top


def check(eng_mod, top, kw, classes):
    o = oracle.Oracle(top, **kw)
    eo, go = o.energy_grad()
    for prec, gtol, rtol, atol in ((FP64, 1e-12, 1e-8, 1e-7), (MIXED, 1e-5, 1e-5, 1e-2)):
        with eng_mod.Engine(top, precision=prec, **kw) as e:
            ene, g = e.energy_grad()
            assert e.pair_count() == o.npairs_cut
            assert e.list_stats()[1] == o.npairs_listed
            if classes:
                np.testing.assert_allclose(e.get_lambda()[1], o.get_lambda()[1], rtol=rtol, atol=atol)
        assert rms_rel(g, go) < gtol
        np.testing.assert_allclose(ene, eo, rtol=rtol, atol=atol)
    return eo


def test_alsd_sequences(eng_mod, drop):
    top = systems.alsd_replica(dict(drop), ncluster=2, seed=1)
    check(eng_mod, top, dict(KW, method=abi.JP_METHOD_GE, alsd=abi.JP_ALSD_LMD, lambda0=0.8), True)


def test_hbond_list(eng_mod, drop):
    top = systems.with_hbond(dict(drop))
    eo = check(eng_mod, top, dict(KW, method=abi.JP_METHOD_CANO), False)
    assert eo[abi.JP_E_HBOND] < -1.0
