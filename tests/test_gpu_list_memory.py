"""A large single system on a device that is nearly full.  The pair list has room for every pair
of 32-atom blocks (there is no overflow to handle), so the bytes of one possible tile decide the
largest system that fits: 1,373 with the tile arrays that the one-kernel list build replaced.
With that much free for each, and 2 KB an atom, the context must still fit; its list, built in
parts, and its gradient against the oracle and against the build in one launch.
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


def test_fits_in_the_earlier_bytes_of_a_possible_tile(eng_mod):
    import torch
    top = systems.solvated_polymer(0, 50500, seed=3)
    kw = dict(method=abi.JP_METHOD_MICR)
    o = oracle.Oracle(top, **kw)
    go = o.energy_grad()[1]
    with eng_mod.Engine(top, precision=abi.JP_PREC_MIXED, **kw) as e:
        nblk = e.list_stats()[2] // 32
        assert e.list_stats()[1] == o.npairs_listed
        g1 = e.energy_grad()[1]
        launches = e.launch_counts()[1]
    need = nblk * (nblk + 1) // 2 * 1373 + 2048 * top["natom"]
    ballast = torch.empty(torch.cuda.mem_get_info()[0] - need, dtype=torch.uint8, device="cuda")
    try:
        with eng_mod.Engine(top, precision=abi.JP_PREC_MIXED, **kw) as e:
            e.rebuild()
            assert e.launch_counts()[1] == launches + 2
            assert e.list_stats()[1] == o.npairs_listed
            g3 = e.energy_grad()[1]
    finally:
        del ballast
        torch.cuda.empty_cache()
    assert rms_rel(g1, go) < 1e-5
    np.testing.assert_array_equal(g1, g3)     # sums do not depend on the records' order
