"""A droplet inside its cut-off: each of its few half blocks has a hundred records and more, and many
warps add to the same i atoms' forces at once.  A record's pair time stays near that of a water
box of as many records (some 1.1 times; with every lane group adding its own sums 1.5 times).
"""
import pytest

from j_presto_b200 import abi, engine, systems

pytestmark = pytest.mark.gpu


def us_per_1000_records(top, **kw):
    with engine.Engine(top, precision=abi.JP_PREC_MIXED, method=abi.JP_METHOD_MICR, **kw) as e:
        e.set_timing(True)
        best = 1e9
        for _ in range(6):
            e.step(20, energies=False, temps=False)
            _, ms, calls = e.last_timing()
            best = min(best, ms[0] / calls[0])
        return 1e6 * best / e.list_stats()[0]


def test_pair_time_per_record(engine_lib):
    dense = us_per_1000_records(systems.droplet(8, 3050, seed=3), bounda=abi.JP_BOUND_NONE, cutoff=90.0)
    box = us_per_1000_records(systems.solvated_polymer(0, 16000, seed=3))
    assert dense < 1.3 * box, (dense, box)
