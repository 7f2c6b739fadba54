"""A batch of many small boxes, where most but not all pair records need an image per pair: the
packed pair kernel takes the records of one image form after those of the other.  In turn, both
forms' code competed for the instruction cache, and a record took 1.7 times what it takes in
boxes of 45 A; apart, some 1.2 times.
"""
import pytest

from j_presto_b200 import abi, engine, systems

pytestmark = pytest.mark.gpu


def us_per_1000_records(tops):
    with engine.Engine(tops, precision=abi.JP_PREC_MIXED, method=abi.JP_METHOD_MICR) as e:
        e.set_timing(True)
        best = 1e9
        for _ in range(6):
            e.step(20, energies=False, temps=False)
            _, ms, calls = e.last_timing()
            best = min(best, ms[0] / calls[0])
        return 1e6 * best / e.list_stats()[0]


def test_pair_time_per_record(engine_lib):
    small = us_per_1000_records([systems.solvated_polymer(0, 700, seed=s % 3) for s in range(60)])
    large = us_per_1000_records([systems.solvated_polymer(0, 3000, seed=s % 3) for s in range(14)])
    assert small < 1.4 * large, (small, large)
