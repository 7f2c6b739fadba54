"""A batch stepped from host memory whose replicas differ in size on both sides of the box edge
where the largest blocks need per-pair images (small and large boxes in turn): the pair kernel
takes one image form for all of them.  With a form per replica both stood in the instruction
cache at once, and such a step's pair kernel took up to 1.7 times a resident step's; one form
for all takes some 1.15 times.  Energies of the host-state step are those of the resident one.
"""
import numpy as np
import pytest

from j_presto_b200 import abi, engine, systems

pytestmark = pytest.mark.gpu


def test_pair_time_of_a_host_state_step(engine_lib):
    small, large = systems.solvated_polymer(0, 3000, seed=5), systems.solvated_polymer(0, 7411, seed=6)
    with engine.Engine([small, large] * 8, precision=abi.JP_PREC_MIXED, method=abi.JP_METHOD_CANO, update=0) as e:
        n = sum(e.natoms)
        x, v = np.empty((n, 3)), np.empty((n, 3))
        e.set_timing(True)
        e.step(3, energies=False, temps=False)

        def pair(host):
            best = 1e9
            for _ in range(6):
                e.step_io(x if host else None, v if host else None, x, v, nsteps=1)
                _, ms, calls = e.last_timing()
                best = min(best, ms[0] / calls[0])
            return best

        resident = pair(False)
        host = pair(True)
    assert host < 1.4 * resident, (host, resident)
