"""The per-phase integrator (systems beyond the cooperative grid; forced here by a one-block
grid) on warps whose units are whole runs of waters and on the others: water counts around a
warp's 32 units, a chain whose units break the runs, a batch in which a warp spans two
replicas, per-sub-system temperatures.  Against the oracle over 10 steps with the suite's
trajectory tolerances: 1e-8 A (FP64), 1e-4 A (mixed).
"""
import numpy as np
import pytest

import oracle
from j_presto_b200 import abi, systems

pytestmark = pytest.mark.gpu

FP64, MIXED = abi.JP_PREC_FP64, abi.JP_PREC_MIXED


@pytest.fixture(scope="module")
def eng_mod(engine_lib):
    from j_presto_b200 import engine
    return engine


SETS = {
    "waters_256": [(0, 256, 0)], "waters_257": [(0, 257, 0)], "waters_255": [(0, 255, 0)],
    "ions": [(0, 300, 3)],
    "chain": [(6, 500, 0)],
    "batch": [(0, 260, 0), (4, 400, 0), (0, 271, 2)],
}


@pytest.mark.parametrize("prec,tol", [(FP64, 1e-8), (MIXED, 1e-4)])
@pytest.mark.parametrize("tempco", [1, 2])
@pytest.mark.parametrize("name", list(SETS))
def test_phase_launches_vs_oracle(eng_mod, name, tempco, prec, tol):
    tops = [systems.solvated_polymer(r, w, nion_pairs=i, seed=5 + k) for k, (r, w, i) in enumerate(SETS[name])]
    kw = dict(method=abi.JP_METHOD_CANO, tempco=tempco, cutoff=7.0)
    with eng_mod.Engine(tops if len(tops) > 1 else tops[0], precision=prec, **kw) as e:
        e.set_grid_limit(1)
        e.step(10)
        got = [e.get_state(rep=r) for r in range(len(tops))]
    for top, (x, v) in zip(tops, got):
        o = oracle.Oracle(top, **kw)
        assert o.run(10)[0] == 0
        xo, vo = o.get_state()
        assert np.abs(x - xo).max() < tol
        # a position error of tol between two steps is a velocity error of tol / dt at most twice
        assert np.abs(v - vo).max() < 2.0 * tol / 1.0


@pytest.mark.parametrize("prec,tol", [(FP64, 1e-8), (MIXED, 1e-4)])
def test_partial_scaling_vs_oracle(eng_mod, prec, tol):
    """The class-1 gradient of a partial-McMD replica scaled apart, its class holding waters."""
    top = dict(systems.solvated_polymer(6, 500, seed=21))
    top["cluster"] = (np.arange(top["natom"]) >= top["natom"] - 3 * 200).astype(np.int32)
    kw = dict(method=abi.JP_METHOD_CANO, alsd=abi.JP_GEPS_AND, psetmp=600.0, cutoff=7.0)
    o = oracle.Oracle(top, **kw)
    assert o.run(10)[0] == 0
    xo, _ = o.get_state()
    with eng_mod.Engine(top, precision=prec, **kw) as e:
        e.set_grid_limit(1)
        e.step(10)
        x, _ = e.get_state()
    assert np.abs(x - xo).max() < tol
