"""Two live contexts whose LJ tables differ in size: a context created later, with fewer types,
must leave the earlier one's kernels as they were -- its evaluations, its steps (whose graph is
captured after the second context exists) and its minimisation.  Against the oracle at the
suite's tolerances.
"""
import numpy as np
import pytest

import oracle
from j_presto_b200 import abi, systems
from tests._util import rms_rel
from tests.test_gpu_pair_packed import spread_types

pytestmark = pytest.mark.gpu
FP64, MIXED = abi.JP_PREC_FP64, abi.JP_PREC_MIXED


@pytest.fixture(scope="module")
def eng_mod(engine_lib):
    from j_presto_b200 import engine
    return engine


def waters_with(ntype):
    """A water box whose tables hold its own two types among `ntype`."""
    top = systems.solvated_polymer(0, 700, seed=3)
    keep = [systems.T_OW, systems.T_HW] + [t for t in range(9) if t not in (systems.T_OW, systems.T_HW)]
    new = np.argsort(keep)
    keep = keep[:ntype]
    return dict(top, ntype=ntype, c6=top["c6"][np.ix_(keep, keep)], c12=top["c12"][np.ix_(keep, keep)],
                s14_vdw=top["s14_vdw"][keep], s14_ele=top["s14_ele"][keep],
                atype=new[top["atype"]].astype(np.int32))


@pytest.mark.parametrize("big,small", [(9, 2), (9, 3), (11, 9), (27, 13)])
@pytest.mark.parametrize("prec,alsd", [(FP64, False), (MIXED, False), (MIXED, True)])
def test_smaller_tables_later(eng_mod, prec, alsd, big, small):
    kw, lam = dict(method=abi.JP_METHOD_CANO, cutoff=9.0), {}
    top = spread_types(systems.solvated_polymer(6, 700, seed=17), big)
    if alsd:
        top = systems.alsd_replica(top, ncluster=2, seed=1)
        lam = dict(alsd=abi.JP_ALSD_LMD, lambda0=0.8)
        kw["method"] = abi.JP_METHOD_GE
    later = waters_with(small) if small < 9 else spread_types(systems.solvated_polymer(0, 700, seed=3), small)
    o = oracle.Oracle(top, **kw, **lam)
    eo, go = o.energy_grad()
    gtol, rtol, atol, xtol = (1e-12, 1e-8, 1e-7, 1e-8) if prec == FP64 else (1e-5, 1e-5, 1e-2, 1e-4)
    with eng_mod.Engine(top, precision=prec, **kw, **lam) as e:
        with eng_mod.Engine(later, precision=prec, method=abi.JP_METHOD_CANO, cutoff=9.0) as f:
            f.energy_grad()
            ene, g = e.energy_grad()
            assert rms_rel(g, go) < gtol
            np.testing.assert_allclose(ene, eo, rtol=rtol, atol=atol)
            e.step(3)
            x, _ = e.get_state()
    assert o.run(3)[0] == 0
    assert np.abs(x - o.get_state()[0]).max() < xtol


@pytest.mark.parametrize("prec", [FP64, MIXED])
def test_steps_captured_later(eng_mod, prec):
    """The step graph alone (no evaluation before it that would report a refused launch)."""
    kw = dict(method=abi.JP_METHOD_CANO, cutoff=9.0)
    top = systems.solvated_polymer(6, 700, seed=17)
    o = oracle.Oracle(top, **kw)
    assert o.run(3)[0] == 0
    with eng_mod.Engine(top, precision=prec, **kw) as e, eng_mod.Engine(waters_with(2), precision=prec, **kw):
        e.step(3)
        x, _ = e.get_state()
    assert np.abs(x - o.get_state()[0]).max() < (1e-8 if prec == FP64 else 1e-4)


@pytest.mark.parametrize("prec", [FP64, MIXED])
def test_minimisation_later(eng_mod, prec):
    kw = dict(shake_method=abi.JP_SHAKE_NONE, cutoff=9.0)
    top = systems.solvated_polymer(6, 700, seed=17)
    with eng_mod.Engine(top, precision=prec, **kw) as e:
        alone = e.minimize(max_loop=12, convgr=1e-3)[1]
    with eng_mod.Engine(top, precision=prec, **kw) as e, eng_mod.Engine(waters_with(2), precision=prec, **kw):
        pair = e.minimize(max_loop=12, convgr=1e-3)[1]
    # (sums vary in their last bits with the order of the atomics)
    np.testing.assert_allclose(pair, alone, rtol=1e-9)
