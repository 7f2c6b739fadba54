"""The FP64 pair kernel on both sides of its image rule (an i block's atoms and the entries in
their images nearest to the block, where half the box exceeds the cut-off by the block's half
extent and 2 A; else an image per pair), after coordinates were put into other images without
a list build, and on lists of a few records.  Against the oracle: gradient RMS relative
1e-12, energies 1e-8 relative.
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


@pytest.mark.parametrize("shift", [False, True])
@pytest.mark.parametrize("nwat", [700, 1300, 1800, 2500])   # boxes of 28, 34, 38 and 42 A
def test_energy_grad_vs_oracle(eng_mod, nwat, shift):
    top = systems.solvated_polymer(0, nwat, seed=31, nion_pairs=2)
    kw = dict(method=abi.JP_METHOD_MICR)
    o = oracle.Oracle(top, **kw)
    eo, go = o.energy_grad()
    x = top["cord"] + 0.0
    if shift:   # whole molecules by whole box lengths; the energy and the gradient stay
        mol = np.concatenate([[0], np.cumsum(np.diff(top["molecule"] != systems.MOL_WATER) | (top["atype"][1:] == systems.T_OW))])
        x += np.random.default_rng(1).integers(-1, 2, (mol.max() + 1, 3))[mol] * top["box"]
    with eng_mod.Engine(top, precision=abi.JP_PREC_FP64, **kw) as e:
        ene, g = e.energy_grad(cord=x) if shift else e.energy_grad()
        assert e.pair_count() == o.npairs_cut
    # an image shift rounds a coordinate of up to 84 A once more: 2^-53 * 128 A in a distance
    assert rms_rel(g, go) < 1e-12
    np.testing.assert_allclose(ene, eo, rtol=1e-8, atol=1e-7)
