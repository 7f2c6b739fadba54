"""The packed pair kernel leaves the LJ term out over entries of types without one: no such
type, some (waters' hydrogens), all types, and a tile of ions and waters whose record groups mix
both.  Energies, gradients and pair counts against the oracle at the suite's mixed tolerances
(gradient RMS relative 1e-5, energies 1e-5 relative or 1e-2); ALSD classes likewise.
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


def _top(kind):
    top = dict(systems.solvated_polymer(6, 700, nion_pairs=8, seed=9))
    c6, c12 = top["c6"].copy(), top["c12"].copy()
    if kind == "none":          # every type with an LJ term: the water hydrogens take the polar H's
        h, w = systems.T_H, systems.T_HW
        for t in (c6, c12):
            t[w], t[:, w] = t[h], t[:, h]
            t[w, w] = t[h, h]
    elif kind == "all":
        c6[:], c12[:] = 0.0, 0.0
    elif kind == "one":         # an LJ term between one pair of types alone
        keep = np.zeros_like(c6)
        keep[systems.T_NA, systems.T_OW] = keep[systems.T_OW, systems.T_NA] = 1.0
        c6, c12 = c6 * keep, c12 * keep
    top["c6"], top["c12"] = c6, c12
    return top


@pytest.mark.parametrize("alsd", [0, 1])
@pytest.mark.parametrize("kind", ["some", "none", "all", "one"])
def test_lj_free_entries_vs_oracle(eng_mod, kind, alsd):
    top = _top(kind)
    kw = dict(method=abi.JP_METHOD_CANO, cutoff=8.0)
    if alsd:
        top["cluster"] = (np.arange(top["natom"]) < 30).astype(np.int32)
        kw.update(alsd=abi.JP_ALSD_LMD, lambda0=0.7)
        top["shake_n"], top["shake_atoms"] = top["shake_n"][:0], top["shake_atoms"][:0]
        top["shake_dist"] = top["shake_dist"][:0]
        kw["shake_method"] = abi.JP_SHAKE_NONE
    o = oracle.Oracle(top, **kw)
    eo, go = o.energy_grad()
    with eng_mod.Engine(top, precision=abi.JP_PREC_MIXED, **kw) as e:
        ene, g = e.energy_grad()
        assert e.pair_count() == o.npairs_cut
    assert rms_rel(g, go) < 1e-5
    np.testing.assert_allclose(ene, eo, rtol=1e-5, atol=1e-2)


@pytest.mark.parametrize("kind", ["some", "none", "all", "one"])
def test_lj_free_entries_fp64(eng_mod, kind):
    """The FP64 kernel's groups without the LJ term: the suite's FP64 tolerances."""
    top = _top(kind)
    kw = dict(method=abi.JP_METHOD_CANO, cutoff=8.0)
    o = oracle.Oracle(top, **kw)
    eo, go = o.energy_grad()
    with eng_mod.Engine(top, precision=abi.JP_PREC_FP64, **kw) as e:
        ene, g = e.energy_grad()
        assert e.pair_count() == o.npairs_cut
    assert rms_rel(g, go) < 1e-12
    np.testing.assert_allclose(ene, eo, rtol=1e-8, atol=1e-7)
