"""The packed pair kernel at the edges of its dispatch: type counts on both sides of the
type-triple table's limit (it ends at 11 types and the dummy one), boxes with and without
per-pair images, plain and ALSD contexts, lists of a few records.  Mixed path against the
oracle with the suite's tolerances: gradient RMS relative 1e-5, energies 1e-5 relative.
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


def spread_types(top, ntype, seed=5):
    """The same system with its nine types spread over `ntype` equal copies of them."""
    rng = np.random.default_rng(seed)
    src = np.concatenate([np.arange(9), rng.integers(0, 9, ntype - 9)])
    t = dict(top, ntype=ntype, c6=top["c6"][np.ix_(src, src)], c12=top["c12"][np.ix_(src, src)],
             s14_vdw=top["s14_vdw"][src], s14_ele=top["s14_ele"][src])
    t["atype"] = np.array([rng.choice(np.flatnonzero(src == a)) for a in top["atype"]], np.int32)
    return t


@pytest.mark.parametrize("ntype", [9, 11, 12, 27])
@pytest.mark.parametrize("nwat,nres,alsd", [(700, 0, False), (3601, 6, False), (700, 6, True), (3601, 6, True)])
def test_energy_grad_vs_oracle(eng_mod, ntype, nwat, nres, alsd):
    top = spread_types(systems.solvated_polymer(nres, nwat, seed=17), ntype)
    kw = dict(method=abi.JP_METHOD_MICR)
    if alsd:
        top = systems.alsd_replica(top, ncluster=2, seed=1)
        kw = dict(method=abi.JP_METHOD_GE, alsd=abi.JP_ALSD_LMD, lambda0=0.8)
    o = oracle.Oracle(top, **kw)
    eo, go = o.energy_grad()
    with eng_mod.Engine(top, precision=abi.JP_PREC_MIXED, **kw) as e:
        ene, g = e.energy_grad()
        # FP32 places a pair within 4e-6 A of the cut-off on either side: 1e-6 of the pairs
        assert abs(e.pair_count() - o.npairs_cut) <= 2 + 1e-5 * o.npairs_cut
        if alsd:
            np.testing.assert_allclose(e.get_lambda()[1], o.get_lambda()[1], rtol=1e-5, atol=1e-2)
    assert rms_rel(g, go) < 1e-5
    np.testing.assert_allclose(ene, eo, rtol=1e-5, atol=1e-2)


@pytest.mark.parametrize("natom", [2, 33, 65, 130])
def test_few_records(eng_mod, natom):
    """Lone ions on a lattice: lists of one to a few records, most lanes of a group empty."""
    n = int(np.ceil(natom ** (1 / 3)))
    x = np.stack(np.meshgrid(*[3.6 * np.arange(n)] * 3, indexing="ij"), -1).reshape(-1, 3)[:natom] + 5.0
    x += np.random.default_rng(natom).uniform(-0.3, 0.3, x.shape)
    ion = dict(systems.solvated_polymer(0, 1, nion_pairs=1, seed=3))
    empty = {k: v[:0] for k, v in ion.items() if isinstance(v, np.ndarray) and k.split("_")[0] in
             ("bond", "angle", "tors", "impr", "shake")}
    typ = np.where(np.arange(natom) % 2 == 0, systems.T_NA, systems.T_CL).astype(np.int32)
    top = dict(ion, **empty, natom=natom, cord=x, vel=np.zeros_like(x), box=np.full(3, 40.0), atype=typ,
               mass=np.full(natom, 30.0), charge=np.where(np.arange(natom) % 2 == 0, 1.0, -1.0),
               molecule=np.zeros(natom, np.int32), excl_ptr=np.zeros(natom + 1, np.int32),
               excl_idx=np.zeros(0, np.int32))
    kw = dict(method=abi.JP_METHOD_MICR)
    o = oracle.Oracle(top, **kw)
    eo, go = o.energy_grad()
    with eng_mod.Engine(top, precision=abi.JP_PREC_MIXED, **kw) as e:
        ene, g = e.energy_grad()
        assert e.pair_count() == o.npairs_cut
    assert rms_rel(g, go) < 1e-5
    np.testing.assert_allclose(ene, eo, rtol=1e-5, atol=1e-2)


@pytest.mark.parametrize("nwat", [700, 2900])
def test_replaced_coordinates_without_a_build(eng_mod, nwat):
    """Molecules put into other periodic images without a list build: the records' image flags no
    longer hold, and pairs take their own images as the FP64 path does."""
    top = systems.solvated_polymer(0, nwat, seed=23)
    x = top["cord"] + np.repeat(np.random.default_rng(1).integers(-1, 2, (nwat, 3)), 3, axis=0) * top["box"]
    out = []
    for prec in (abi.JP_PREC_MIXED, abi.JP_PREC_FP64):
        with eng_mod.Engine(top, precision=prec, method=abi.JP_METHOD_MICR) as e:
            out.append(e.energy_grad(cord=x))
    assert rms_rel(out[0][1], out[1][1]) < 1e-5
    np.testing.assert_allclose(out[0][0], out[1][0], rtol=1e-5, atol=1e-2)
