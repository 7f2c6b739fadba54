"""The 4-atom SHAKE solve on both sides of its pivot rule: a methyl-like group takes the natural
order, a group whose first bond is far shorter than the others needs the pivot search (an
entry of its Newton matrix is more than 16 times the first pivot).  FP64 CANO steps against
the oracle, which always pivots: the suite's trajectory tolerance, 1e-8 A; both forms of the
integrator.
"""
import numpy as np
import pytest

import oracle
from j_presto_b200 import abi, systems

pytestmark = pytest.mark.gpu
PAIRS = [(0, 1), (1, 2), (2, 0), (3, 0), (2, 3), (1, 3)]
METHYL = 1.09 / np.sqrt(3.0) * np.array([[0, 0, 0], [1, 1, 1], [1, -1, -1], [-1, 1, -1]], float)
UNEVEN = np.array([[0, 0, 0], [0.04, 0, 0], [1.5, 0.9, 0.3], [0.4, -1.2, 1.1]], float)


@pytest.fixture(scope="module")
def eng_mod(engine_lib):
    from j_presto_b200 import engine
    return engine


def first_ratio(x, im):
    """largest entry below the first pivot of the gradient matrix, in units of the pivot"""
    d = np.array([x[a] - x[b] for a, b in PAIRS])
    inc = np.zeros((4, 6))
    for q, (a, b) in enumerate(PAIRS):
        inc[a, q], inc[b, q] = 1.0, -1.0
    A = 2.0 * (inc.T @ np.diag(im) @ inc) * (d @ d.T)
    return np.abs(A[1:, 0]).max() / abs(A[0, 0])


@pytest.mark.parametrize("grid", [0, 1])
@pytest.mark.parametrize("geom,pivots", [(METHYL, False), (UNEVEN, True)])
def test_four_atom_group_vs_oracle(eng_mod, geom, pivots, grid):
    mass = np.array([12.011, 1.008, 1.008, 1.008])
    assert (first_ratio(geom, 1.0 / mass) > 16.0) == pivots
    rng = np.random.default_rng(2)
    n = 4                                   # groups, between the ions of a 6 A lattice
    ions = np.stack(np.meshgrid(*[6.0 * np.arange(5)] * 3, indexing="ij"), -1).reshape(-1, 3) + 4.0
    at = ions[rng.choice(len(ions) - 40, n, replace=False)] + 3.0
    x = np.concatenate([geom + c for c in at] + [ions])
    na = len(x)
    typ = np.concatenate([np.full(4 * n, systems.T_HW), np.where(np.arange(len(ions)) % 2, systems.T_NA, systems.T_CL)])
    m = np.concatenate([np.tile(mass, n), np.full(len(ions), 30.0)])
    v = rng.normal(size=x.shape) * np.sqrt(8.31451e-7 * 300.0 / m)[:, None]
    v[:4 * n] *= 0.02                       # the short bond stays short in a step
    base = systems.solvated_polymer(0, 1, nion_pairs=1, seed=3)
    ex = [[4 * (i // 4) + k for k in range(4) if 4 * (i // 4) + k != i] if i < 4 * n else [] for i in range(na)]
    top = dict(base, **{k: val[:0] for k, val in base.items() if isinstance(val, np.ndarray)
                        and k.split("_")[0] in ("bond", "angle", "tors", "impr")})
    top.update(natom=na, box=np.full(3, 40.0), cord=x, vel=v, mass=m, atype=typ.astype(np.int32),
               charge=np.concatenate([np.zeros(4 * n), np.where(np.arange(len(ions)) % 2, 0.2, -0.2)]),
               molecule=np.zeros(na, np.int32), shake_n=np.full(n, 4),
               excl_ptr=np.concatenate([[0], np.cumsum([len(e) for e in ex])]).astype(np.int32),
               excl_idx=np.array([j for e in ex for j in e], np.int32),
               shake_atoms=np.arange(4 * n).reshape(n, 4),
               shake_dist=np.tile([np.linalg.norm(geom[a] - geom[b]) for a, b in PAIRS], (n, 1)))
    kw = dict(method=abi.JP_METHOD_CANO, tempco=1, dt=1.0)
    o = oracle.Oracle(top, **kw)
    ier, eo, _ = o.run(8)
    assert ier == 0
    with eng_mod.Engine(top, precision=abi.JP_PREC_FP64, **kw) as e:
        if grid:
            e.set_grid_limit(grid)
        e.step(8)
        xe, _ = e.get_state()
    np.testing.assert_allclose(xe, o.get_state()[0], rtol=0, atol=1e-8)
