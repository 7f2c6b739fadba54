"""A 4-atom SHAKE group's Newton systems are solved the same way whichever groups share its
warp: a replica of methyl-like groups beside one of groups that need the pivot search, and
beside one of its own kind, steps bit for bit alike (mixed path, whose sums are integers).
Two groups a replica, so that a warp's four are half of each; both forms of the integrator.  A
loose SHAKE tolerance ends the iteration before its later steps take the first one's rounding
back; the two solutions then differ by some 1e-16 of a correction of 1e-3 to 1e-2 A, which moves a
last bit of one coordinate in some thousands: 64 groups over 200 steps show it.
"""
import numpy as np
import pytest

from j_presto_b200 import abi, systems
from tests.test_gpu_quad_pivot import METHYL, PAIRS, UNEVEN

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng_mod(engine_lib):
    from j_presto_b200 import engine
    return engine


def replica(geom, seed, n=2):
    """n groups between the ions of a 6 A lattice"""
    mass = np.array([12.011, 1.008, 1.008, 1.008])
    rng = np.random.default_rng(seed)
    ions = np.stack(np.meshgrid(*[6.0 * np.arange(5)] * 3, indexing="ij"), -1).reshape(-1, 3) + 4.0
    at = ions[rng.choice(len(ions) - 40, n, replace=False)] + 3.0
    x = np.concatenate([geom + c for c in at] + [ions])
    na = len(x)
    typ = np.concatenate([np.full(4 * n, systems.T_HW), np.where(np.arange(len(ions)) % 2, systems.T_NA, systems.T_CL)])
    m = np.concatenate([np.tile(mass, n), np.full(len(ions), 30.0)])
    v = rng.normal(size=x.shape) * np.sqrt(8.31451e-7 * 300.0 / m)[:, None]
    if geom is UNEVEN:
        v[:4 * n] *= 0.02                   # the short bond stays short in a step
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
    return top


@pytest.mark.parametrize("grid", [0, 1])
def test_neighbours_do_not_change_a_group(eng_mod, grid):
    out = []
    for other in (METHYL, UNEVEN):
        with eng_mod.Engine([replica(METHYL if r % 2 == 0 else other, r) for r in range(64)], precision=abi.JP_PREC_MIXED,
                            method=abi.JP_METHOD_CANO, tempco=1, dt=2.0, shake_tol=1e-3) as e:
            if grid:
                e.set_grid_limit(grid)
            e.step(200)
            out.append(np.array([e.get_state(r) for r in range(0, 64, 2)]))
    np.testing.assert_array_equal(out[0], out[1])
