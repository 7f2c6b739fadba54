"""The list build's per-tile image rule (j_presto_b200/csrc/jp_cells.cu, k_block_list): with c the
minimum image of two block references' separation and h the blocks' half extents, a tile whose
L - (|c| + h_i + h_j) exceeds a radius on every axis holds no pair that is within that radius
in another image than the tile's.  Checked on random orthorhombic boxes, block shapes and
positions for the list radius, and for the cut-off with atoms moved after the build by up to
the rule's margin (2 A between the two atoms).
"""
import numpy as np
import pytest

RC, RLIM = 12.0, 13.5


@pytest.mark.parametrize("seed", range(8))
def test_unflagged_tiles_need_no_pair_images(seed):
    rng = np.random.default_rng(seed)
    flagged = pairs = 0
    for _ in range(400):
        box = rng.uniform(27.0, 60.0, 3)
        h = rng.uniform(1.0, 7.0, (2, 3))
        ref = rng.uniform(0.0, 1.0, (2, 3)) * box
        d = ref[0] - ref[1]
        shift = box * np.round(d / box)
        other = box - (np.abs(shift - d) + h.sum(0))
        xi = ref[0] + rng.uniform(-1.0, 1.0, (32, 3)) * h[0]
        xj = ref[1] + rng.uniform(-1.0, 1.0, (32, 3)) * h[1]
        if (other > RLIM + 0.01).all():
            tile = xi[:, None] - xj[None] - shift
            best = tile - box * np.round(tile / box)
            near = (best ** 2).sum(-1) <= RLIM ** 2
            np.testing.assert_allclose(tile[near], best[near], atol=1e-9)
            pairs += int(near.sum())
        else:
            flagged += 1
        if (other > RC + 2.0).all():
            u = rng.normal(size=(2, 32, 3))
            u /= np.linalg.norm(u, axis=-1, keepdims=True)
            tile = (xi + u[0])[:, None] - (xj + u[1])[None] - shift
            best = tile - box * np.round(tile / box)
            near = (best ** 2).sum(-1) <= RC ** 2
            np.testing.assert_allclose(tile[near], best[near], atol=1e-9)
    assert flagged and pairs    # both sides of the rule were met
