"""The 4-wide traversal at the smallest trees: a root that is itself a leaf (one
triangle up to a full leaf), the first trees with an inner node, and leaves of
one triangle and of eight; closest hits of camera rays and images (closest hits
and occlusion along paths) equal the binary tree's, bit for bit.
"""
import dataclasses

import numpy as np
import pytest

from rendertoy_gb300 import scenes

pytestmark = pytest.mark.gpu


def _few(n):
    """n triangles of the Cornell box: a wall's first, then the light's."""
    sc = scenes.cornell_box()
    light = np.any(sc.mats[sc.mesh_mat[sc.tri_mesh], 3:6] > 0, axis=1)
    walls = np.flatnonzero(~light)
    keep = np.concatenate([walls[:1], np.flatnonzero(light), walls[1:]])[:n]
    return dataclasses.replace(sc, verts=sc.verts[keep], norms=sc.norms[keep], tri_mesh=sc.tri_mesh[keep],
                               sky=np.full(3, 0.5, np.float32))


@pytest.mark.parametrize("leaf", [1, 4, 8])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 8, 9, 17])
def test_smallest_trees(ctx, n, leaf):
    import rendertoy_gb300 as rt
    old = ctx.get_option(rt.OPT_LEAF_SIZE), ctx.get_option(rt.OPT_TRAVERSAL)
    got = {}
    try:
        ctx.set_option(rt.OPT_LEAF_SIZE, leaf)
        ctx.upload(_few(n))
        for trav in (0, 2):
            ctx.set_option(rt.OPT_TRAVERSAL, trav)
            got[trav] = list(ctx.primary(33, 31)) + [ctx.render_pt(33, 31, 4, 5, seed=3)]
    finally:
        ctx.set_option(rt.OPT_LEAF_SIZE, old[0])
        ctx.set_option(rt.OPT_TRAVERSAL, old[1])
    for a, b in zip(got[0], got[2]):
        assert np.array_equal(np.ascontiguousarray(a).view(np.uint32), np.ascontiguousarray(b).view(np.uint32)), (n, leaf)
    assert got[2][-1].max() > 0
