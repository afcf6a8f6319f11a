"""The material sort at the edges of its bins and chunks: one material up to the
most that are sorted (4,095 and the misses' bin) and one more, waves below one
chunk of 2,048 paths, of a whole number of chunks and just beyond.  Only the
order of shading changes, so images equal the unsorted ones bit for bit.
"""
import dataclasses

import numpy as np
import pytest

from helpers import bits
from rendertoy_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_mats", [4, 36, 257, 4095, 4096])
@pytest.mark.parametrize("W, H, spp", [(7, 5, 1), (64, 32, 1), (64, 64, 2), (117, 71, 3)])
def test_sorted_equals_unsorted(ctx, n_mats, W, H, spp):
    import rendertoy_gb300 as rt
    sc = scenes.cornell_box()
    n = sc.n_tris
    mats = sc.mats[sc.mesh_mat[sc.tri_mesh]]  # one mesh and material per triangle, then unused ones
    if n_mats < n:
        mesh_mat = np.minimum(sc.mesh_mat[sc.tri_mesh], n_mats - 1)
        mats = sc.mats[:n_mats]
    else:
        mesh_mat = np.linspace(0, n_mats - 1, n).astype(np.int32)
        full = np.repeat(mats[:1], n_mats, axis=0)
        full[mesh_mat] = mats
        mats = full
    sc = dataclasses.replace(sc, tri_mesh=np.arange(n, dtype=np.int32), mesh_mat=mesh_mat.astype(np.int32),
                             mesh_smooth=np.zeros(n, np.uint8), mats=np.ascontiguousarray(mats))
    old = ctx.get_option(rt.OPT_SORT_MATERIAL)
    got = []
    try:
        ctx.upload(sc)
        for on in (0, 1):
            ctx.set_option(rt.OPT_SORT_MATERIAL, on)
            got.append(ctx.render_pt(W, H, spp, 5, seed=8))
    finally:
        ctx.set_option(rt.OPT_SORT_MATERIAL, old)
    assert np.array_equal(bits(got[0]), bits(got[1]))
