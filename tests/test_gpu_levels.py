"""Octree levels at the sizes where the ranking and listing of a build change
their route: one 2048-word region or many (res 50/51, 64, 100), the mesh's own
last CTA or a kernel of its own finishing the pyramid (res 512/513), keys
listed with the other levels or from the non-empty blocks (res 256/257),
level-0 regions tracked (res 513 and up), and octrees whose top lies below
level 3 of a big grid."""
import numpy as np
import pytest

from conftest import random_mesh
from parity import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("res", [1, 2, 50, 51, 64, 100, 128, 129, 256, 257, 512, 513, (300, 40, 7)])
def test_route_edges(gpu_ctx, oracle_mod, res):
    v, f = random_mesh(21, 12, "sliver")
    if res == 1:
        v = np.concatenate([v, v[:1] + 1])  # still a single voxel: undefined in the reference
        with pytest.raises(Exception):
            gpu_ctx.build(v, f, res)
        return
    assert_same(gpu_ctx.build(v, f, res), oracle_mod.build_svo(v, f, res))


def test_route_edges_in_one_batch(gpu_ctx, oracle_mod):
    """More than 8 regions per SM in one batch, meshes of every size in it."""
    meshes = [(*random_mesh(30 + i, 10, "sliver"), res) for i, res in enumerate((16, 512, 64, 257, 256, 300, 40, 1024))]
    results, st, rc = gpu_ctx.build_batch(meshes)
    assert rc == 0 and st == [0] * len(meshes)
    for (p, t, res), r in zip(meshes, results):
        assert_same(r, oracle_mod.build_svo(p, t, res))


def few_voxels(span, res):
    """One triangle over `span` voxels along x at the grid's origin corner; two
    vertices of no triangle pin the grid."""
    u = 1.0 / res
    tri = [[0.3 * u, 0.3 * u, 0.3 * u], [(span - 0.6) * u, 0.3 * u, 0.4 * u], [0.3 * u, 0.5 * u, 0.3 * u]]
    return np.array(tri + [[0, 0, 0], [1, 1, 1]], dtype=np.float32), np.array([[0, 1, 2]], dtype=np.int32)


@pytest.mark.parametrize("res", [16, 256, 300, 1024, 2048])
@pytest.mark.parametrize("span,depth", [(2, 2), (4, 3), (8, 4), (16, 5)])
def test_low_top(gpu_ctx, oracle_mod, res, span, depth):
    v, f = few_voxels(span, res)
    g = gpu_ctx.build(v, f, res)
    assert g.depth == depth
    assert_same(g, oracle_mod.build_svo(v, f, res))
