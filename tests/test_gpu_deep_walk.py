"""Binary walks on deep trees: the traversal stack holds one entry per
interior node above the walk, so trees whose depth comes near the limit of 96
exercise its upper entries. Triangles that halve in size and distance from one
to the next make a binned-SAH tree that peels off a few of them per level.
Hits and any-hit answers must equal the oracle's bit for bit (no tolerance:
both run the same arithmetic)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("builder", ["sah", "lbvh"])
@pytest.mark.parametrize("count", [2, 33, 90, 119])
def test_walks_on_deep_trees_match_the_oracle(device, count, builder):
    import torch

    import nan_b200
    from nan_b200.scene_node import Material, Mesh, SceneNode
    from oracle.oracle import OracleScene

    rng = np.random.default_rng(count)
    scale = (2.0 ** -np.arange(count))[:, None, None]
    p = (scale * (np.array([[1.0, 0.0, 0.0]]) + rng.uniform(-0.2, 0.2, size=(count, 3, 3)))).reshape(-1, 3)
    v = np.zeros((3 * count, 8), np.float32)
    v[:, :3] = p * 1000.0
    node = SceneNode(name=f"halving_{count}")
    mesh = node.add_mesh(Mesh(v, np.arange(3 * count, dtype=np.uint32).reshape(-1, 3)))
    node.add_instance(mesh, node.add_material(Material(double_sided=True)),
                      node.add_transform(np.eye(4, dtype=np.float32)))
    try:
        scene = nan_b200.Scene(device, node, bvh_builder=builder)
    except nan_b200._native.NanError as e:
        assert "deeper than the traversal stack" in str(e)  # rejected, never walked
        return
    orc = OracleScene(**scene.host)
    world = orc.world_triangles().reshape(-1, 3, 3).astype(np.float64)
    n = 2000
    rays = np.zeros((n, 8), np.float32)
    rays[:, :3] = rng.uniform(-1.0, 1.0, size=(n, 3)) * 1000.0 * 2.0 ** -rng.integers(0, min(count, 40), size=(n, 1))
    b = rng.dirichlet([1, 1, 1], size=n)
    d = np.einsum("kj,kjc->kc", b, world[rng.integers(0, count, n)]) - rays[:, :3]
    rays[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays[:, 7] = 1e30
    gpu = torch.from_numpy(rays).cuda()
    ids, tb = scene.intersect(gpu)
    o_ids, o_tb, _ = orc.intersect(rays, mode=0)
    ids = ids.cpu().numpy().view(np.uint32)
    np.testing.assert_array_equal(ids, o_ids)
    valid = ids[:, 0] == 1
    np.testing.assert_array_equal(tb.cpu().numpy()[valid], o_tb[valid])
    np.testing.assert_array_equal(scene.occluded(gpu).cpu().numpy(), 1.0 - valid.astype(np.float32))
    device.check()
