"""Scenes with a few vertices very far away (a backdrop, a marker): the boxes
that hold them are as large, and the slab test's products with a direction's
reciprocal must not cull the near triangles in such a box. Hits and any-hit
answers of rays along the axes and of others must equal the oracle's brute
force bit for bit (no tolerance: both run the same arithmetic on every
triangle)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("far,builder", [(far, builder) for far in (1e4, 1e12, 1e17, 1e19, 1e25, 1e30, 1e38)
                                         for builder in ("sah", "lbvh", "ploc")
                                         if builder != "ploc" or far < 1e19])  # PLOC refuses infinite areas
def test_hits_beside_far_vertices(device, far, builder):
    import torch

    import nan_b200
    from nan_b200.scene_node import Material, Mesh, SceneNode
    from oracle.oracle import OracleScene

    rng = np.random.default_rng(7)
    near = rng.uniform(-1.0, 1.0, size=(60, 1, 3)) + rng.uniform(-0.5, 0.5, size=(60, 3, 3))
    away = np.array([[1, 0, 0], [0, 1, 0], [0, 0, 1], [-1, 0, 0], [1, 1, 0], [0, -1, 0]], np.float64)
    small = away[:, None, :] * far + rng.uniform(-1.0, 1.0, size=(6, 3, 3)) * far * 1e-3
    v = np.zeros((3 * 66, 8), np.float32)
    v[:, :3] = np.concatenate([near, small]).reshape(-1, 3)
    node = SceneNode(name="far")
    mesh = node.add_mesh(Mesh(v, np.arange(3 * 66, dtype=np.uint32).reshape(-1, 3)))
    node.add_instance(mesh, node.add_material(Material(double_sided=True)),
                      node.add_transform(np.eye(4, dtype=np.float32)))
    scene = nan_b200.Scene(device, node, bvh_builder=builder)
    n = 3000
    rays = np.zeros((n, 8), np.float32)
    k = np.arange(n)
    axis, sign = k % 3, np.where(k % 2 == 0, 1.0, -1.0)
    rays[:, :3] = rng.uniform(-1.0, 1.0, size=(n, 3))
    rays[k, axis] = -3.0 * sign
    rays[k, 4 + axis] = sign
    tilted = rng.random(n) < 0.5
    rays[tilted, 4:7] += rng.normal(size=(int(tilted.sum()), 3)) * rng.choice([1e-21, 1e-12, 1e-3, 0.3],
                                                                             size=(int(tilted.sum()), 1))
    rays[:, 7] = 1000.0
    gpu = torch.from_numpy(rays).cuda()
    ids, tb = scene.intersect(gpu)
    want_ids, want_tb, _ = OracleScene(**scene.host).intersect(rays, mode=0)
    ids = ids.cpu().numpy().view(np.uint32)
    valid = want_ids[:, 0] == 1
    assert 0.5 < valid.mean() < 1.0
    np.testing.assert_array_equal(ids, want_ids)
    np.testing.assert_array_equal(tb.cpu().numpy()[valid], want_tb[valid])
    np.testing.assert_array_equal(scene.occluded(gpu).cpu().numpy(), 1.0 - valid.astype(np.float32))
    device.check()
