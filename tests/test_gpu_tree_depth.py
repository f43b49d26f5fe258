"""Binned-SAH trees near the traversal stack's limit of 96 levels and past it.
Triangles that shrink toward the origin along the six half axes are peeled off
one by one: each level's bins hold the outermost ones apart and all the rest in
the middle. A tree of 85 to 96 levels is built and its hits equal the oracle's
brute force bit for bit (no tolerance: the same arithmetic on every triangle);
a deeper one is refused by the build, and the context keeps no scene."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HALF_AXES = np.array([[1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [0, 0, 1], [0, 0, -1]], np.float64)


def shrinking(count: int, largest: float, coincident: int = 0):
    from nan_b200.scene_node import Material, Mesh, SceneNode

    rng = np.random.default_rng(1)
    p = np.array([largest * 0.7 ** i * (HALF_AXES[i % 6] + rng.uniform(-0.02, 0.02, size=(3, 3)))
                  for i in range(count)])
    tiny = np.repeat(np.array([[[0, 0, 0], [1e-38, 0, 0], [0, 1e-38, 0]]]), coincident, axis=0)
    p = np.concatenate([p, tiny]) if coincident else p
    v = np.zeros((3 * p.shape[0], 8), np.float32)
    v[:, :3] = p.reshape(-1, 3)
    node = SceneNode(name=f"shrinking_{count}")
    mesh = node.add_mesh(Mesh(v, np.arange(v.shape[0], dtype=np.uint32).reshape(-1, 3)))
    node.add_instance(mesh, node.add_material(Material(double_sided=True)),
                      node.add_transform(np.eye(4, dtype=np.float32)))
    return node, p


def test_a_tree_near_the_limit_is_walked(device):
    import torch

    import nan_b200
    from oracle.oracle import OracleScene

    count = 280
    node, p = shrinking(count, 1e10)
    scene = nan_b200.Scene(device, node)
    assert 85 <= scene.info()["max_depth"] <= 96
    rng = np.random.default_rng(2)
    n = 3000
    # from around the shells: toward a triangle of the same size or a few sizes larger
    k = rng.integers(0, count, n)
    b = rng.dirichlet([1, 1, 1], size=n)
    target = np.einsum("kj,kjc->kc", b, p[k])
    size = 1e10 * 0.7 ** np.minimum(k + rng.integers(0, 12, n), count - 1)
    rays = np.zeros((n, 8), np.float32)
    rays[:, :3] = rng.uniform(-1.0, 1.0, size=(n, 3)) * size[:, None]
    d = target - rays[:, :3]
    rays[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays[:, 7] = 1e30
    gpu = torch.from_numpy(rays).cuda()
    ids, tb = scene.intersect(gpu)
    want_ids, want_tb, _ = OracleScene(**scene.host).intersect(rays, mode=0)
    ids = ids.cpu().numpy().view(np.uint32)
    valid = want_ids[:, 0] == 1
    assert valid.mean() > 0.3
    np.testing.assert_array_equal(ids, want_ids)
    np.testing.assert_array_equal(tb.cpu().numpy()[valid], want_tb[valid])
    np.testing.assert_array_equal(scene.occluded(gpu).cpu().numpy(), 1.0 - valid.astype(np.float32))
    device.check()


def test_a_deeper_tree_is_refused(device):
    import nan_b200
    from nan_b200 import _native, scenes

    node, _ = shrinking(355, 1e18, coincident=64)
    with pytest.raises(_native.NanError, match="deeper than the traversal stack"):
        nan_b200.Scene(device, node)
    # the same on a context that held a scene: it holds none afterwards, and takes the next one
    scene = nan_b200.Scene(device, scenes.cornell_box(32, 32))
    deep = nan_b200.Scene(device, node, bvh_builder="lbvh")
    ctx, lib = scene.context, _native.lib()
    rc = lib.nan_scene_build(ctx.handle, ctypes.byref(deep._desc), _native.stream_handle(None))
    assert rc == _native.NAN_ERR_LIMIT
    info = _native.NanSceneInfo()
    assert lib.nan_scene_info(ctx.handle, ctypes.byref(info)) == _native.NAN_ERR_NO_SCENE
    _native.check(lib.nan_scene_build(ctx.handle, ctypes.byref(scene._desc), _native.stream_handle(None)))
    assert scene.info()["triangle_count"] == 36
    device.check()
