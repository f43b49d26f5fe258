"""The binned-SAH builder around the sizes where its kernels hand over: a warp
up to 64 triangles, a block up to 1024, the whole GPU above; nodes whose
centroids coincide, and sets that peel off a few triangles a split. The tree
must be the CPU restatement's (same node count, cost to the 1e-9 of its
unordered sum) and its hits, binary and 8-wide, the oracle's bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _node(kind, n):
    from nan_b200.scene_node import Material, Mesh, SceneNode

    rng = np.random.default_rng(n)
    if kind == "soup":
        p = rng.uniform(-10.0, 10.0, size=(n, 1, 3)) + rng.normal(scale=0.6, size=(n, 3, 3))
    elif kind == "coincident":  # boxes [-s, s]: every centroid is the origin
        s = rng.uniform(0.5, 2.0, size=(n, 1, 3))
        p = np.concatenate([-s, s, rng.uniform(-1.0, 1.0, size=(n, 1, 3)) * s], axis=1)
    elif kind == "clusters":  # copies of 40 places, each below or above 64 triangles
        c = rng.uniform(-10.0, 10.0, size=(40, 3, 3))
        p = c[np.minimum(rng.geometric(0.08, size=n) - 1, 39)]
    else:  # "peeled": distances that grow by powers, a few triangles to a split
        r = 1.5 ** (np.arange(n) % 45)
        p = r[:, None, None] * (np.array([1.0, 0.3, 0.1]) + rng.uniform(-0.2, 0.2, size=(n, 3, 3)))
    v = np.zeros((3 * n, 8), np.float32)
    v[:, :3] = p.reshape(-1, 3)
    node = SceneNode(name=f"{kind}_{n}")
    mesh = node.add_mesh(Mesh(v, np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)))
    node.add_instance(mesh, node.add_material(Material(double_sided=True)),
                      node.add_transform(np.eye(4, dtype=np.float32)))
    return node


@pytest.mark.parametrize("kind,n", [("soup", 2), ("soup", 65), ("soup", 513), ("soup", 1023), ("soup", 1024),
                                    ("soup", 1025), ("soup", 2049), ("soup", 7001), ("coincident", 1024),
                                    ("coincident", 1025), ("coincident", 4099), ("clusters", 900),
                                    ("clusters", 6000), ("peeled", 1000), ("peeled", 5000)])
def test_tree_and_hits_match_the_restatement(device, kind, n):
    import torch

    import nan_b200
    from oracle.oracle import OracleScene, sah_build_stats

    scene = nan_b200.Scene(device, _node(kind, n), bvh_builder="sah")
    orc = OracleScene(**scene.host)
    world = orc.world_triangles()
    info, want = scene.info(), sah_build_stats(world)
    assert info["node_count"] == want["nodes"]
    assert abs(info["sah_cost"] - want["sah_cost"]) <= 1e-9 * want["sah_cost"]
    rng = np.random.default_rng(3)
    tri = world.reshape(-1, 3, 3).astype(np.float64)
    rays = np.zeros((3000, 8), np.float32)
    rays[:, :3] = rng.uniform(tri.min((0, 1)), tri.max((0, 1)), size=(3000, 3))
    d = np.einsum("kj,kjc->kc", rng.dirichlet([1, 1, 1], size=3000), tri[rng.integers(0, n, 3000)]) - rays[:, :3]
    rays[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays[:, 7] = 1e30
    o_ids, o_tb, _ = orc.intersect(rays, mode=0)
    for width in (2, 8):
        scene.configure(bvh_width=width)
        ids, tb = scene.intersect(torch.from_numpy(rays).cuda())
        ids = ids.cpu().numpy().view(np.uint32)
        np.testing.assert_array_equal(ids, o_ids)
        valid = ids[:, 0] == 1
        np.testing.assert_array_equal(tb.cpu().numpy()[valid], o_tb[valid])
    scene.configure()
    device.check()
