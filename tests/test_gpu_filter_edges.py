"""Surface filter at the sizes where its warps can go wrong: faces of three
texels (ten faces to a warp), instances smaller than a warp, texel counts
around a warp's 32 and its 128, double-sided instances beside one-sided ones.
GPU against oracle; the bound is the 1e-5 relative of the filter's other tests
(acos and exp come from different libraries), counts are equal."""

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _strip(instances, triangles, seed):
    from nan_b200.scene_node import Material, Mesh, SceneNode, make_transform

    rng = np.random.default_rng(seed)
    n = triangles + 2
    v = np.zeros((n, 8), np.float32)
    v[:, 0] = np.arange(n) // 2
    v[:, 1] = rng.uniform(-0.3, 0.3, n)
    v[:, 2] = np.arange(n) % 2
    i = np.arange(triangles)
    tri = np.where((i % 2 == 0)[:, None], np.stack([i, i + 1, i + 2], 1), np.stack([i + 1, i, i + 2], 1))
    node = SceneNode(name="strip")
    mesh = node.add_mesh(Mesh(v, tri.astype(np.uint32)))
    mats = [node.add_material(Material(double_sided=d)) for d in (False, True)]
    for k in range(instances):
        node.add_instance(mesh, mats[(k // 3) % 2], node.add_transform(make_transform((0.0, float(k), 0.0))))
    return node


@pytest.mark.parametrize("instances,triangles,resolution", [(1, 1, 1), (1, 2, 1), (1, 11, 1), (1, 43, 1), (5, 2, 1),
                                                            (40, 1, 2), (7, 5, 4), (3, 2, 64), (130, 3, 1),
                                                            (120, 23, 16), (180, 31, 16)])
def test_filter_matches_oracle(device, instances, triangles, resolution):
    import torch

    import nan_b200
    from nan_b200.mesh_colors import MeshColorsLayout, layout_adjacency, layout_face_normals
    from oracle.oracle import filter_mesh_colors

    node = _strip(instances, triangles, seed=instances + triangles)
    layout = MeshColorsLayout.build(node, texels_per_unit=1.0, min_resolution=resolution, max_resolution=resolution,
                                    max_total_texels=4_000_000)
    rng = np.random.default_rng(3)
    data = np.zeros((layout.total_payload_count, 4), np.float32)
    data[:, :3] = rng.uniform(0.0, 2.0, (data.shape[0], 3))
    data.view(np.uint32)[:, 3] = rng.integers(1, 100, data.shape[0])
    src = torch.from_numpy(data.view(np.int32)).cuda()
    dst = torch.zeros_like(src)
    scene = nan_b200.Scene(device, node)
    nan_b200.MeshColorsSurfaceFilter(device, scene, layout).execute(None, src, dst)
    ref = filter_mesh_colors(layout.face_array, layout.instance_array, layout.side_array, layout_adjacency(node),
                             layout_face_normals(node), data.view(np.uint32).copy(), math.exp(-0.5), math.radians(30.0))
    got = dst.cpu().numpy()
    np.testing.assert_allclose(got.view(np.float32)[:, :3], np.asarray(ref).view(np.float32)[:, :3], rtol=1e-5,
                               atol=1e-7)
    np.testing.assert_array_equal(got.view(np.uint32)[:, 3], np.asarray(ref).view(np.uint32)[:, 3])
    device.check()
