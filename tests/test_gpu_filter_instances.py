"""Surface filter over instances of a few texels, where a warp's 32 texels lie
in many instances, with runs of instances without any texel between them (31,
32, 33 and more: a search among the next 32 instances would miss the rest).
GPU against oracle; the bound is the 1e-5 relative of the filter's other tests,
counts are equal."""

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gap", [0, 1, 30, 31, 32, 33, 200])
@pytest.mark.parametrize("run", [1, 9, 40])
def test_filter_with_empty_instances(device, gap, run):
    import torch

    import nan_b200
    from nan_b200.mesh_colors import MeshColorsLayout, layout_adjacency, layout_face_normals
    from nan_b200.scene_node import Material, Mesh, SceneNode, make_transform
    from oracle.oracle import filter_mesh_colors

    node = SceneNode(name="gaps")
    v = np.zeros((3, 8), np.float32)
    v[1, 0] = v[2, 2] = 1.0
    one = node.add_mesh(Mesh(v, np.array([[0, 1, 2]], np.uint32)))
    none = node.add_mesh(Mesh(v.copy(), np.zeros((0, 3), np.uint32)))
    material = node.add_material(Material())
    count = 0
    for part in range(4):
        for mesh, times in ((one, run), (none, gap)):
            for _ in range(times):
                node.add_instance(mesh, material, node.add_transform(make_transform((0.0, float(count), 0.0))))
                count += 1
    node.add_instance(one, material, node.add_transform(make_transform((0.0, float(count), 0.0))))
    layout = MeshColorsLayout.build(node, texels_per_unit=1.0, min_resolution=1, max_resolution=1)
    assert layout.total_surface_texels == 3 * (4 * run + 1)
    rng = np.random.default_rng(gap + run)
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
