"""Binary walks at the last entry of the traversal stack and past it. The nodes
of nan_scene_build_noalloc lie in the caller's buffers, so a chain of any depth
can be written there: every node's boxes hold the whole scene, its first child
is the next node and its second a leaf, and a walk therefore stacks one entry a
node before it comes to the first triangle. Up to 96 entries the hits equal the
oracle's brute force bit for bit; from the 97th on the walk stays inside its
stack and the context reports the overflow. The tables of links and leaves are
checked on the host before a ray is walked."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STACK = 96
NODE = 16  # words of a node: 12 of boxes, the two children, two unused


def chain_nodes(length: int, triangles: int) -> np.ndarray:
    """`length` nodes that stack `length` leaves, then test them all; the
    triangles left over hang below the last node, eight to a leaf at most."""
    nodes = np.zeros((triangles - 1, NODE), np.float32)
    # (c0.c.x, c1.c.x, c0.c.y, c1.c.y), (c0.c.z, c1.c.z, c0.h.x, c1.h.x), (c0.h.y, c1.h.y, c0.h.z, c1.h.z)
    nodes[:, 6:12] = 1e6
    child = nodes[:, 12:14].view(np.int32)
    for i in range(length):
        child[i, 1] = ~(i << 3)
        child[i, 0] = i + 1
    rest = triangles - length
    assert 1 <= rest <= 8
    child[length - 1, 0] = ~((length << 3) | (rest - 1))
    return nodes


def check_chain(nodes: np.ndarray, length: int, triangles: int) -> None:
    """Every link of the chain goes to a later node of it, every leaf holds
    triangles that exist, and each triangle is in one leaf."""
    child = nodes[:, 12:14].view(np.int32)
    seen = []
    for i in range(length):
        for c in child[i]:
            if c >= 0:
                assert i < c < length
            else:
                first, count = (~c) >> 3, ((~c) & 7) + 1
                assert first + count <= triangles
                seen.extend(range(first, first + count))
    assert sorted(seen) == list(range(triangles))


@pytest.mark.parametrize("length", [1, 2, STACK - 1, STACK, STACK + 1, STACK + 2, 3 * STACK])
def test_a_chain_fills_the_stack(device, length):
    import torch

    import nan_b200
    from nan_b200 import _native
    from nan_b200.scene_node import Material, Mesh, SceneNode
    from oracle.oracle import OracleScene

    triangles = length + 3
    rng = np.random.default_rng(length)
    p = rng.uniform(-1.0, 1.0, size=(triangles, 1, 3)) + rng.uniform(-0.4, 0.4, size=(triangles, 3, 3))
    v = np.zeros((3 * triangles, 8), np.float32)
    v[:, :3] = p.reshape(-1, 3)
    node = SceneNode(name=f"chain_{length}")
    mesh = node.add_mesh(Mesh(v, np.arange(3 * triangles, dtype=np.uint32).reshape(-1, 3)))
    node.add_instance(mesh, node.add_material(Material(double_sided=True)),
                      node.add_transform(np.eye(4, dtype=np.float32)))
    scene = nan_b200.Scene(device, node)
    ctx = device.new_context()
    dev = device.torch_device
    nodes = torch.empty((triangles - 1, NODE), dtype=torch.float32, device=dev)
    tris = torch.empty((triangles * 12,), dtype=torch.float32, device=dev)
    refs = torch.empty((triangles * 2,), dtype=torch.int32, device=dev)
    stream = _native.stream_handle(None)
    lib = _native.lib()
    _native.check(lib.nan_scene_build_noalloc(ctx.handle, ctypes.byref(scene._desc), nodes.data_ptr(),
                                              nodes.numel() * 4, tris.data_ptr(), tris.numel() * 4, refs.data_ptr(),
                                              refs.numel() * 4, stream))
    host = chain_nodes(length, triangles)
    check_chain(host, length, triangles)
    nodes.copy_(torch.from_numpy(host))

    n = 512
    rays = np.zeros((n, 8), np.float32)
    rays[:, :3] = rng.uniform(-2.0, 2.0, size=(n, 3))
    d = rng.uniform(-1.0, 1.0, size=(n, 3)) - rays[:, :3]
    rays[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays[:, 7] = 1e30
    gpu = torch.from_numpy(rays).to(dev)
    ids = torch.empty((n, 4), dtype=torch.int32, device=dev)
    tb = torch.empty((n, 3), dtype=torch.float32, device=dev)
    vis = torch.empty((n,), dtype=torch.float32, device=dev)
    for call in ("closest", "any"):
        if call == "closest":
            _native.check(lib.nan_intersect(ctx.handle, gpu.data_ptr(), n, ids.data_ptr(), tb.data_ptr(), stream))
        else:
            _native.check(lib.nan_occluded(ctx.handle, gpu.data_ptr(), n, vis.data_ptr(), stream))
        if length > STACK:
            with pytest.raises(_native.NanError, match="traversal stack overflowed"):
                ctx.check()
        else:
            ctx.check()
    ctx.check()  # the report was taken; nothing else is left behind
    if length <= STACK:
        want_ids, want_tb, _ = OracleScene(**scene.host).intersect(rays, mode=0)
        got = ids.cpu().numpy().view(np.uint32)
        np.testing.assert_array_equal(got, want_ids)
        valid = got[:, 0] == 1
        assert 0 < valid.sum() < n
        np.testing.assert_array_equal(tb.cpu().numpy()[valid], want_tb[valid])
        np.testing.assert_array_equal(vis.cpu().numpy(), 1.0 - valid.astype(np.float32))
    ctx.close()
