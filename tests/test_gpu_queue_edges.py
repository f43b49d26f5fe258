"""Wavefront queues at the sizes where they can go wrong: one path, a warp's
and a block's worth and one more or less, a queue that fills the traversal
grid's warps unevenly; paths that are closed a round after they end, restart
for further samples and turn to their back side. Every result must equal the
one-thread-per-unit kernels' bit for bit (no tolerance: the same arithmetic in
the same order)."""

import pytest

pytestmark = pytest.mark.gpu


def _forms(scene, run):
    results = []
    for integrator in ("megakernel", "wavefront"):
        scene.configure(integrator)
        scene.context.read_counters(reset=True)
        out = run()
        c = scene.context.read_counters(reset=True)
        results.append((out, (c["extend_rays"], c["shadow_rays"], c["units"], c["paths"])))
    scene.configure("wavefront")
    return results


@pytest.mark.parametrize("width,height", [(1, 1), (31, 1), (33, 1), (255, 1), (257, 1), (130, 131), (641, 480)])
@pytest.mark.parametrize("vertices", [1, 2, 5])
def test_screen_queue_sizes(device, width, height, vertices):
    import torch

    import nan_b200
    from nan_b200 import scenes

    node = scenes.reference_demo()
    scene = nan_b200.Scene(device, node)
    tracer = nan_b200.PathTracer(device, scene, max_vertices=vertices)
    node.camera.begin_frame(width, height)

    def run():
        out = torch.zeros((height, width, 4), dtype=torch.float32, device="cuda")
        tracer.execute(None, out, 11)
        return out

    (a, ca), (b, cb) = _forms(scene, run)
    torch.testing.assert_close(a, b, rtol=0, atol=0)
    assert ca == cb
    device.check()


@pytest.mark.parametrize("texels", [1, 32, 255, 256, 257, 1000])
@pytest.mark.parametrize("samples,bounces", [(1, 1), (1, 3), (3, 2)])
def test_texel_queue_sizes_with_back_sides(device, texels, samples, bounces):
    import torch

    import nan_b200
    from nan_b200 import scenes
    from nan_b200.mesh_colors import MeshColorsLayout

    node = scenes.reference_demo()  # its walls are double-sided
    scene = nan_b200.Scene(device, node)
    layout = MeshColorsLayout.build(node, texels_per_unit=12.0, min_resolution=2, max_resolution=16)
    tracer = nan_b200.TextureSpacePathTracer(device, scene, layout, samples_per_texel=samples, max_bounces=bounces)
    begin = layout.total_surface_texels // 3

    def run():
        slots = torch.zeros((layout.total_payload_count, 4), dtype=torch.int32, device="cuda")
        for it in range(2):
            tracer.execute(None, slots, it, reset=(it == 0), texel_range=(begin, begin + texels))
        return slots

    (a, ca), (b, cb) = _forms(scene, run)
    torch.testing.assert_close(a, b, rtol=0, atol=0)
    assert ca == cb
    device.check()


@pytest.mark.parametrize("sites", [1, 33, 256, 300])
@pytest.mark.parametrize("samples,bounces", [(1, 1), (5, 3)])
def test_probe_queue_sizes(device, sites, samples, bounces):
    import torch

    import nan_b200
    from nan_b200 import scenes

    node = scenes.reference_demo()
    scene = nan_b200.Scene(device, node)
    probes = nan_b200.SurfaceProbeSiteLayout.build(node, sites, seed=4)
    geometry = nan_b200.SurfaceProbeGpuGeometry.create(device, probes)
    baker = nan_b200.SurfaceProbeDiffuseIrradianceBaker(device, scene, geometry, samples_per_probe=samples,
                                                        max_bounces=bounces)

    def run():
        rt = nan_b200.SurfaceProbeRuntimeBuffers.acquire(nan_b200.RenderData(device), geometry.probe_count)
        for it in range(2):
            baker.execute(None, rt.field, rt.attachments, it, reset=(it == 0))
        return torch.cat([t.view(torch.int32) for t in (rt.field.values, rt.field.sample_counts,
                                                        rt.attachments.self_hit_counts,
                                                        rt.attachments.radial_moments)])

    (a, ca), (b, cb) = _forms(scene, run)
    torch.testing.assert_close(a, b, rtol=0, atol=0)
    assert ca == cb
    device.check()
