"""Kernel timing on: a round's closest-hit and shadow rays then run as a launch
each, of kernels that nothing else launches (but for the forms that refill
lanes, 1 to 4). Pixels, texel slots, probe fields and the ray counts of every
form, with timing and without, equal the default's bit for bit (no tolerance:
the same arithmetic in the same order), at sizes from one path to a queue that
fills the grid's warps unevenly, and the times say that both kinds of launches
ran."""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("builder,option", [("sah", {}), ("lbvh", {}), ("sah", {"traversal": 2}),
                                            ("lbvh", {"traversal": 5}), ("sah", {"traversal": 6}),
                                            ("sah", {"bvh_width": 8})])
@pytest.mark.parametrize("width,height,sites", [(1, 1, 1), (33, 1, 33), (130, 131, 300), (641, 480, 3000)])
def test_timing_does_not_change_results(device, width, height, sites, builder, option):
    import torch

    import nan_b200
    from nan_b200 import scenes
    from nan_b200.mesh_colors import MeshColorsLayout

    node = scenes.terrain_boxes(seed=5, grid=41, boxes=30)
    scene = nan_b200.Scene(device, node, bvh_builder=builder)
    layout = MeshColorsLayout.build(node, texels_per_unit=6.0, min_resolution=2, max_resolution=16)
    probes = nan_b200.SurfaceProbeSiteLayout.build(node, sites, seed=2)
    geometry = nan_b200.SurfaceProbeGpuGeometry.create(device, probes)
    begin = layout.total_surface_texels // 4
    texels = (begin, min(layout.total_surface_texels, begin + width * height))
    node.camera.begin_frame(width, height)  # one jitter for both
    results = []
    for form, timing in (({}, False), (option, False), (option, True)):
        scene.configure(kernel_timing=timing, **form)
        scene.context.read_kernel_times(reset=True)
        scene.context.read_counters(reset=True)
        out = torch.zeros((height, width, 4), dtype=torch.float32, device="cuda")
        nan_b200.PathTracer(device, scene, max_vertices=3).execute(None, out, 5)
        slots = torch.zeros((layout.total_payload_count, 4), dtype=torch.int32, device="cuda")
        tracer = nan_b200.TextureSpacePathTracer(device, scene, layout, samples_per_texel=2, max_bounces=2)
        for it in range(2):
            tracer.execute(None, slots, it, reset=(it == 0), texel_range=texels)
        rt = nan_b200.SurfaceProbeRuntimeBuffers.acquire(nan_b200.RenderData(device), geometry.probe_count)
        baker = nan_b200.SurfaceProbeDiffuseIrradianceBaker(device, scene, geometry, samples_per_probe=3, max_bounces=2)
        for it in range(2):
            baker.execute(None, rt.field, rt.attachments, it, reset=(it == 0))
        c = scene.context.read_counters(reset=True)
        times = scene.context.read_kernel_times(reset=True)
        if timing:
            assert times["extend_launches"] > 0 and times["extend_ms"] > 0.0
            assert times["shadow_launches"] > 0 and times["shadow_ms"] > 0.0
            assert times["stage_launches"] > 0 and times["stage_ms"] > 0.0
        else:
            assert all(v == 0 for v in times.values())
        results.append(([out, slots, rt.field.values.clone(), rt.attachments.radial_moments.clone()],
                        (c["extend_rays"], c["shadow_rays"], c["units"], c["paths"])))
    scene.configure()
    a, ca = results[0]
    for b, cb in results[1:]:
        for x, y in zip(a, b):
            torch.testing.assert_close(x.view(torch.int32), y.view(torch.int32), rtol=0, atol=0)
        assert ca == cb and ca[0] > 0
    device.check()
