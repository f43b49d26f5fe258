"""A multi-scene batch whose context has kernel timing on: the batch's launches
are not among those that the timing covers, so a captured frame holds no event
records, the times stay readable (and zero) after capture, replay and plain
frames, and the results do not change (no tolerance: the same launches)."""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("independent", [False, True])
def test_batch_with_kernel_timing(device, independent):
    import torch

    import nan_b200
    from nan_b200 import scenes

    items = []
    for i in range(2):
        node = scenes.terrain_boxes(seed=20 + i, grid=24, boxes=4)
        scene = nan_b200.Scene(device, node)
        sites = nan_b200.SurfaceProbeSiteLayout.build(node, 150 + 40 * i, seed=i)
        geometry = nan_b200.SurfaceProbeGpuGeometry.create(device, sites)
        baker = nan_b200.SurfaceProbeDiffuseIrradianceBaker(device, scene, geometry, samples_per_probe=4)
        rt = nan_b200.SurfaceProbeRuntimeBuffers.acquire(nan_b200.RenderData(device), geometry.probe_count)
        items.append((baker, rt.field, rt.attachments))
    batch = nan_b200.ProbeBatch(device, items, independent_samples=independent, wavefront=True)
    results = []
    for timing in (False, True):
        batch.context.configure(kernel_timing=timing)
        for it in range(2):
            batch.execute(None, it, 4, 3, reset=(it == 0))
        plain = [f.values.clone() for _, f, _ in items]
        batch.capture(0, True, 4, 3)
        batch.replay(2)
        torch.cuda.synchronize()
        results.append((plain, [f.values.clone() for _, f, _ in items]))
        times = batch.context.read_kernel_times(reset=True)
        assert all(v == 0 for v in times.values()), times
    for a, b in zip(results[0], results[1]):
        for x, y in zip(a, b):
            torch.testing.assert_close(x, y, rtol=0, atol=0)
    for x, y in zip(*results[0]):
        torch.testing.assert_close(x, y, rtol=0, atol=0)
    batch.close()
    device.check()
