"""Probe resolve where its warps can go wrong: images that end inside a pixel
tile, warps whose pixels see several instances, the sky or instances without
probes, gathers that fall back to twice the radius in some lanes only, more
than 96 candidates. GPU against oracle bit for bit on at least 99.9 % of the
pixels (the bound of the resolve's other tests; all of fewer than 1000)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height", [(1, 1), (7, 5), (33, 9), (64, 48)])
@pytest.mark.parametrize("sites,min_gather", [(40, 24), (2000, 4), (12000, 32)])
def test_resolve_matches_oracle(device, width, height, sites, min_gather):
    import torch

    import nan_b200
    from nan_b200 import scenes
    from oracle.oracle import OracleScene

    node = scenes.terrain_boxes(seed=9, grid=33, boxes=60)
    scene = nan_b200.Scene(device, node)
    orc = OracleScene(**scene.host)
    probes, _ = scenes.surface_sites(node, sites, seed=5)
    # some instances without any probe; a wide kernel where candidates overflow
    inst = probes["meta"][:, 3] >> 8
    probes = probes[(inst % 7 != 3) | (inst == 0)]
    layout = nan_b200.SurfaceProbeSiteLayout.from_sites(node, probes,
                                                        kernel_radius_scale=8.0 if sites == 12000 else 2.5)
    geometry = nan_b200.SurfaceProbeGpuGeometry.create(device, layout)
    n = layout.total_probe_count
    rng = np.random.default_rng(sites + width)
    values = rng.uniform(0.0, 2.0, (n, 3)).astype(np.float32)
    counts = rng.integers(0, 40, n).astype(np.uint32)
    self_hits = rng.integers(0, 10, n).astype(np.uint32)
    mean = rng.uniform(0.1, 2.0, (n, 16)).astype(np.float32)
    moments = np.stack([mean, mean * mean + 0.1 * rng.random((n, 16), dtype=np.float32)], -1).astype(np.float16)
    radial = np.ascontiguousarray(moments).view(np.uint32).reshape(n, 16)
    rt = nan_b200.SurfaceProbeRuntimeBuffers.acquire(nan_b200.RenderData(device), n)
    for buf, host in ((rt.field.values, values), (rt.field.sample_counts, counts),
                      (rt.attachments.self_hit_counts, self_hits), (rt.attachments.radial_moments, radial)):
        buf.copy_(torch.from_numpy(np.ascontiguousarray(host).view(np.uint8).reshape(-1)).cuda())
    out = torch.zeros((height, width, 4), dtype=torch.float32, device="cuda")
    node.camera.begin_frame(width, height)
    nan_b200.SurfaceProbeResolve(device, scene, layout, geometry).execute(None, rt.field, rt.attachments, out,
                                                                          min_gather_count=min_gather)
    px = np.stack(np.meshgrid(np.arange(width), np.arange(height), indexing="xy"), -1).reshape(-1, 2)
    ref = orc.resolve_probes(scene.lighting, node.camera, width, height, px, layout, values, counts, self_hits, radial,
                             frame_index=scene.frame_index, min_gather_count=min_gather)
    exact = np.all(out.cpu().numpy().reshape(-1, 4) == ref, axis=1)
    assert (~exact).sum() <= exact.size // 1000, (~exact).sum()
    device.check()
