"""The visibility caster's ray order at its edges: ray counts around a warp's
32, a sum's 64 and the largest table, and tables of the caller's own whose
directions all lie in one cell, repeat, or have no direction at all. Masks and
SH sums must be bit-identical to the oracle's, or for the caller's tables to
the library's any-hit query and a sum in the caster's order."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(device, count):
    import nan_b200
    from nan_b200 import scenes

    node = scenes.terrain_boxes(seed=7, grid=33, boxes=20)
    probes, _ = scenes.surface_sites(node, count, seed=3, double_sided_backs=False)
    return (nan_b200.Scene(device, node), np.ascontiguousarray(probes["position_radius"][:, :3]),
            np.ascontiguousarray(probes["normal_side"][:, :3]))


@pytest.mark.parametrize("rays", [1, 31, 32, 33, 64, 65, 127, 1023, 1024])
def test_ray_counts_match_the_oracle(device, oracle_mod, rays):
    import nan_b200
    from oracle import visibility as ov

    scene, sites, normals = _scene(device, 67)
    normals[3] = 0.0
    sh, counts = nan_b200.trace_pmr_visibility_sh(scene, sites, normals, ray_count=rays, max_distance=1000.0,
                                                  self_bias=1e-3)
    expect, expect_counts = ov.visibility_sh16(oracle_mod.OracleScene(**scene.host), sites, normals, rays, 1000.0, 1e-3)
    np.testing.assert_array_equal(counts.cpu().numpy(), expect_counts)
    np.testing.assert_array_equal(sh.cpu().numpy().view(np.uint32), expect.view(np.uint32))
    device.check()


@pytest.mark.parametrize("kind,rays", [("one cell", 1024), ("repeated", 200), ("random", 70), ("no direction", 40)])
def test_tables_of_the_callers_own(device, kind, rays):
    import torch

    import nan_b200

    scene, sites, normals = _scene(device, 20)
    sites = (sites + np.float32(0.05) * normals).astype(np.float32)
    rng = np.random.default_rng(rays)
    d = rng.normal(size=(rays, 3))
    if kind == "one cell":
        d = np.array([0.3, 0.9, 0.2]) + 1e-4 * d
    elif kind == "repeated":
        d = d[rng.integers(0, 3, rays)]
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    if kind == "no direction":
        d[::3] = 0.0
    table = np.zeros((rays, 20), np.float32)
    table[:, :3] = d
    table[:, 4:] = rng.normal(size=(rays, 16))
    sh, counts = nan_b200.trace_pmr_visibility_sh(scene, sites, normals, ray_count=rays, max_distance=50.0,
                                                  self_bias=0.0, table=torch.from_numpy(table).cuda())
    q = np.zeros((sites.shape[0], rays, 8), np.float32)
    q[:, :, :3] = sites[:, None]
    q[:, :, 4:7] = table[None, :, :3]
    q[:, :, 7] = 50.0
    seen = scene.occluded(torch.from_numpy(q.reshape(-1, 8)).cuda()).cpu().numpy().reshape(-1, rays) != 0.0
    np.testing.assert_array_equal(counts.cpu().numpy(), seen.sum(1))
    want = np.zeros((sites.shape[0], 16), np.float32)
    for i in range(sites.shape[0]):
        for b in range(0, rays, 64):
            batch = np.zeros(16, np.float32)
            for r in range(b, min(b + 64, rays)):
                if seen[i, r]:
                    batch = batch + table[r, 4:]
            want[i] = want[i] + batch
    np.testing.assert_array_equal(sh.cpu().numpy().view(np.uint32), want.view(np.uint32))
    device.check()
