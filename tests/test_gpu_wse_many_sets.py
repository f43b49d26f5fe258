"""Sample elimination of many small sets in one call: enough candidates that a
few lanes share a candidate's lists in the first rounds and more in the last
ones, sets of other sizes side by side (the search for a candidate's cells ends
at its set), sets of one candidate among them. Each set must keep what it keeps
when it is eliminated alone (no tolerance: the weights are whole numbers)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("adaptive", [False, True])
@pytest.mark.parametrize("sizes", [(40,) * 1000, (1, 2, 17, 90, 333) * 100, (15000, 1, 14000, 3, 12000)])
def test_sets_together_equal_sets_alone(device, sizes, adaptive):
    import torch

    from nan_b200.surface_probe_sampler import SurfaceProbeSampler

    sampler = SurfaceProbeSampler(device)
    rng = np.random.default_rng(len(sizes))
    n = sum(sizes)
    offsets = np.concatenate([[0], np.cumsum(sizes)])
    p = np.zeros((n, 3), np.float32)
    for k, count in enumerate(sizes):
        side = np.sqrt(count / 90.0)
        p[offsets[k]:offsets[k + 1], ::2] = rng.uniform(0.0, side, size=(count, 2)) + rng.uniform(-3.0, 3.0, size=(1, 2))
    p[:, 1] = 0.05 * np.sin(3.0 * p[:, 0])
    normal = np.tile(np.array([[0.0, 1.0, 0.0]], np.float32), (n, 1))
    density = rng.uniform(0.5, 2.0, size=n).astype(np.float32)
    want = [max(1, c // 5) for c in sizes]
    area = [c / 90.0 for c in sizes]
    P, N, D = (torch.from_numpy(x).cuda() for x in (p, normal, density))

    def eliminate(first, last):
        a, b = int(offsets[first]), int(offsets[last])
        keep, radii = sampler.eliminate(P[a:b].contiguous(), N[a:b].contiguous(),
                                        [int(x) - a for x in offsets[first:last + 1]], want[first:last],
                                        area[first:last],
                                        relative_densities=D[a:b].contiguous() if adaptive else None)
        return np.asarray(keep.cpu() if hasattr(keep, "cpu") else keep), np.asarray(radii)

    keep, radii = eliminate(0, len(sizes))
    picks = rng.permutation(len(sizes))[:40]
    for k in sorted(picks):
        alone, r = eliminate(k, k + 1)
        np.testing.assert_array_equal(keep[offsets[k]:offsets[k + 1]], alone)
        assert radii[k] == r[0]
        assert int(np.count_nonzero(alone)) == want[k]
    device.check()
