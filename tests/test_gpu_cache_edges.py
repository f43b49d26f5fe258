"""The learned cache at the edges of its tiles and its table.

Counts around the 128-query tile and the pairs of tiles a block takes; tables
so small that every level wraps, where the corners of a cell along x are
neighbours for even cells only; and lazy steps that touch few entries, single
ones among them, or nearly all. Bounds as in test_gpu_cache.py.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cache(device, log2_table, base, n, table_update="dense"):
    import torch

    import nan_b200
    from oracle import lrc

    cfg = lrc.CacheConfig(log2_table=log2_table, base_resolution=base, max_resolution=8 * base,
                          bounds_min=(-2.0, -1.0, -3.0), bounds_max=(2.0, 3.0, 1.0))
    cache = nan_b200.RadianceCache(device, cfg.bounds_min, cfg.bounds_max, log2_table=log2_table,
                                   base_resolution=base, max_resolution=cfg.max_resolution, table_update=table_update)
    rng = np.random.default_rng(n)
    params, _ = lrc.init_params(cfg, seed=n)
    table = rng.uniform(-0.5, 0.5, lrc.LEVELS * cfg.table_size * 2).astype(np.float32)
    cache.set_params(torch.from_numpy(params).cuda(), torch.from_numpy(table).cuda())
    q = np.zeros((n, 8), np.float32)
    q[:, 0:3] = rng.uniform(np.array(cfg.bounds_min) - 0.2, np.array(cfg.bounds_max) + 0.2, (n, 3))
    nrm = rng.normal(size=(n, 3))
    q[:, 4:7] = nrm / np.linalg.norm(nrm, axis=1, keepdims=True)
    y = np.zeros((n, 4), np.float32)
    y[:, :3] = rng.uniform(0.0, 3.0, (n, 3))
    return cfg, cache, params, table, table.astype(np.float16), q, y


@pytest.mark.parametrize("log2_table,base,n", [(10, 4, 1), (10, 9, 127), (10, 64, 129), (12, 7, 257), (14, 16, 385)])
def test_forward_and_gradients_match_oracle(device, log2_table, base, n):
    import torch

    from oracle import lrc

    cfg, cache, params, _, table16, q, y = _cache(device, log2_table, base, n)
    out = cache.infer(torch.from_numpy(q).cuda()).cpu().numpy()[:, :3].astype(np.float64)
    ref = lrc.forward(cfg, table16, params, q)
    assert np.abs(out - ref).max() <= 1e-3 * np.abs(ref).max()

    if n > 2:
        y[n // 2, 3] = -1.0  # a sample without a point
    cache.backward(torch.from_numpy(q).cuda(), torch.from_numpy(y).cuda(), batch=n)
    keep = y[:, 3] >= 0.0
    g, gt, loss = (t.cpu().numpy().astype(np.float64) for t in cache.gradients())
    ref_loss, ref_g, ref_gt = lrc.loss_and_grads(cfg, table16, params, q[keep], y[keep], batch=n)
    assert abs(loss[0] - ref_loss) <= 1e-4 * abs(ref_loss)
    off = 0
    for rows, cols in lrc.LAYER_SHAPES:
        a, b = g[off:off + rows * cols], ref_g[off:off + rows * cols]
        assert np.linalg.norm(a - b) <= 1e-3 * max(np.linalg.norm(b), 1e-30)
        off += rows * cols
    assert np.linalg.norm(gt - ref_gt) <= 1e-3 * np.linalg.norm(ref_gt)
    cache.check()


@pytest.mark.parametrize("log2_table,base,n", [(10, 4, 1), (10, 64, 2000), (11, 16, 3), (14, 16, 700)])
def test_lazy_step_updates_the_touched_entries(device, log2_table, base, n):
    import torch

    from oracle import lrc

    cfg, cache, params, table, _, q, y = _cache(device, log2_table, base, n, table_update="lazy")
    cache.backward(torch.from_numpy(q).cuda(), torch.from_numpy(y).cuda())
    gt = cache.gradients()[1].cpu().numpy().astype(np.float64)
    cache.step()
    after = cache.get_params()[1].cpu().numpy()
    touched = np.repeat((gt.reshape(-1, 2) != 0.0).any(1), 2)
    assert touched.any()
    np.testing.assert_array_equal(after[~touched], table[~touched])
    zero = np.zeros(table.size, np.float64)
    want, _, _ = lrc.adam(cfg, table.astype(np.float64), zero, zero, gt, 1)
    assert np.allclose(after[touched], want[touched], rtol=1e-5, atol=1e-6)
    assert float(cache.gradients()[1].abs().max()) == 0.0
    cache.check()
