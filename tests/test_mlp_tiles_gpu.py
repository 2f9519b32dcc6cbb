"""The fp32 network's 64-row tiles against the float64 reference: one row, batches around
one tile, and batches where a block takes a second tile."""
import numpy as np
import pytest

from oracle import mlp_ref
from genoaligner_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [(0, 1), (0, 15), (0, 63), (0, 64), (0, 65), (32, 1), (64, 0), (64, 65)])
def test_forward_and_gradient(rows):
    torch = pytest.importorskip("torch")
    per_sm, extra = rows
    n = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + extra
    rng = np.random.default_rng(n)
    params = api.cost_model_init(seed=11)
    params[-2:] = [1.0, -0.5]
    api.cost_model_set(params)
    x = rng.normal(0, 1, size=(n, 66)).astype(np.float32)
    t = rng.normal(2, 1, size=(n, 2)).astype(np.float32)
    xt, tt = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    y_ref, _ = mlp_ref.forward(params, x)
    g_ref, loss_ref = mlp_ref.gradient(params, x, t)
    y = api.mlp_forward(xt).cpu().numpy()
    g, loss = api.mlp_gradient(xt, tt)
    # fp32 sums of up to 128 terms a layer: 128 * 2^-24 of the terms' size, over three layers
    tol = 3 * 128 * 2.0 ** -24
    assert np.abs(y - y_ref).max() <= tol * np.abs(y_ref).max()
    assert abs(loss - loss_ref) <= 4 * tol * loss_ref
    assert np.linalg.norm(g - g_ref) <= 4 * tol * np.linalg.norm(g_ref)
