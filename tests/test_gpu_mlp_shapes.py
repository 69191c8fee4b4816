"""The warm-start MLP at the edges of its tiles: 64- and 128-column GEMM tiles, weight gradients
in one range of rows and in many, batches that end inside a tile, the smallest and widest
models; an output array of any alignment, written in its own rows only. Against
oracle/mlp_oracle.py with the bars of test_gpu_mlp.py."""
import ctypes

import numpy as np
import pytest
import torch

from filsim_b200.configs import params_for
from filsim_b200.fcm import Context
from filsim_b200.learn import WarmStartModel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nw,hidden,cap,n", [(2, 128, 128, 1), (2, 128, 128, 128), (5, 384, 1280, 1217),
                                             (32, 256, 640, 513), (11, 128, 4096, 4000), (3, 1024, 2560, 2559)])
def test_forward_and_gradients(oracle, gpu_lib, nw, hidden, cap, n):
    from oracle import mlp_oracle
    ctx = Context(params_for(32), max_beads=64, max_filaments=8)
    m = WarmStartModel(ctx, nw=nw, hidden=hidden, batch_capacity=cap, seed=nw)
    rng = np.random.default_rng(n)
    feats = rng.standard_normal((n, m.n_features)).astype(np.float32)
    tgts = rng.standard_normal((n, m.n_targets)).astype(np.float32)
    sd, mu = rng.uniform(0.5, 2, m.n_targets).astype(np.float32), rng.normal(size=m.n_targets).astype(np.float32)
    m.set_normalization(np.zeros(m.n_features), np.ones(m.n_features), mu, sd)
    x, t = np.zeros((m.capacity, m.k_in), np.float32), np.zeros((m.capacity, m.k_out), np.float32)
    x[:n, :m.n_features], t[:n, :m.n_targets] = feats, np.clip((tgts - mu) / sd, -10, 10)
    layers = mlp_oracle.unflatten(m.params(), m.dims)
    yr = mlp_oracle.forward(layers, x)[0][:n, :m.n_targets] * sd + mu
    f = torch.as_tensor(feats, device="cuda")
    size = n * m.n_targets
    out = torch.full((size + 9,), -7.0, device="cuda")
    ctx.call("fs_mlp_forward", ctypes.c_void_p(f.data_ptr()), n, ctypes.c_void_p(out[1:].data_ptr()))
    y = out[1:size + 1].view(n, m.n_targets).cpu().numpy()
    assert np.linalg.norm(y - yr) / np.linalg.norm(yr) < 2e-2
    assert out[0] == -7.0 and bool((out[size + 1:] == -7.0).all())
    g, loss = m.gradients(f, torch.as_tensor(tgts))
    loss_ref, grads = mlp_oracle.loss_and_gradients(layers, x, t, n, m.n_targets)
    assert abs(loss - loss_ref) / loss_ref < 1e-3
    for a, b in zip(mlp_oracle.unflatten(g, m.dims), grads):
        assert all(np.linalg.norm(u - v) / np.linalg.norm(v) < 2e-2 for u, v in zip(a, b))
    ctx.close()
