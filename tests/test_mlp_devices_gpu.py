"""GPU test of the scorer in contexts on two devices of one process: each opts its kernels in to their shared
memory on its own device."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_two_devices(nb):
    import torch

    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    rng = np.random.default_rng(1)
    x, t = rng.normal(size=(512, 24)).astype(np.float32), rng.random(512).astype(np.float32)
    got = []
    for device in (0, 1):
        ctx = nb.Context(device)
        try:
            ctx.mlp_init(3)
            ctx.mlp_train(x, t, steps=5, batch=128)
            got.append((ctx.mlp_get(), ctx.mlp_infer(x)))
        finally:
            ctx.close()
    assert all(np.array_equal(a, b) for a, b in zip(*got))
