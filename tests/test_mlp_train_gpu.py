"""The scorer's training kernels at the batch sizes where their tiling can go wrong: a half tile of 128
rows, splits that begin and end in the middle of a tile, one split and many, a batch larger than the
sample set. Reference: the float64 restatement with the device's BF16 roundings; the bounds are those
of the 512-row test (a BF16 rounding flip of one operand, 2^-9, spread over the sums)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _samples(n, seed):
    rng = np.random.default_rng(seed)
    x = np.abs(rng.standard_normal((n, 24), np.float32)) * rng.uniform(0.2, 4.0, 24).astype(np.float32)
    t = np.log1p(np.abs(x[:, 0] * 2 + x[:, 5] - 0.5 * x[:, 11] ** 2)).astype(np.float32)
    return np.ascontiguousarray(x), t


@pytest.fixture(scope="module")
def ctx(nb):
    c = nb.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("batch", [64, 128, 192, 320, 576, 1088, 4160])
def test_gradient_by_batch_size(ctx, batch):
    from oracle import residency as ores

    x, t = _samples(batch, batch)
    ctx.mlp_init(4)
    ctx.mlp_train(x, t, steps=0, batch=batch)  # stores the feature statistics only
    blob = ctx.mlp_get()
    g, loss = ctx.mlp_gradient(x, t)
    r, rloss = ores.mlp_gradient(blob, x, t)
    assert abs(loss - rloss) <= 1e-4 * rloss
    o = ores._blob_parts(blob)
    for a, b in [("w1", "b1"), ("b1", "w2"), ("w2", "b2"), ("b2", "w3"), ("w3", "b3"), ("b3", "mean")]:
        ga, ra = g[o[a]:o[b]].astype(np.float64), r[o[a]:o[b]]
        assert np.abs(ga - ra).max() <= 2e-3 * np.abs(ra).max(), a
    g2, _ = ctx.mlp_gradient(x, t)
    assert np.array_equal(g, g2)
    assert ctx.status() == 0


@pytest.mark.parametrize("n,batch", [(64, 128), (100, 64), (4096, 4096)])
def test_step_and_losses(ctx, n, batch):
    """One AdamW step against the restatement (n = 64: the batch holds every sample twice), and the
    losses of a longer run against the runs of its first steps."""
    from oracle import residency as ores

    x, t = _samples(n, n + 1)
    ctx.mlp_init(6)
    blob = ctx.mlp_get()
    loss = ctx.mlp_train(x, t, steps=5, batch=batch, lr=1e-3, seed=9)
    end = ctx.mlp_get()
    ctx.mlp_set(blob)
    first = ctx.mlp_train(x, t, steps=2, batch=batch, lr=1e-3, seed=9)
    assert np.array_equal(loss[:2], first)
    ctx.mlp_set(blob)
    assert np.array_equal(ctx.mlp_train(x, t, steps=5, batch=batch, lr=1e-3, seed=9), loss)
    assert np.array_equal(ctx.mlp_get(), end)
    if n != 100:
        ctx.mlp_set(blob)
        ctx.mlp_train(x, t, steps=1, batch=batch, lr=1e-3, weight_decay=1e-2, seed=9)
        got = ctx.mlp_get()
        o = ores._blob_parts(blob)
        start = got.copy()
        start[:o["mean"]] = blob[:o["mean"]]
        rep = batch // n
        r, rloss = ores.mlp_gradient(start, np.tile(x, (rep, 1)), np.tile(t, rep))
        assert abs(loss[0] - rloss) <= 1e-4 * rloss
        z = np.zeros(blob.size, np.float32)
        want, _, _ = ores.adamw_step(start, r, z, z, 1, 1e-3, 1e-2)
        sig = np.abs(r[:o["mean"]]) > 1e-3 * np.abs(r[:o["mean"]]).max()  # sign(g) decides step 1
        assert np.abs(got - want)[:o["mean"]][sig].max() <= 1e-6
