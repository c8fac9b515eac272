"""GPU test of the residency selection at the edges of its score order (tiles of 2,048 keys, 32 objects a
block), of its shared memory and of the light table (4,096 lights a pass): flags, toggles and
applied order equal the restatement exactly, and the shaded image, whose lights are the resident ones,
agrees with the oracle in the share of pixels that the residency tests use."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,grid_z,quads,frac,max_toggles", [
    (1, 1, 1, 0.5, 0), (8, 4, 3, 0.3, 5), (64, 32, 2, 0.45, 0), (64, 48, 4200, 0.6, 100), (128, 100, 40, 0.15, 0)])
def test_selection_sizes(nb, orc, grid, grid_z, quads, frac, max_toggles):
    from oracle import residency as ores

    scene = nb.synth_city(seed=5, grid=grid, grid_z=grid_z, size_m=1500.0, target_tris=30 * grid * grid_z + 200,
                          median_tris=12, max_tris=200, emissive_quads=quads)
    sb = nb.SceneBVH(scene)
    ctx = nb.Context(0)
    try:
        ctx.upload(sb)
        nbytes = ctx.object_bytes()
        budget = int(frac * nbytes.sum())
        prm = nb.ResidencyParams.make(nb.POLICY_RAYHIT_BUDGET, budget_bytes=budget, camera_motion=0.7,
                                      memory_pressure=0.5, min_active=1, max_toggles=max_toggles,
                                      resident_key_bonus=0.25)
        flags = ctx.residency_flags()
        for frame, pos in enumerate([(0, 80, -700), (90, 60, -500)]):
            view = nb.view_pinhole(pos, (0, 0, 0), width=80, height=45, spp=1, max_depth=2, seed=frame)
            ctx.reset_object_hits()
            ctx.render(view, count_hits=True)
            toggles = ctx.residency_step(prm, view)
            feats, keys = ctx.residency_last()
            visible = feats[:, 2] > 0.5
            reserve = ores.reserve_count(sb.object_count, 0.02, 0.06, 0.7)
            want, want_t = ores.select(keys, visible, nbytes, budget, reserve, 1, flags, max_toggles=max_toggles,
                                       resident_bonus=0.25)
            got = ctx.residency_flags()
            assert np.array_equal(got, want)
            assert toggles == want_t
            flags = got
        root = sb.instances["blas_root_index"].copy()
        root[flags == 0] = -1
        ref = orc.OracleScene(sb, blas_root=root)
        view = nb.view_pinhole((0, 60, -400), (0, 0, 0), width=48, height=27, spp=2, max_depth=2, seed=9)
        want_img, _, _ = orc.render(ref, sb.materials, view)
        assert (ctx.render(view)[0].reshape(-1, 3) == want_img).all(1).mean() > 0.99
    finally:
        ctx.close()


def test_budget_walk_many_failures(nb):
    """Objects of 1, L, 1, L - 1, ... triangles in score order under the bytes of one L: nearly every
    second candidate would fit by itself and fails after its neighbour, more often than the
    block's rounds, so the last part falls to the warp."""
    from oracle import residency as ores

    sizes = np.ravel(np.column_stack([np.ones(60, int), np.arange(60, 0, -1)]))
    n = int(sizes.sum())
    rng = np.random.default_rng(2)
    geom = np.zeros((n, 15), np.float32)
    centre = np.repeat(rng.uniform(-50, 50, (sizes.size, 3)), sizes, 0)
    for k in range(3):
        geom[:, 3 * k:3 * k + 3] = centre + rng.uniform(-1, 1, (n, 3))
    mat = np.full((n, 20), 0.5, np.float32)
    cuts = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32)
    ctx = nb.Context(0)
    try:
        ctx.upload(nb.SceneBVH(nb.HostScene(np.ones(n, np.int32), geom, mat, cuts[:-1], np.diff(cuts))))
        nbytes = ctx.object_bytes()
        for budget in (int(nbytes[1]), int(nbytes[1]) * 3 // 2, int(nbytes[0]) - 4, int(nbytes.sum())):
            prm = nb.ResidencyParams.make(nb.POLICY_RAYHIT_BUDGET, budget_bytes=budget, min_active=0)
            flags = ctx.residency_flags()
            view = nb.view_pinhole((0, 0, -200), (0, 0, 0), width=8, height=8, spp=1, max_depth=1)
            ctx.residency_step(prm, view)
            feats, keys = ctx.residency_last()
            reserve = ores.reserve_count(sizes.size, 0.02, 0.06, 0.0)
            want, _ = ores.select(keys, feats[:, 2] > 0.5, nbytes, budget, reserve, 0, flags)
            assert np.array_equal(ctx.residency_flags(), want)
    finally:
        ctx.close()
