"""ReSTIR's light search without its step table, which lights whose weights add up to infinity do not have: a draw
takes the same slot as the oracle's, so images agree where they are finite and are not finite in the same places."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("reference", [False, True])
def test_infinite_total(nb, orc, reference):
    scene = nb.synth_city(seed=21, grid=6, size_m=200.0, target_tris=20_000, median_tris=300, max_tris=5_000,
                          emissive_quads=4, emissive_tris=200, emissive_sigma=1.5)
    lit = np.nonzero(scene.prim_material[:, 11] > 0)[0]
    scene.prim_material[lit[::3], 8:11] = 1.0
    scene.prim_material[lit[::3], 11] = 1e38  # ten of these and the total is infinite
    sb = nb.SceneBVH(scene)
    ctx = nb.Context(0)
    try:
        ctx.upload(sb)
        kw = dict(candidates=16, temporal=True)
        if not reference:
            kw.update(spatial=3, radius_px=30.0, m_cap=20.0)
        ctx.set_restir(reference_mode=reference, **kw)
        ref = orc.RestirOracle(orc.OracleScene(sb), sb.materials, reference_mode=reference, **kw)
        for f in range(2):
            v = nb.view_pinhole((0.5 * f, 50, -150), (0, 10, 0), width=61, height=37, spp=1, max_depth=2, seed=3, frame=f,
                                flags=nb.VIEW_RESTIR)
            got = ctx.render(v)[0].reshape(-1, 3)
            want, _ = ref.render(v)
            assert np.array_equal(np.isfinite(got), np.isfinite(want))
            same = np.where(np.isfinite(want), got == want, True).all(1)
            assert same.mean() > 0.99, (f, same.mean())
        assert ctx.status() == 0
    finally:
        ctx.close()
