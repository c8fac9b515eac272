"""ReSTIR's candidate draw over the light counts and shapes its branches depend on: a handful, a
staged table, more than the staged limit of 8,192, with spheres, rectangles and slivers among them;
candidate counts around the half ring of 32; both estimators. Images against the scalar oracle with
the bounds of the two-frame parity tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(nb, tris):
    base = nb.synth_city(seed=21, grid=6, size_m=200.0, target_tris=20_000, median_tris=300, max_tris=5_000,
                         emissive_quads=4, emissive_tris=tris, emissive_sigma=1.5)
    rng = np.random.default_rng(tris)
    n = 24
    typ = np.repeat([nb.native.PRIM_SPHERE, nb.native.PRIM_RECTANGLE, nb.native.PRIM_TRIANGLE], n // 3).astype(np.int32)
    geom = np.zeros((n, 15), np.float32)
    geom[:, 0:3] = rng.uniform([-90, 2, -90], [90, 40, 90], (n, 3))
    for i in range(n):
        if typ[i] == nb.native.PRIM_SPHERE:
            geom[i, 3] = rng.uniform(0.2, 3.0)
        elif typ[i] == nb.native.PRIM_RECTANGLE:
            geom[i, 3:9] = rng.normal(size=6)
        else:  # slivers: two far corners close together
            far = rng.normal(size=3) * 5
            geom[i, 3:6] = geom[i, 0:3] + far
            geom[i, 6:9] = geom[i, 0:3] + far * 1.01 + rng.normal(size=3) * 1e-3
    mat = np.tile(base.prim_material[0], (n, 1))
    mat[:, 8:11] = rng.uniform(0.2, 1.0, (n, 3))
    mat[:, 11] = rng.lognormal(0.0, 1.5, n)
    return nb.SceneBVH(nb.HostScene(
        np.concatenate([base.prim_type, typ]), np.concatenate([base.prim_geom, geom]),
        np.concatenate([base.prim_material, mat]), np.append(base.object_first, base.prim_count),
        np.append(base.object_prims, n)))


@pytest.mark.parametrize("reference", [False, True])
@pytest.mark.parametrize("tris,candidates", [(0, 1), (0, 33), (600, 31), (600, 64), (9000, 32)])
def test_candidates(nb, orc, tris, candidates, reference):
    sb = _scene(nb, tris)
    ctx = nb.Context(0)
    try:
        ctx.upload(sb)
        kw = dict(candidates=candidates, temporal=True)
        if not reference:
            kw.update(spatial=3, radius_px=30.0, m_cap=20.0)
        ctx.set_restir(reference_mode=reference, **kw)
        ref = orc.RestirOracle(orc.OracleScene(sb), sb.materials, reference_mode=reference, **kw)
        for f in range(2):
            v = np.concatenate([nb.view_pinhole((0.5 * f, 50, -150), (0, 10, 0), width=61, height=37, spp=1, max_depth=2,
                                                seed=3, frame=f, flags=nb.VIEW_RESTIR),
                                nb.view_pinhole((40, 30, 20), (0, 5, 0), width=9, height=7, spp=3, max_depth=1,
                                                seed=4, frame=f, flags=nb.VIEW_RESTIR)])
            got = np.concatenate([i.reshape(-1, 3) for i in ctx.render(v)])
            want, _ = ref.render(v)
            exact = (got == want).all(1).mean()
            err = (np.abs(got - want).sum(1) / np.maximum(np.abs(want).sum(1), 1e-6)).mean()
            assert err < 1e-4 and exact > 0.99, (f, err, exact)
        assert ctx.status() == 0
    finally:
        ctx.close()
