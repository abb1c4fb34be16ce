"""GPU: a server's large batches, drawn in several raster launches (one per group of views), give the
same bits as each request drawn alone."""
import numpy as np
import pytest

from hsr import scenes
from hsr import serve as hserve

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rp(gpu):
    r = hserve.ResidentPool(scenes.mesh_pool((("grid", 32), ("sphere", 4), ("sphere", 5)), seed=21),
                            scenes.pool_textures(2, 256, seed=5))
    yield r
    r.release()


def test_server_batches_in_raster_groups_equal_alone(gpu, rp):
    """Batches with enough results to copy are drawn in several raster launches, in an order of their
    own, and draw only the planes asked for: every plane asked for equals the request alone."""
    sizes = [(2400, 1500), (1900, 1400), (1700, 1100), (1500, 1300), (640, 480), (1300, 900), (300, 211), (1201, 1003),
             (96, 64), (1100, 700), (1000, 1000), (33, 47)]
    planes = [("color",), ("color", "depth", "prim"), ("depth",), ("prim", "color"), ()]
    rng = np.random.default_rng(3)
    reqs, outs, kinds = [], [], {"color": (np.uint8, 4), "depth": (np.float32, 0), "prim": (np.uint32, 0)}
    for i, (w, h) in enumerate(sizes):
        m = i % len(rp.pool)
        sh = 512 if i % 3 else 0
        sd = scenes.U.shader_data(scenes.orbit_eye(rng, rp.pool[m].kind), w, h, enable_shadow=bool(sh))
        reqs.append(scenes.Request(m, i % 2, int(scenes.REQUEST_SHADERS[i % 6]), w, h, sh, sd, 0.0))
        outs.append({k: np.full((h, w, 4) if kinds[k][1] else (h, w), 7, kinds[k][0]) for k in planes[i % 5]})
    srv = gpu.Server(4 << 30, 16, 2)
    try:
        for _ in range(2):  # the second time everything is queued behind the first's batches
            tks = [srv.submit(rp.meshes[r.mesh], r.shader, r.sd, r.width, r.height, diffuse=rp.textures[r.tex][0],
                              normal=rp.textures[r.tex][1], shadow_size=r.shadow, out=o) for r, o in zip(reqs, outs)]
            assert all(srv.wait(t)["status"] == gpu.OK for t in tks)
    finally:
        srv.close()
    for r, o in zip(reqs, outs):
        vb = hserve.ViewBatch(rp, [r])
        try:
            vb.draw_all()
            alone = vb.download(0)
        finally:
            vb.release()
        for k, v in o.items():
            assert np.array_equal(v, alone[k]), (r.width, r.height, k)
