"""GPU: a batch whose results are copied in groups is drawn in several raster launches, and every plane that
was asked for is written again by each of them."""
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


def _request(rng, rp, i, w, h, shadow):
    m = i % len(rp.pool)
    sd = scenes.U.shader_data(scenes.orbit_eye(rng, rp.pool[m].kind), w, h, enable_shadow=bool(shadow))
    return scenes.Request(m, i % 2, int(scenes.REQUEST_SHADERS[i % 6]), w, h, shadow, sd, 0.0)


def _sequence(gpu, rp, reqs):
    """Launches of one sequence over these requests, and each one's planes."""
    vb = hserve.ViewBatch(rp, reqs)
    try:
        vb.draw_all()
        return gpu.last_timing()["launches"], [vb.download(k) for k in range(len(reqs))]
    finally:
        vb.release()


def test_a_queued_batch_is_drawn_in_several_raster_launches(gpu, rp):
    """One slot, held by a large request with results in pageable memory, while twelve more queue up:
    they share one batch, which launches more rasters than one sequence does."""
    rng = np.random.default_rng(9)
    sizes = [(2400, 1500), (1900, 1400), (1700, 1100), (1500, 1300), (640, 480), (1300, 900), (300, 211), (1201, 1003),
             (96, 64), (1100, 700), (1000, 1000), (33, 47)]
    planes = [("color",), ("color", "depth", "prim"), ("depth",), ("prim", "color")]
    kinds = {"color": (np.uint8, (4,)), "depth": (np.float32, ()), "prim": (np.uint32, ())}
    first = _request(rng, rp, 2, 3840, 2160, 0)
    reqs = [_request(rng, rp, i, w, h, 512 if i % 3 else 0) for i, (w, h) in enumerate(sizes)]
    alone_first, _ = _sequence(gpu, rp, [first])
    one_sequence, expect = _sequence(gpu, rp, reqs)
    all_reqs = [first] + reqs
    outs = [{k: np.empty((r.height, r.width) + kinds[k][1], kinds[k][0]) for k in p}
            for r, p in zip(all_reqs, [("color", "depth", "prim")] + [planes[i % 4] for i in range(len(reqs))])]
    srv = gpu.Server(8 << 30, 16, 1)
    shared = 0
    try:
        for fill in (7, 9, 11):
            for o in outs:
                for v in o.values():
                    v.fill(fill)
            before = gpu.stats()
            tks = [srv.submit(rp.meshes[r.mesh], r.shader, r.sd, r.width, r.height, diffuse=rp.textures[r.tex][0],
                              normal=rp.textures[r.tex][1], shadow_size=r.shadow, out=o) for r, o in zip(all_reqs, outs)]
            sts = [srv.wait(t) for t in tks]
            after = gpu.stats()
            assert all(s["status"] == gpu.OK for s in sts)
            for r, o, e in zip(reqs, outs[1:], expect):
                for k, v in o.items():
                    assert np.array_equal(v, e[k]), (r.width, r.height, k)
            if {s["batch_requests"] for s in sts[1:]} == {len(reqs)} and after["retries"] == before["retries"]:
                shared += 1
                launches = after["kernel_launches"] - before["kernel_launches"]
                assert launches - alone_first > one_sequence, (launches, alone_first, one_sequence)
    finally:
        srv.close()
    assert shared, "the twelve never shared a batch"
