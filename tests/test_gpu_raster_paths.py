"""The raster's two ways of handing out tiles (a warp per tile, a CTA per tile where tiles are
few) and the order of draws into one target, against the oracle.

Depth, primitive ids and alpha are exact, RGB within 1 LSB (powf)."""
import numpy as np
import pytest

import golden_io
import oracle
from hsr import frame as hframe
from hsr import scenes
from hsr import uniforms as U

pytestmark = pytest.mark.gpu


@pytest.fixture
def tuned(gpu):
    old = gpu.get_tuning()
    yield gpu
    gpu.set_tuning(tile=old.tile, warps_per_cta=old.warps_per_cta, ctas_per_sm=old.ctas_per_sm)


def _check(got, rb, label):
    golden_io.assert_pass(got, {"depth": rb.depth, "color": rb.color, "prim": rb.prim}, "main", label, 1)


# one CTA per SM puts the line between the paths at a few hundred tiles, eight at a few thousand
@pytest.mark.parametrize("ctas", [1, 8])
@pytest.mark.parametrize("tile,warps", [(8, 4), (8, 8), (16, 4), (32, 4)])
@pytest.mark.parametrize("size", [(1, 1), (37, 29), (518, 391)])
def test_tiles_by_warp_and_by_cta_vs_oracle(tuned, size, tile, warps, ctas):
    """A tie soup of heavy overdraw and a shadowed normal-map frame at one tile, few and many."""
    tuned.set_tuning(tile=tile, warps_per_cta=warps, ctas_per_sm=ctas)
    w, h = size
    soup = scenes.soup_frame(3000, w, h, seed=w + tile, median_edge_px=max(2.0, w / 12), dup_frac=0.05)
    shaded = scenes.sphere_frame(3, w, h, shader=scenes.NORMALMAP, eye=(0.3, 0.4, 2.2), tex_size=32, seed=3, shadow=96,
                                 nm_size=16)
    for fr in (soup, shaded):
        g = hframe.GpuFrame(fr)
        try:
            g.render()
            got = g.download()
        finally:
            g.release()
        for k, rb in oracle.render_frame(fr).items():
            _check(got[k], rb, f"{fr.name} {k} tile{tile}x{warps} ctas{ctas}")


@pytest.mark.parametrize("ctas", [1, 8])
@pytest.mark.parametrize("tile", [8, 16, 32])
@pytest.mark.parametrize("size", [(90, 70), (700, 400)])
def test_draws_into_one_target_follow_each_other(tuned, size, tile, ctas):
    """Four objects into one target and one shadow map in one batch (only the first of each clears),
    some tiles without records in some of them: each draw tests against what the earlier ones left,
    and every main draw sees the whole shadow map."""
    import hsr

    tuned.set_tuning(tile=tile, warps_per_cta=4, ctas_per_sm=ctas)
    w, h = size
    rng = np.random.default_rng(w + tile)
    objs, clear = [], ((0, 0, 0, 255), 1.0)
    for k in range(4):
        fr = scenes.sphere_frame(2 + k % 2, w, h, shader=scenes.BLINN, tex_size=16, seed=k)
        place = U.Mat4.identity()
        for i in range(3):
            place.r[i][3] = np.float32(rng.uniform(-0.4, 0.4))
            place.r[i][i] = np.float32(0.55)
        objs.append((fr, U.shader_data((0.2, 0.3, 2.5), w, h, model=place, enable_shadow=True)))
    main, smap = hsr.Target(w, h), hsr.Target(64, 64)
    meshes, texs = [hsr.Mesh(f.mesh) for f, _ in objs], [hsr.Texture(f.diffuse) for f, _ in objs]
    try:
        descs = [hsr.make_desc(m, scenes.SHADOW, sd, smap, t, clear=clear if k == 0 else None)
                 for k, (m, t, (_, sd)) in enumerate(zip(meshes, texs, objs))]
        descs += [hsr.make_desc(m, scenes.BLINN, sd, main, t, shadow_map=smap, prim_base=1000 * k,
                                clear=clear if k == 0 else None) for k, (m, t, (_, sd)) in enumerate(zip(meshes, texs, objs))]
        hsr.draw_batch(descs)
        got, got_s = main.download(), smap.download()
    finally:
        for o in [main, smap, *meshes, *texs]:
            o.release()
    rb, rs = oracle.Buffers(w, h, *clear), oracle.Buffers(64, 64, *clear)
    for fr, sd in objs:
        oracle.draw(fr.mesh, scenes.SHADOW, sd, rs, fr.diffuse)
    for k, (fr, sd) in enumerate(objs):
        oracle.draw(fr.mesh, scenes.BLINN, sd, rb, fr.diffuse, shadow_map=rs, prim_base=1000 * k)
    _check(got_s, rs, "shadow map")
    _check(got, rb, "main")


@pytest.mark.parametrize("tile", [8, 16, 32])
@pytest.mark.parametrize("edge", [1, 5, 6, 9, 17, 40])
def test_ranges_of_every_width_and_exact_records_vs_oracle(tuned, edge, tile):
    """Triangles whose pixel ranges hold less than a window of 32 candidates, exactly whole ones, or
    whole ones and a remainder, every second one with a corner within 2^-8 of a pixel from the
    left or bottom border (those records take the literal divisions)."""
    tuned.set_tuning(tile=tile, warps_per_cta=4, ctas_per_sm=8)
    w, h, n = 70, 52, 400
    rng = np.random.default_rng(edge * 100 + tile)
    p = np.empty((n, 3, 2))
    p[:, 0] = rng.uniform(0, (w, h), (n, 2))
    p[:, 1] = p[:, 0] + rng.uniform(0.3, edge, (n, 2)) * (1, -1)
    p[:, 2] = p[:, 0] + rng.uniform(0.3, edge, (n, 2))
    p = np.clip(p, 0, (w - 1e-3, h - 1e-3))
    p[::4, 0, 0] = rng.uniform(1e-5, 3e-3, len(p[::4]))
    p[2::4, 1, 1] = rng.uniform(1e-5, 3e-3, len(p[2::4]))
    pos = np.zeros((n, 3, 3), np.float32)
    pos[:, :, 0] = p[:, :, 0] / w * 2 - 1
    pos[:, :, 1] = p[:, :, 1] / h * 2 - 1
    pos[:, :, 2] = rng.integers(0, 40, (n, 1)) / 50  # many equal depths
    tri = np.arange(3 * n, dtype=np.int32).reshape(n, 3)
    faces = np.zeros((n, 3, 3), np.int32)
    faces[:, :, 0] = tri
    mesh = scenes.Mesh(pos.reshape(-1, 3), np.array([[0, 0, 1]], np.float32), np.zeros((1, 2), np.float32), faces)
    fr = scenes.Frame(mesh, scenes.FLAT, U.shader_data((0, 0, 1), w, h, identity_mvp=True), w, h, name=f"ranges{edge}")
    g = hframe.GpuFrame(fr)
    try:
        g.render()
        got = g.download()
    finally:
        g.release()
    rb = oracle.render_frame(fr)["main"]
    assert (rb.prim > 0).any()
    _check(got["main"], rb, f"{fr.name} tile{tile}")


@pytest.mark.parametrize("tile", [8, 16, 32])
@pytest.mark.parametrize("edge", [4, 12, 60])
def test_hidden_candidates_of_overdrawn_tiles_vs_oracle(tuned, edge, tile):
    """Draws of few and of many candidates per pixel (the second kind leaves out what lies behind the
    buffer): steep triangles, equal depths and neighbours one unit apart, depths of zero and next to it,
    and a second draw over the first one's depth."""
    import hsr

    tuned.set_tuning(tile=tile, warps_per_cta=4, ctas_per_sm=8)
    w, h, n = 75, 58, 500
    rng = np.random.default_rng(edge + tile)
    main = hsr.Target(w, h)
    rb = oracle.Buffers(w, h, (0, 0, 0, 255), 1.0)
    held = [main]
    try:
        for k in range(2):
            p = np.clip(rng.uniform(0, (w, h), (n, 1, 2)) + rng.uniform(-edge / 2, edge / 2, (n, 3, 2)), 0.01, (w - 0.01, h - 0.01))
            z = rng.uniform(-0.9, 0.95, (n, 3)).astype(np.float32)  # steep
            flat = np.float32(0.25) + np.spacing(np.float32(0.25)) * rng.integers(-2, 3, (n, 1)).astype(np.float32)
            z[n // 2:] = flat[n // 2:]
            tiny = np.array([-1, -1 + 2.0**-24, -1 + 2.0**-20, -0.999, -0.5], np.float32)
            z[::29] = tiny[rng.integers(0, 5, (len(z[::29]), 3))]
            pos = np.zeros((n, 3, 3), np.float32)
            pos[:, :, 0] = p[:, :, 0] / w * 2 - 1
            pos[:, :, 1] = p[:, :, 1] / h * 2 - 1
            pos[:, :, 2] = z
            faces = np.zeros((n, 3, 3), np.int32)
            faces[:, :, 0] = np.arange(3 * n, dtype=np.int32).reshape(n, 3)
            mesh = scenes.Mesh(pos.reshape(-1, 3), np.array([[0, 0, 1]], np.float32), np.zeros((1, 2), np.float32), faces)
            sd = U.shader_data((0, 0, 1), w, h, identity_mvp=True)
            gm = hsr.Mesh(mesh)
            held.append(gm)
            hsr.draw_batch([hsr.make_desc(gm, scenes.FLAT, sd, main, clear=((0, 0, 0, 255), 1.0) if k == 0 else None,
                                          prim_base=1000 * k)])
            oracle.draw(mesh, scenes.FLAT, sd, rb, prim_base=1000 * k)
        got = main.download()
    finally:
        for o in held:
            o.release()
    assert (rb.prim > 1000).any() and (rb.depth < 1.0).any()
    _check(got, rb, f"hidden edge{edge} tile{tile}")


@pytest.mark.parametrize("more", [-1, 0, 1])
def test_large_meshes_around_a_position_a_face_vs_oracle(gpu, more):
    """More than 2^18 faces: with fewer positions than faces the screen vertices are computed first,
    else by the pass that culls the faces."""
    w, h, n = 640, 360, (1 << 18) + 37
    rng = np.random.default_rng(7 + more)
    npos = n + more
    walk = np.cumsum(rng.normal(0, 2.5, (npos, 2)), axis=0) + rng.uniform(0, 100, 2)
    p = np.abs((walk + (w, h)) % (2 * w, 2 * h) - (w, h)) * (1.02, 1.02) - (0.01 * w, 0.01 * h)  # some leave the target
    pos = np.empty((npos, 3), np.float32)
    pos[:, 0], pos[:, 1] = p[:, 0] / w * 2 - 1, p[:, 1] / h * 2 - 1
    pos[:, 2] = rng.uniform(-1.001, 1.0, npos)
    faces = np.zeros((n, 3, 3), np.int32)
    faces[:, :, 0] = (np.arange(n)[:, None] + np.arange(3)) % npos
    mesh = scenes.Mesh(pos, np.array([[0, 0, 1]], np.float32), np.zeros((1, 2), np.float32), faces)
    fr = scenes.Frame(mesh, scenes.FLAT, U.shader_data((0, 0, 1), w, h, identity_mvp=True), w, h, name=f"walk{more}")
    g = hframe.GpuFrame(fr)
    try:
        g.render()
        got = g.download()
    finally:
        g.release()
    rb = oracle.render_frame(fr)["main"]
    assert (rb.prim > 0).mean() > 0.5
    _check(got["main"], rb, fr.name)


@pytest.mark.parametrize("size", [(200, 160), (2100, 2090)])
@pytest.mark.parametrize("nbig", [0, 1, 3, 300, 6000])
def test_split_triangles_and_the_scan_behind_them_vs_oracle(tuned, nbig, size):
    """No, few (many warps each) and many (several rounds of warps) triangles that are split, small and
    clipped ones among them, before a scan of one block and of more than 32 (8x8 tiles)."""
    tuned.set_tuning(tile=8, warps_per_cta=4, ctas_per_sm=8)
    w, h = size
    rng = np.random.default_rng(nbig + w)
    n = nbig + 500
    edge = np.full(n, 5.0)
    edge[rng.permutation(n)[:nbig]] = min(w, h) if nbig < 10 else 110.0
    c = rng.uniform(0, (w, h), (n, 1, 2)) if nbig >= 10 else rng.uniform(0.3, 0.7, (n, 1, 2)) * (w, h)
    ang = rng.uniform(0, 2 * np.pi, (n, 1)) + np.arange(3) * (2 * np.pi / 3)
    p = c + edge[:, None, None] / 2 * np.stack([np.cos(ang), np.sin(ang)], axis=2)
    pos = np.empty((n, 3, 3), np.float32)
    pos[:, :, 0], pos[:, :, 1] = p[:, :, 0] / w * 2 - 1, p[:, :, 1] / h * 2 - 1
    pos[:, :, 2] = rng.uniform(-0.9, 0.9, (n, 1)).astype(np.float32)
    faces = np.zeros((n, 3, 3), np.int32)
    faces[:, :, 0] = np.arange(3 * n, dtype=np.int32).reshape(n, 3)
    mesh = scenes.Mesh(pos.reshape(-1, 3), np.array([[0, 0, 1]], np.float32), np.zeros((1, 2), np.float32), faces)
    fr = scenes.Frame(mesh, scenes.FLAT, U.shader_data((0, 0, 1), w, h, identity_mvp=True), w, h, name=f"split{nbig}")
    g = hframe.GpuFrame(fr)
    try:
        g.render()
        split = tuned.last_timing()["split_triangles"]
        got = g.download()
    finally:
        g.release()
    assert split >= nbig // 3 if nbig else split == 0
    _check(got["main"], oracle.render_frame(fr)["main"], fr.name)
