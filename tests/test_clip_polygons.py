"""Triangles along a corner line of the frustum: rounding bends their polygons, one plane cuts them more
than twice, and they reach more than the ten vertices of exact arithmetic."""
import os
import re

import numpy as np
import pytest

import golden_io
import oracle
from hsr import scenes
from hsr import uniforms as U

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hana-softwarerenderer_gb300", "csrc")
h = float.fromhex
# 4, 5, 6, 7, 9, 11, 12 vertices after the planes W, +X, -X, +Y, -Y, +Z, -Z
CORNER_LINE = np.array([[h("-0x1.525044p-1"), h("0x1.528a66p-1"), h("-0x1.529d74p-1"), h("-0x1.52268ep-1")],
                        [h("0x1.2b5e1ep+4"), h("-0x1.2b921cp+4"), h("0x1.2ba3a8p+4"), h("0x1.2b836cp+4")],
                        [h("0x1.dfd63p-10"), h("-0x1.dfff66p-10"), h("0x1.e00b1cp-10"), h("0x1.dfd4f8p-10")]], np.float32)


def _slivers(rng, n):
    """Clip positions [n][3][4] near the eight corner lines."""
    corner = np.concatenate([rng.choice([-1, 1], (n, 1, 3)), np.ones((n, 1, 1))], 2)
    off = np.exp2(rng.uniform(-23, -12, (n, 1, 1))) * rng.normal(0, 1, (n, 3, 4))
    out = (CORNER_LINE * np.array([1, -1, 1, 1]) * corner * (1 + off)).astype(np.float32)
    out[0] = CORNER_LINE
    return out


def test_polygon_buffers_hold_what_rounding_makes():
    counts = oracle.clip_counts(_slivers(np.random.default_rng(1), 20000))
    assert counts[0].tolist() == [4, 5, 6, 7, 9, 11, 12]
    src = open(os.path.join(CSRC, "kernels_geom.cu")).read()
    places = int(re.search(r"constexpr int kMaxPoly = (\d+);", open(os.path.join(CSRC, "hsr_internal.h")).read()).group(1))
    assert re.search(r"__shared__ float poly\[[^\]]+\]\[2\]\[2\]\[kMaxPoly \* kPolyStride\];", src)
    assert counts.max() <= places
    # and no write goes past the last place, whatever the count
    assert re.search(r"if \(pin != cin && m < kMaxPoly\)", src) and re.search(r"if \(cin && m < kMaxPoly\)", src)


@pytest.mark.gpu
@pytest.mark.parametrize("large", [False, True])
def test_polygons_of_many_vertices_vs_oracle(gpu, large):
    """Each sliver in a mesh of triangles through the same corners' positions (their neighbours in the
    clipper's shared memory), as the first and as a later face; `large`: with enough faces beside
    them that the clipper runs in a grid of its own."""
    import hsr

    rng = np.random.default_rng(2)
    c = _slivers(rng, 4000)
    n = oracle.clip_counts(c).max(1)
    pick = np.concatenate([[0], np.nonzero(n == 11)[0][:4], np.nonzero(n >= 12)[0][:7], np.nonzero(n == 10)[0][:2]])
    assert n.max() >= 12
    w, hgt, more = 150, 110, (1 << 21) if large else 0
    for i in pick[:3] if large else pick:
        # positions are weights of the three corners (the last column is zero), so a corner's clip
        # position is the corner itself
        pos = np.concatenate([np.eye(3), rng.normal(0, 1, (90, 3))]).astype(np.float32)
        tri = np.concatenate([[[0, 1, 2]], rng.integers(3, 93, (60, 3)), [[0, 1, 2], [2, 1, 0], [1, 2, 0]],
                              rng.integers(0, 93, (50, 3)), np.full((more, 3), 5)]).astype(np.int32)
        faces = np.repeat(tri[:, :, None], 3, axis=2)
        faces[:, :, 1:] = 0
        mesh = scenes.Mesh(pos, np.array([[0, 0, 1]], np.float32), np.zeros((1, 2), np.float32), faces)
        sd = U.shader_data((0, 0, 1), w, hgt, identity_mvp=True)
        m = np.zeros((4, 4), np.float32)
        m[:, :3] = c[i].T
        sd["camera_vp_matrix"] = m.reshape(sd["camera_vp_matrix"].shape)
        rb = oracle.Buffers(w, hgt, (0, 0, 0, 255), 1.0)
        oracle.draw(mesh, scenes.FLAT, sd, rb)
        target, gm = hsr.Target(w, hgt), hsr.Mesh(mesh)
        try:
            hsr.draw_batch([hsr.make_desc(gm, scenes.FLAT, sd, target, clear=((0, 0, 0, 255), 1.0))])
            got = target.download()
        finally:
            gm.release()
            target.release()
        golden_io.assert_pass(got, {"depth": rb.depth, "color": rb.color, "prim": rb.prim}, "main", f"sliver {i}", 1)
