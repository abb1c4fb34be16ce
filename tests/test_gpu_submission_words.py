"""GPU: the submission word of a record (face, fan, clipped) up to its highest bit: a mesh of more than 2^26
faces, of which the first and the last few hundred show."""
import numpy as np
import pytest

import golden_io
import oracle
from hsr import scenes
from hsr import uniforms as U

pytestmark = pytest.mark.gpu


def test_ties_between_the_first_and_the_last_faces_of_a_huge_mesh(gpu):
    """Equal depths everywhere, clipped triangles among them: the later face wins, whatever the word's
    sign, and its primitive id is its own."""
    w, h, k, n = 160, 120, 300, (1 << 26) + 777
    rng = np.random.default_rng(5)
    p = rng.uniform(-1.3, 1.3, (2 * k, 1, 2)) + rng.normal(0, 0.25, (2 * k, 3, 2))
    pos = np.zeros((6 * k + 1, 3), np.float32)
    pos[:-1, :2] = p.reshape(-1, 2)
    pos[:-1, 2] = np.repeat(rng.integers(-1, 2, 2 * k) / 4, 3)
    shown = np.zeros((2 * k, 3, 3), np.int32)
    shown[:, :, 0] = np.arange(6 * k).reshape(2 * k, 3)
    one = (np.array([[0, 0, 1]], np.float32), np.zeros((1, 2), np.float32))
    faces = np.zeros((n, 3, 3), np.int32)  # the others: a point each
    faces[k:-k, :, 0] = 6 * k
    faces[:k], faces[-k:] = shown[:k], shown[k:]
    sd = U.shader_data((0, 0, 1), w, h, identity_mvp=True)
    clear = ((0, 0, 0, 255), 1.0)
    target, gm = gpu.Target(w, h), gpu.Mesh(scenes.Mesh(pos, *one, faces))
    try:
        gpu.draw_batch([gpu.make_desc(gm, scenes.SHADOW, sd, target, clear=clear)])
        got = target.download()
    finally:
        gm.release()
        target.release()
    rb = oracle.Buffers(w, h, *clear)
    oracle.draw(scenes.Mesh(pos, *one, shown), scenes.SHADOW, sd, rb)
    prim = np.where(rb.prim > k, rb.prim + (n - 2 * k), rb.prim).astype(np.uint32)
    assert (rb.prim > k).any() and ((rb.prim > 0) & (rb.prim <= k)).any()
    golden_io.assert_pass(got, {"depth": rb.depth, "color": rb.color, "prim": prim}, "main", "2^26 faces", 1)
