"""GPU: meshes that the library keeps in an order of its own (2^15 faces and more), their upload's memory,
and normals replaced after the upload.

Depth, primitive ids and alpha are exact against the oracle, RGB within 1 LSB (powf); draws of the same
triangles through two ways of keeping them give the same bytes."""
import numpy as np
import pytest

import golden_io
import oracle
from hsr import frame as hframe
from hsr import scenes
from hsr import uniforms as U

pytestmark = pytest.mark.gpu
CLEAR = ((0, 0, 0, 255), 1.0)


def _draw(hsr, mesh, shader, sd, w, h, diffuse=None, normal=None, update=None):
    """The planes of one draw of `mesh` (a scenes.Mesh), its normals replaced by `update` first."""
    held = [hsr.Target(w, h), hsr.Mesh(mesh)]
    try:
        tex = [None if t is None else hsr.Texture(t) for t in (diffuse, normal)]
        held += [t for t in tex if t]
        if update is not None:
            held[1].update_normals(update)
        hsr.draw_batch([hsr.make_desc(held[1], shader, sd, held[0], *tex, clear=CLEAR)])
        return held[0].download()
    finally:
        for o in reversed(held):
            o.release()


def _oracle(mesh, shader, sd, w, h, diffuse=None, normal=None):
    rb = oracle.Buffers(w, h, *CLEAR)
    oracle.draw(mesh, shader, sd, rb, diffuse, normal)
    return {"depth": rb.depth, "color": rb.color, "prim": rb.prim}


def _equal(a, b):
    for p in ("color", "depth", "prim"):
        assert np.array_equal(a[p].view(np.uint8), b[p].view(np.uint8)), p


@pytest.fixture
def faults(gpu):
    yield gpu
    gpu.set_fault_injection(0, 0)


def test_a_large_mesh_without_scratch_keeps_the_callers_order(faults):
    """More than 2^20 positions, faces and normals (several pieces): with the ordering scratch and without
    it the same bytes."""
    n = 370
    fr = scenes.sphere_frame(3, 300, 260, shader=scenes.BLINN, tex_size=32, seed=1)
    pos, tri = fr.mesh.pos, fr.mesh.faces[:, :, 0]
    rng = np.random.default_rng(0)
    size = np.exp(rng.uniform(-3, 0, n)).astype(np.float32)
    off = rng.uniform(-1, 1, (n, 3)).astype(np.float32)
    many = scenes.Mesh((pos[None] * size[:, None, None] + off[:, None]).reshape(-1, 3), np.tile(fr.mesh.nrm, (n, 1)),
                       np.tile(fr.mesh.uv, (n, 1)),
                       (np.repeat(tri[None] + (np.arange(n) * len(pos))[:, None, None], 1, 0).reshape(-1, 3)[:, :, None]
                        * np.ones(3, np.int32)).astype(np.int32))
    # faces past one piece: each object four times
    many.faces = np.ascontiguousarray(np.tile(many.faces, (4, 1, 1)))
    far = np.repeat(many.pos[:1], (1 << 20) - len(many.pos) + 5000, 0)  # positions no face uses
    many.pos = np.concatenate([many.pos, far])
    many.nrm = np.concatenate([many.nrm, np.repeat(many.nrm[:1], len(far), 0)])
    assert len(many.faces) > 1 << 20 and len(many.pos) > 1 << 20 and len(many.nrm) > 1 << 20
    kept = _draw(faults, many, fr.shader, fr.sd, 300, 260, fr.diffuse)
    faults.set_fault_injection(faults.FAULT_UPLOAD_SCRATCH, 0)
    plain = _draw(faults, many, fr.shader, fr.sd, 300, 260, fr.diffuse)
    assert (kept["prim"] > 0).mean() > 0.2
    _equal(kept, plain)


def test_upload_gives_its_scratch_back(gpu):
    """The scratch of a mesh of 2M triangles (some 200 MB) does not stay reserved once it is released."""
    import torch

    n = 2000000
    rng = np.random.default_rng(1)
    faces = np.zeros((n, 3, 3), np.int32)
    faces[:, :, 0] = np.arange(3 * n, dtype=np.int32).reshape(n, 3)
    mesh = scenes.Mesh(rng.uniform(-1, 1, (3 * n, 3)).astype(np.float32), np.array([[0, 0, 1]], np.float32),
                       np.zeros((1, 2), np.float32), faces)
    small = scenes.sphere_frame(2, 8, 8, shader=scenes.FLAT, tex_size=8, seed=1).mesh
    gpu.Mesh(small).release()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    gpu.Mesh(mesh).release()
    torch.cuda.synchronize()
    assert before - torch.cuda.mem_get_info()[0] <= 64 << 20


def _grid(cells, seed, split):
    """A height field of 2 * cells^2 triangles; `split`: uvs and normals in arrays of their own order."""
    m = scenes.grid_mesh(cells, cells, seed)
    if split:
        rng = np.random.default_rng(seed)
        m.faces = m.faces.copy()
        for k, name in ((1, "uv"), (2, "nrm")):
            at = rng.permutation(len(m.pos)).astype(np.int32)
            v = np.empty_like(getattr(m, name))
            v[at] = getattr(m, name)
            setattr(m, name, v)
            m.faces[:, :, k] = at[m.faces[:, :, k]]
    return m


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("cells", [20, 127, 128, 200])  # 2^15 faces at 128
@pytest.mark.parametrize("shader", [scenes.GROUND, scenes.BLINN])
def test_normals_replaced_after_the_upload(gpu, cells, split, shader):
    """The same bytes as a mesh uploaded with those normals, and the oracle's picture."""
    w, h = 320, 200
    mesh = _grid(cells, cells, split)
    rng = np.random.default_rng(cells)
    new = scenes.fixed_point_normals((mesh.nrm + rng.normal(0, 0.3, mesh.nrm.shape)).astype(np.float32))
    sd = U.shader_data((0.4, 1.3, 1.9), w, h)
    tex = scenes.noise_texture(64, 64, 4, 3)
    got = _draw(gpu, mesh, shader, sd, w, h, tex, update=new)
    with_new = scenes.Mesh(mesh.pos, new, mesh.uv, mesh.faces)
    _equal(got, _draw(gpu, with_new, shader, sd, w, h, tex))
    exp = _oracle(with_new, shader, sd, w, h, tex)
    assert (exp["prim"] > 0).mean() > 0.1
    assert not np.array_equal(exp["color"], _oracle(mesh, shader, sd, w, h, tex)["color"])
    golden_io.assert_pass(got, exp, "main", f"normals {cells}", 1)


@pytest.mark.parametrize("kind", ["inf", "nan", "huge", "all-nan", "one-point"])
def test_positions_without_a_place_in_the_grid(faults, kind):
    """Positions that are not finite, span more than a float, or none at all: the order changes nothing."""
    w, h = 300, 200
    mesh = _grid(150, 5, False)
    mesh.pos = mesh.pos.copy()
    rng = np.random.default_rng(6)
    some = rng.choice(len(mesh.pos), len(mesh.pos) // 20, replace=False)
    at = (some, rng.integers(0, 3, len(some)))
    if kind == "inf":
        mesh.pos[at] = rng.choice([np.inf, -np.inf], len(some))
    elif kind == "nan":
        mesh.pos[at] = np.nan
    elif kind == "huge":
        mesh.pos[at] = rng.choice([3.4e38, -3.4e38, 1e-42], len(some))
    elif kind == "all-nan":
        mesh.pos[:] = np.nan
    else:
        mesh.pos[:] = mesh.pos[7]
    sd = U.shader_data((0.4, 1.3, 1.9), w, h)
    got = _draw(faults, mesh, scenes.GROUND, sd, w, h)
    exp = _oracle(mesh, scenes.GROUND, sd, w, h)
    assert (exp["prim"] > 0).any() == (kind in ("inf", "nan", "huge"))
    golden_io.assert_pass(got, exp, "main", kind, 1)
    faults.set_fault_injection(faults.FAULT_UPLOAD_SCRATCH, 0)
    _equal(got, _draw(faults, mesh, scenes.GROUND, sd, w, h))
