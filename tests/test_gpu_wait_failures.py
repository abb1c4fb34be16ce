"""GPU: the bounded waits between draws into one target and between the scan and the blocks that split large
triangles run out with a status and leave the device usable.

As in test_gpu_failures, nothing is faulted or hung: the host lowers the poll limit and has the report that
the wait is for withheld (hsr_set_fault_injection); the kernel gives up, the call returns
HSR_ERR_TIMEOUT, and the next draw on the same context is exact."""
import time

import numpy as np
import pytest

import golden_io
import oracle
from hsr import scenes
from hsr import uniforms as U

pytestmark = pytest.mark.gpu
CLEAR = ((0, 0, 0, 255), 1.0)


@pytest.fixture
def faults(gpu):
    old = gpu.get_tuning()
    yield gpu
    gpu.set_fault_injection(0, 0)
    gpu.set_tuning(tile=old.tile, warps_per_cta=old.warps_per_cta, ctas_per_sm=old.ctas_per_sm)


def _times_out(gpu, descs, fault):
    gpu.set_fault_injection(fault, 4000)
    t0 = time.perf_counter()
    with pytest.raises(gpu.HsrError) as e:
        gpu.draw_batch(descs)
    assert e.value.code == gpu.ERR_TIMEOUT
    assert time.perf_counter() - t0 < 10.0
    gpu.set_fault_injection(0, 0)


# one CTA per SM: a warp per tile, eight: a CTA per tile
@pytest.mark.parametrize("ctas", [1, 8])
def test_wait_for_an_earlier_draws_tile_runs_out_and_the_next_draw_is_exact(faults, ctas):
    gpu = faults
    gpu.set_tuning(tile=8, warps_per_cta=4, ctas_per_sm=ctas)
    w, h = 500, 300
    fr = [scenes.sphere_frame(3, w, h, shader=scenes.BLINN, tex_size=16, seed=k, eye=(0.3 * k, 0.2, 2.5)) for k in range(2)]
    main = gpu.Target(w, h)
    held = [main] + [gpu.Mesh(f.mesh) for f in fr] + [gpu.Texture(f.diffuse) for f in fr]
    try:
        descs = [gpu.make_desc(held[1 + k], scenes.BLINN, f.sd, main, held[3 + k], prim_base=5000 * k,
                               clear=CLEAR if k == 0 else None) for k, f in enumerate(fr)]
        _times_out(gpu, descs, gpu.FAULT_DEPENDENCY_STALL)
        gpu.draw_batch(descs)
        got = main.download()
    finally:
        for o in reversed(held):
            o.release()
    rb = oracle.Buffers(w, h, *CLEAR)
    for k, f in enumerate(fr):
        oracle.draw(f.mesh, scenes.BLINN, f.sd, rb, f.diffuse, prim_base=5000 * k)
    golden_io.assert_pass(got, {"depth": rb.depth, "color": rb.color, "prim": rb.prim}, "main", "after a tile timeout", 1)


def test_wait_for_the_splitters_runs_out_and_no_target_is_written(faults):
    gpu = faults
    gpu.set_tuning(tile=8, warps_per_cta=4, ctas_per_sm=8)
    w, h, n = 700, 500, 40
    rng = np.random.default_rng(4)
    ang = rng.uniform(0, 2 * np.pi, (n, 1)) + np.arange(3) * (2 * np.pi / 3)
    pos = np.empty((n, 3, 3), np.float32)
    pos[:, :, 0], pos[:, :, 1] = 0.9 * np.cos(ang), 0.9 * np.sin(ang)
    pos[:, :, 2] = rng.uniform(-0.9, 0.9, (n, 1))
    faces = np.zeros((n, 3, 3), np.int32)
    faces[:, :, 0] = np.arange(3 * n, dtype=np.int32).reshape(n, 3)
    mesh = scenes.Mesh(pos.reshape(-1, 3), np.array([[0, 0, 1]], np.float32), np.zeros((1, 2), np.float32), faces)
    sd = U.shader_data((0, 0, 1), w, h, identity_mvp=True)
    main, gm = gpu.Target(w, h), gpu.Mesh(mesh)
    try:
        descs = [gpu.make_desc(gm, scenes.FLAT, sd, main, clear=CLEAR)]
        main.clear((7, 7, 7, 7), 0.5)
        before = main.download()
        _times_out(gpu, descs, gpu.FAULT_SCAN_STALL)
        after = main.download()
        for p in ("color", "depth", "prim"):
            assert np.array_equal(before[p], after[p]), p  # the stalled sequence drew nothing
        gpu.draw_batch(descs)
        assert gpu.last_timing()["split_triangles"] == n
        got = main.download()
    finally:
        gm.release()
        main.release()
    rb = oracle.Buffers(w, h, *CLEAR)
    oracle.draw(mesh, scenes.FLAT, sd, rb)
    golden_io.assert_pass(got, {"depth": rb.depth, "color": rb.color, "prim": rb.prim}, "main", "after a split timeout", 1)
