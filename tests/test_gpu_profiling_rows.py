"""GPU: with profiling on, each stage of a sequence has a time of its own, and the picture is the same."""
import numpy as np
import pytest

from hsr import frame as hframe
from hsr import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture
def profiled(gpu):
    yield gpu
    gpu.set_profiling(False)


@pytest.mark.parametrize("size", [(100, 80), (1300, 900)])
def test_every_stage_that_ran_has_a_time(profiled, size):
    """A frame over a ground plane: clipped faces, and triangles of many tiles."""
    w, h = size
    fr = scenes.displaced_frame(4, w, h, shadow=256, tex_size=64, seed=3)
    g = hframe.GpuFrame(fr)
    try:
        profiled.set_profiling(False)
        g.render(batched=True)
        plain, t0 = g.download(), profiled.last_timing()
        profiled.set_profiling(True)
        g.render(batched=True)
        got, t = g.download(), profiled.last_timing()
    finally:
        g.release()
    assert t["clipped_faces"] > 0 and t["split_triangles"] > 0
    assert t["launches"] == t0["launches"] + 2
    ms = t["kernel_ms"]
    assert all(ms[k] > 0 for k in ("cull", "emit", "clip", "split", "scan", "scatter", "raster")), ms
    for k in ("records", "bin_pairs", "clipped_faces", "split_triangles", "shaded_pixels", "fragments", "payload_bytes"):
        assert t[k] == t0[k], k
    for k in got:
        for p in ("color", "depth", "prim"):
            assert np.array_equal(got[k][p], plain[k][p]), (k, p)
