"""The kernels of a launch sequence are resident while the kernel before them still writes (hsr_launch.cuh),
so they may read what it writes by ordinary loads alone: read-only loads (__ldg, and what the compiler
makes of a const __restrict__ parameter) are defined only for memory that nobody writes meanwhile."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hana-softwarerenderer_gb300", "csrc")
SRC = {os.path.basename(f): open(f).read() for f in glob.glob(os.path.join(CSRC, "*.cu*"))}
# written before a sequence begins, by launches that it follows in stream order
STATIC = {"px", "py", "pz", "p4", "n4", "fv", "fvt", "fvn", "pk", "uv", "tex"}


def _chained():
    return {m for s in SRC.values() for m in re.findall(r"launch_chained\((k_\w+)", s)}


def test_chained_kernels_take_no_restricted_pointers():
    chained, found = _chained(), set()
    assert {"k_setup", "k_scan", "k_raster"} <= chained
    for name, s in SRC.items():
        for kernel, params in re.findall(r"__global__ void __launch_bounds__\([^{;]*?\)\s*(k_\w+)\(([^{;]*?)\)\s*\{", s):
            if kernel in chained:
                found.add(kernel)
                assert "__restrict__" not in params, (name, kernel)
        # nor the functions inlined into them
        assert not re.search(r"DView\* __restrict__", s), name
    assert found == chained


def test_read_only_loads_are_of_meshes_and_textures():
    for name in ("kernels_geom.cu", "kernels_bin.cu", "kernels_raster.cu", "hsr_device.cuh"):
        for at in re.findall(r"__ldg\(([^()]*(?:\[[^\]]*\])?)", SRC[name]):
            assert set(re.findall(r"\w+", at)) & STATIC and "sv" not in re.findall(r"\w+", at), (name, at)


def test_emit_leaves_on_an_overflow_as_one_block():
    """Clipping blocks set the error word while emitting blocks of the same grid begin; those add up
    their warps' sums behind a barrier, so their warps must not part over it."""
    body = re.search(r"k_emit\(const DView\* views.*?\n}\n", SRC["kernels_geom.cu"], re.S).group(0)
    assert re.search(r"if \(__syncthreads_or\(\(sc\.ctl->error & kErrCapacity\) != 0u\)\) return;", body)
    assert body.count("ctl->error") == 1
