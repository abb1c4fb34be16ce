"""CPU: bench.py's byte model follows the kernels that run."""
import os
import re
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

import bench  # noqa: E402

SOUP = {"faces": 4_000_000, "vertices": 11_880_000, "records": 2_900_000, "bin_pairs": 5_000_000, "pixels": 8_294_400,
        "shaded_pixels": 8_289_000, "clipped_faces": 9_000, "raster_pixels": 8_294_400, "tiles": 32_400,
        "split_triangles": 1_000, "payload_bytes": 0}


def test_no_vertex_pass_where_the_cull_pass_computes_the_screen_vertices():
    kb = bench.kernel_bytes(SOUP)
    assert kb["vertex"] == 0
    assert kb["cull"] == 4_000_000 * 16 + 11_880_000 * 12 + 2_900_000 * 64
    shared = bench.kernel_bytes(dict(SOUP, vertices=2_000_000))
    assert shared["vertex"] == 2_000_000 * 28 and shared["cull"] == 4_000_000 * 16 + 2_000_000 * 16 + 2_900_000 * 64
    assert bench.kernel_bytes(dict(SOUP, faces=1 << 18, vertices=1000))["vertex"] == 0
    src = open(os.path.join(ROOT, "hana-softwarerenderer_gb300", "csrc", "kernels_geom.cu")).read()
    assert "kOwnVertexFaces = (size_t)1 << 18;" in src
    assert re.search(r"return faces <= kOwnVertexFaces \|\| positions >= faces;", src)


def test_emit_writes_no_payload_index():
    assert bench.kernel_bytes(SOUP)["emit"] == 2_900_000 * 48 + 1_450_000 * 32
