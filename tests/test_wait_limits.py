"""The default limits of the bounded device waits."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hana-softwarerenderer_gb300", "csrc")


def _src(f):
    return open(os.path.join(CSRC, f)).read()


def test_a_dependency_wait_lasts_a_second_before_it_gives_up():
    """hsr.h documents about one second; a slow shadow pass within it must not be refused."""
    s = _src("hsr_internal.h")
    ns = int(re.search(r"constexpr int kPollNs = (\d+);", s).group(1))
    polls = 1 << int(re.search(r"constexpr long kDepWaitPolls = 1L << (\d+);", s).group(1))
    assert polls * ns >= 1e9
    for f in ("kernels_raster.cu", "kernels_bin.cu"):
        assert set(re.findall(r"__nanosleep\(([^)]*)\)", _src(f))) == {"kPollNs"}


def test_splitters_show_themselves_whatever_the_size_of_a_triangle():
    """The scan's wait for the splitters counts from their last sign.  With many triangles queued a warp
    takes each alone, up to 2^26 / 32 steps of it, so the sign cannot wait for the triangle's end: each
    loop over its tiles or sub-records gives one every kStepsToBeat steps."""
    s = _src("kernels_bin.cu")
    body = re.search(r"void split_triangle\(.*?\n}\n", s, re.S).group(0)
    loops = re.findall(r"for \(int \w+ = i0;[^\n]*", body)
    assert len(loops) == 3 and all("beat())" in lp for lp in loops), loops
    steps = int(re.search(r"kStepsToBeat = (\d+);", s).group(1))
    ns = int(re.search(r"constexpr int kPollNs = (\d+);", _src("hsr_internal.h")).group(1))
    polls = 1 << int(re.search(r"constexpr long kScanWaitPolls = 1L << (\d+);", _src("hsr_internal.h")).group(1))
    assert steps & (steps - 1) == 0 and polls * ns >= 100e3 * steps  # 100 us a step (an atomic or a 64-byte store)
    assert re.search(r"s \+ beats != seen", s)


def test_injected_stalls_reach_the_waits_they_are_for():
    """A withheld report, not another wait in its place: of a finished tile to the next draw into its target,
    and of the splitters to the scan."""
    r, b = _src("kernels_raster.cu"), _src("kernels_bin.cu")
    body = re.search(r"void wait_tile\(.*?\n}\n", r, re.S).group(0)
    assert "faults" not in body and "wait_at_least(sc, &sc.tile_fill[t], kTileDone)" in body
    assert re.search(r"!\(sc\.faults & HSR_FAULT_DEPENDENCY_STALL\)\)\s*atomicExch\(&sc\.tile_fill\[t\], kTileDone\)", r)
    assert re.search(r"!\(sc\.faults & HSR_FAULT_SCAN_STALL\)\) \{[^}]*atomicAdd\(split_done", b)
