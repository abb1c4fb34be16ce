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
