"""Every device wait of the Z build is bounded, and by a second: set-up of a job
in any mode goes through these waits, and a limit of a few time slices could
run out while the GPU works for another process."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sodabayes_gb300", "csrc")


def _text(name):
    return open(os.path.join(CSRC, name)).read()


def test_the_waits_of_the_z_build_take_the_long_limit():
    limit = re.search(r"constexpr uint64_t BUILD_WAIT_NS = (\d+)ull;", _text("tc.cuh"))
    assert limit and 1e9 <= int(limit.group(1)) <= 2e9
    for name, waits in (("gram_tc.cuh", 4), ("chol_tc.cuh", 5)):
        assert _text(name).count("mbar_wait(") == waits
        assert _text(name).count("tc::BUILD_WAIT_NS)") == waits
        assert "mbar_try_wait" not in _text(name)
