"""The DRAM traffic in the bench's roofline is that of the kernel the bench
ran: the tile kernel's figure is the one of its own capture."""
import re

import bench


def test_traffic_of_the_kernel_that_runs():
    assert bench.step_kernel(512, "rusanov") == "vert_tile_kernel"
    assert bench.step_kernel(256, "rusanov") == bench.step_kernel(384, "ausm") == "vert_step_kernel"
    text = open(bench.os.path.join(bench.ROOT, "profiles", "vert_step_kernel_globe1deg.md")).read()
    current = text[:text.index("## Earlier builds")]
    m = re.search(r"\| DRAM \| ([0-9.]+) MB read, ([0-9.]+) MB written per launch", current)
    cols = int(re.search(r"with ([0-9,]+) columns", current).group(1).replace(",", ""))
    want = 1e6 * (float(m.group(1)) + float(m.group(2))) / cols
    assert abs(bench.profile_traffic("vert_tile_kernel") / want - 1.0) < 1e-3
