"""prgpu_kernel_launches counts launches: in the sources each CK_LAUNCH(), which adds one, follows a launch of its own,
and each launch is followed by one (or counted by hand behind a cooperative launch)."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "poissonrecon_gpu_gb300", "csrc")
SOURCES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))


@pytest.mark.parametrize("name", SOURCES)
def test_every_count_has_its_launch(name):
    with open(os.path.join(CSRC, name)) as f:
        text = re.sub(r"//[^\n]*|^#define(?:.*\\\n)*.*", "", f.read(), flags=re.M)
    events = [(m.start(), m.group()) for m in re.finditer(
        r"<<<|cudaLaunchCooperativeKernel\(|CK_LAUNCH\(\)|\+\+(?:::prgpu::)?g_kernel_launches", text)]
    open_launch = None
    for at, what in events:
        line = text.count("\n", 0, at) + 1
        if what == "<<<" or what.startswith("cudaLaunch"):
            # (the two sides of an if share the count behind them)
            if open_launch is not None:
                between = text[open_launch:at]
                assert re.search(r"\belse\b", between), "%s: the launch before line %d is not counted" % (name, line)
            open_launch = at
        else:
            assert open_launch is not None, "%s: about line %d a launch is counted that is not made" % (name, line)
            open_launch = None
    assert open_launch is None, "%s: the last launch is not counted" % name
