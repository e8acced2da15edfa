"""What the compiler reports for the counting traversals: their launch bounds leave them enough registers."""
import re

import pytest

from dumbray_gb300 import build


@pytest.mark.parametrize("kernel", ["k_cast", "k_trace", "k_shadow_phys"])
def test_counting_traversals_do_not_spill(kernel):
    log = build.OUT / "ptxas.log"
    if not log.exists():
        pytest.skip("no build log")
    found = re.findall(r"Function properties for (\S*" + kernel + r"ILb1E\S*)\n.*?(\d+) bytes spill stores, (\d+) bytes spill loads", log.read_text())
    assert found
    assert all(int(stores) == int(loads) == 0 for _, stores, loads in found), found
