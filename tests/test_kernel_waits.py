"""Rules on the waits in the kernels' source (no GPU needed)."""
import re

import pytest

from allie_b200 import build

KERNELS = sorted(build.CSRC.glob("*.cu")) + sorted(build.CSRC.glob("*.cuh"))


@pytest.mark.parametrize("path", KERNELS, ids=lambda p: p.name)
def test_warps_that_use_tmem_leave_together(path):
    """TMEM instructions are a whole warp's: where a bounded wait runs out, all lanes get the same verdict, or some would
    leave and the others meet an instruction that waits for them without a limit."""
    code = re.sub(r"//[^\n]*", "", path.read_text())
    if path.name == "ptx.cuh" or not re.search(r"\btmem_(ld|st|alloc)", code):
        pytest.skip("no TMEM here")
    assert not re.findall(r"\bmbar_wait\(", code)
