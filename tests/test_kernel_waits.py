"""Rules on the waits in the kernels' source (no GPU needed)."""
import re

import pytest

from allie_b200 import build


def _code(path) -> str:
    return re.sub(r"//[^\n]*", "", path.read_text())


KERNELS = [p for p in sorted(build.CSRC.glob("*.cu*")) if re.search(r"\btmem_(ld|st)\d", _code(p)) and p.name != "ptx.cuh"]


@pytest.mark.parametrize("path", KERNELS, ids=lambda p: p.name)
def test_warps_that_use_tmem_leave_together(path):
    """TMEM instructions are a whole warp's: where a bounded wait runs out, all lanes get the same verdict, or some would
    leave and the others meet an instruction that waits for them without a limit."""
    assert not re.findall(r"\bmbar_wait\(", _code(path))
