"""Launch attributes belong to a device: no launch may remember in a process-wide flag
that it has set one (a context on a second device would go without)."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "tileink_b200" / "csrc"


@pytest.mark.parametrize("name", sorted(p.name for p in CSRC.glob("*.cu")))
def test_no_process_wide_launch_flag(name):
    assert not re.search(r"^\s*static\s+(bool|int|std::once_flag)\b[^(]*(=|;)", (CSRC / name).read_text(), re.M)
