"""The staged bulk kernel's instances fit their register budget: the build log
lists none that spills (the ragged parity-1 ones did, for code that ragged rows
never reach)."""
import re
from pathlib import Path

import pytest

LOG = Path(__file__).resolve().parents[1] / "simlab_b200" / "_build" / "build.log"


def test_no_staged_bulk_kernel_spills():
    if not LOG.exists():
        pytest.skip("built elsewhere: no build log")
    found = re.findall(r"Function properties for (\S*k_bulk_tma\S*)\n.*?(\d+) bytes spill stores, (\d+) bytes spill loads", LOG.read_text())
    assert found
    assert [f for f in found if f[1:] != ("0", "0")] == []
