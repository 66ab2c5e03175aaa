"""What ptxas reports for kernels whose registers are left to it on purpose (built here by the Makefile)."""
import re

import pytest

from conftest import ROOT


def test_staged_reference_rounding_does_not_spill():
    log = ROOT / "p2z-tests_b200" / "_build" / "p2z_kern_v2_ref.ptxas.txt"
    if not log.exists():
        pytest.skip("no build log here")
    spills = re.findall(r"Compiling entry function '\S*k_staged\S*'.*\n.*\n.*?(\d+) bytes spill stores", log.read_text())
    assert len(spills) == 2 and set(spills) == {"0"}
