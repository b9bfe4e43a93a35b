"""Scans, compactions, sorts and the one-block level pass take scratch or opt
into shared memory, and say so when they cannot run.  A call that went on all
the same would read counts and levels that nobody wrote, and return a wrong
graph: every caller has to use the result (CPU, by reading the sources)."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "culs_b200" / "csrc"
CALLS = r"(?:compact_flags|scan_exclusive|radix_sort_pairs|levels_block)\("


@pytest.mark.parametrize("path", sorted(CSRC.glob("*.cu")), ids=lambda p: p.name)
def test_no_caller_drops_a_result(path):
    dropped = [line.strip() for line in path.read_text().splitlines() if re.match(rf"\s*(?:(?:X\.)?check\()?{CALLS}", line)]
    assert not dropped
