"""The tile counters of the tensor-core engine belong to the caller of a launch.

A launch trusts that its two counters are zero and leaves them so.  Counters that launches of two
streams share can be left at other values for good, and later launches then skip or repeat tiles, so
no counter may be process-wide: each context has its own, cleared once a step.
"""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "pulsesuite_gb300" / "csrc"


def test_no_process_wide_counters():
    engine = (CSRC / "tc_engine.cu").read_text()
    assert not re.search(r"^(?:static\s+|__device__\s+)+(?:unsigned|int|long long)\s*\**\s*\w+\s*(?:=[^()]*)?;",
                         engine, re.M)
    assert "L.sched = sched;" in engine


def test_counters_are_cleared_once_a_step():
    tc = (CSRC / "sbe_tc.cu").read_text()
    prep = tc[tc.index("static int mixed_prep("):]
    prep = prep[:prep.index("\n}\n")]
    take = re.search(r"A->mx = k\.take<unsigned>\((.*)\);", tc).group(1)
    clear = re.search(r"cudaMemsetAsync\(A->mx, 0, sizeof\(unsigned\) \* \((.*)\), s\);", prep).group(1)
    assert take == clear and take.endswith("+ 2")
