"""The persistent batch writes the row records and reads them in one launch, where the read-only path (__ldg) is not
defined; checked on the source, since a stale record cannot be provoked."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fluidisim_b200", "csrc")


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_the_batch_reads_its_own_records_with_plain_loads():
    calls = re.findall(r"(?<!\w)row_general(<\w+>)?\(", source("fd3_batch.cuh"))
    assert calls and set(calls) == {"<true>"}
    fast = source("fd3_fast.cuh")
    row = fast[fast.index("float row_general("):fast.index("const bool unit", fast.index("float row_general("))]
    loads = re.findall(r"(SAME_LAUNCH \? \*\w+ : )?__ldg", row)
    assert loads and all(loads)


def test_the_batch_itself_uses_no_read_only_load():
    assert "__ldg" not in source("fd3_batch.cuh")
