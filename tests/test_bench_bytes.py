"""The bytes that the benchmark declares per task and call are the ones the library uploads."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_declared_view_bytes_are_the_table_entry(slsf):
    source = open(os.path.join(ROOT, "slsf-rs_b200", "csrc", "capi.cu")).read()
    asserted = re.search(r"static_assert\(sizeof\(TaskView\) == (\d+)", source)  # the compiler checks this number
    assert int(asserted.group(1)) == slsf.TASK_VIEW_BYTES
    assert "n * pkg.TASK_VIEW_BYTES" in open(os.path.join(ROOT, "bench.py")).read()
