"""No flag of the library outlives the object it is about.  A launch attribute is set for the current device, and
several threads may each use a context of their own, so a process-wide "already done" flag is wrong on the second
device and a race between threads.  Read from the sources: the second device is not here."""
import glob
import os
import re

from conftest import ROOT

SOURCES = sorted(glob.glob(os.path.join(ROOT, "fmma_b200", "csrc", "*.cu*")))


def test_no_launch_attribute_behind_a_process_wide_flag():
    found = [f"{os.path.basename(p)}:{i}: {line.strip()}" for p in SOURCES for i, line in enumerate(open(p), 1)
             if re.search(r"^\s+static\s+bool\b", line)]
    assert SOURCES and not found, found


def test_shared_tables_are_not_filled_behind_a_flag():
    # tables made on first use are constants (initialised once for all threads), not arrays with an "is filled" flag
    found = [f"{os.path.basename(p)}:{i}: {line.strip()}" for p in SOURCES for i, line in enumerate(open(p), 1)
             if re.search(r"^static\s+(bool|int)\s+\w+(\[[^]]*\])?\s*(=|;)", line)]
    assert not found, found
