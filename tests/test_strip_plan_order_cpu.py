"""A strip plan's first replay must find its last-block ticket zeroed.  The
context's stream is non-blocking, so nothing that is queued on the legacy
stream (cudaMemset without a stream, which does not wait for the device
either) comes before its launches: whatever a kernel relies on is zeroed on a
stream that the launch follows."""
import glob
import os
import re

from conftest import ROOT


def test_no_memset_on_the_legacy_stream():
    for path in glob.glob(os.path.join(ROOT, "openferric_b200", "csrc", "*.cu*")):
        code = re.sub(r"//.*", "", open(path).read())
        assert not re.search(r"\bcudaMemset\s*\(", code), path
