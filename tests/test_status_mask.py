"""Every entry point that reads the device status word treats every fatal bit as an error (read from
the source: a wait that expires cannot be provoked in a tensor-core kernel without copies in flight).
"""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_status_checks_use_all_fatal_bits():
    hdr = open(os.path.join(ROOT, "include", "qkgw.h")).read()
    fatal = set(re.findall(r"(QKD_\w+) = \d+,?\s*/\*[^*]*\(fatal\)", hdr))
    assert fatal == {"QKD_BARRIER_TIMEOUT", "QKD_BAD_INDEX", "QKD_MBAR_TIMEOUT"}
    src = "\n".join(open(f).read() for f in glob.glob(os.path.join(ROOT, "quack_gb300", "csrc", "*.cu*")))
    mask = re.search(r"constexpr int QK_FATAL = ([^;]*);", src).group(1)
    assert set(re.findall(r"QKD_\w+", mask)) == fatal
    calls = re.findall(r"qk_status_check\(\w+, ([^;]*)\);", src)
    assert len(calls) >= 3 and all(c in ("QK_FATAL", "int fatal_mask") for c in calls), calls
