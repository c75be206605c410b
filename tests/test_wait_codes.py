"""Every wait of the tensor-core kernel that can run out has a code, and every code a name."""
import os
import re

from conftest import ROOT
from tennis_b200 import _lib


def test_every_wait_code_has_a_name_of_its_own():
    kernel = open(os.path.join(ROOT, "tennis_b200", "csrc", "conv_tc_kernel.cuh")).read()
    codes = sorted({int(c) for c in re.findall(r"atomicExch\(kp\.status, (\d+)\)", kernel)})
    assert codes == list(range(1, len(codes) + 1))
    lib = _lib.load()
    names = set()
    for code in codes:
        assert lib.tsb_conv2d_i8_status_decode(code) == _lib.ERR_DEVICE_TIMEOUT
        names.add(re.search(r"bounded wait %d \((.*)\);" % code, lib.tsb_last_error().decode()).group(1))
    assert "unknown wait" not in names and len(names) == len(codes)
    header = open(os.path.join(ROOT, "include", "tennis_b200.h")).read()
    assert "(1..%d, which wait)" % codes[-1] in header
