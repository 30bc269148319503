"""The convolution kernel's trace build, its C declaration and the script that reads it agree on the size of the
buffer that is copied out."""
import os
import re

from conftest import ROOT, pkg


def _source(*path):
    with open(os.path.join(ROOT, *path)) as f:
        return f.read()


def test_reader_and_kernel_agree_on_the_buffer():
    kernel = _source("mini-caffe_b200", "csrc", "kernels", "conv_tc.cu")
    slots = int(re.search(r"kTraceSlots = (\d+);", kernel).group(1))
    roles = int(re.search(r"kTraceRoles = (\d+);", kernel).group(1))
    reader = pkg("conv_trace")
    assert (reader.ROLES, reader.SLOTS) == (roles, slots)
    header = _source("include", "mcb200_runtime.h")
    assert re.search(r"Copies (\d+) x (\d+) values", header).groups() == (str(roles), str(slots))
    stamped = {int(r) for r in re.findall(r"MCB200_TRACE\((\d)\);", kernel)}
    assert stamped and max(stamped) < roles and "g_conv_trace[4 * kTraceSlots" in kernel
