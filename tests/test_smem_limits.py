"""A kernel's limit of dynamic shared memory belongs to the function on the device, whichever thread
or context launches it: it is set in one place only, to a size known at compile time."""
import glob
import os
import re

from conftest import ROOT


def test_limits_are_compile_time_constants():
    calls = {}
    for path in glob.glob(os.path.join(ROOT, "pasqual_gb300", "csrc", "*.cu*")):
        calls[os.path.basename(path)] = len(re.findall(r"cuda(?:FuncSetAttribute|FuncAttributeMaxDynamicSharedMemorySize)",
                                                       open(path).read()))
    # the one call of allow_smem, whose size is a template argument
    assert {k: n for k, n in calls.items() if n} == {"pq_common.cuh": 2}
