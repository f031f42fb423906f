"""Kernel attributes (cudaFuncSetAttribute) belong to the device that is current, so
nothing that is set or asked once may be remembered for the whole process: a handle on
another device would launch without its shared memory.  The sources keep such things
in a context of a handle or in a table indexed by the device.  (A process with two
devices cannot be had where these tests run; the sources are read instead.)"""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mnpbem_gb300", "csrc")
FLAG = re.compile(r"^\s+static\s+(?:bool|int|unsigned|size_t)\s+\w+\s*(?:=[^;]*)?;", re.M)


def sources():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, name)) as f:
                yield name, f.read()


def test_no_process_wide_device_state():
    bad = [(name, m.group(0).strip()) for name, text in sources() for m in FLAG.finditer(text)]
    assert not bad, bad

