"""Opt-ins for large shared memory hold per device, not per process.

cudaFuncSetAttribute acts on the current device's context, so a launcher that
remembers in a process-wide flag that it has opted in leaves a kernel without its
shared memory on the next device.  With one device that shows only in the source:
no kernel file keeps such a flag."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "letzelphc_gb300", "csrc")


def test_no_launcher_remembers_its_opt_in():
    files = sorted(glob.glob(os.path.join(CSRC, "*.cu*")))
    assert files
    for f in files:
        with open(f) as fh:
            src = fh.read()
        for m in re.finditer(r"^[ \t]+static bool (\w+)[ \t]*=", src, re.M):
            assert "cudaFuncSetAttribute" not in src[m.start():m.start() + 600], (os.path.basename(f), m.group(1))
