"""Every device and pinned-host allocation of the library goes through
memory.cu, where the allocation hook, the guard regions and tcs_alloc_stats see
it; the CUDA allocation calls are named nowhere else in its sources."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tcstencil_gb300", "csrc")
CALLS = re.compile(r"\bcuda(Malloc\w*|HostAlloc|HostRegister)\s*\(")


def test_allocations_are_made_in_one_file():
    found = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*"))):
        with open(path) as f:
            code = re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)
        if CALLS.search(code):
            found[os.path.basename(path)] = [m.group(0) for m in CALLS.finditer(code)]
    assert set(found) == {"memory.cu"}, found
