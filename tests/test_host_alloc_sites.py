"""CPU test: device memory of calls comes from the block cache, whose allocations find idle blocks'
memory on a full device; what is left are blocks made once and kept (Boys table, fault word) and the
rate probes' 32 KB."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gbasis_b200", "csrc")
DIRECT = {"pools.cu": 2, "runtime.cu": 2, "extras.cu": 2}


def test_calls_allocate_through_the_block_cache():
    found = {}
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        with open(path) as f:
            code = re.sub(r'//[^\n]*|"[^"\n]*"', "", f.read())
        n = len(re.findall(r"\bcudaMalloc(?:Async)?\(", code))
        if n:
            found[os.path.basename(path)] = n
    assert found == DIRECT
