"""Device memory of the library is taken through dev_malloc and given back
through dev_free (csrc/ctx.cu), which hand idle blocks back where the device has
run out: no source file calls cudaMalloc or cudaFree past them."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "verb-4d_b200", "csrc")


def code(path):
    return re.sub(r"//[^\n]*", "", open(path).read())


def test_one_way_to_device_memory():
    calls = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = code(path)
        if os.path.basename(path) == "ctx.cu":
            # the two functions and the blocks beside them end where alloc() begins
            text = text[text.index("int alloc(void** p, size_t bytes)"):]
        found = re.findall(r"\bcuda(?:Malloc|Free)\s*\(", text)
        if found:
            calls[os.path.basename(path)] = len(found)
    assert not calls
