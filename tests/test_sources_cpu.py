"""What the kernels' sources keep to, read as text; no GPU."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "matchattention_b200", "csrc")


def test_chained_kernels_read_by_ordinary_loads():
    """A kernel that begins with chain_begin() is set up while the one before it ends: what it reads is not constant over its
    life, which the non-coherent loads take for granted (and the compiler, of parameters that are const __restrict__)."""
    chained = 0
    for path in glob.glob(os.path.join(CSRC, "*.cu*")) + glob.glob(os.path.join(CSRC, "*.inl")):
        code = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)
        kernels = re.findall(r"__global__(.*?)\{\s*chain_begin\(\);", code, flags=re.S)
        if not kernels:
            continue
        assert re.findall(r"__ldg\w*\s*\(|ld\.global\.nc[\w.:]*", code) == [], path
        for head in kernels:
            assert re.findall(r"const\s+\w+\s*\*\s*__restrict__\s*\w+", head) == [], path
        chained += len(kernels)
    assert chained >= 19
