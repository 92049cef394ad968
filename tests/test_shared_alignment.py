"""Dynamic shared memory that a kernel reads in 8 or 16 bytes starts where such an access may: it is
declared with that alignment (its element type promises 4 bytes) or rounded up by the kernel."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "symmetrix_gb300", "csrc")


def test_dynamic_shared_memory_is_aligned():
    seen = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        with open(path) as f:
            text = f.read()
        for m in re.finditer(r"extern __shared__ (.*?)(\w+)\[\]", text):
            seen += 1
            kind, name = m.group(1), m.group(2)
            rounded = f"reinterpret_cast<uintptr_t>({name}) + 1023) & ~uintptr_t(1023)" in text
            own_type = kind.strip() == "int" and not re.search(rf"reinterpret_cast<\w+\*>\({name}", text)
            assert "__align__(16)" in kind or rounded or own_type, (os.path.basename(path), m.group(0))
    assert seen >= 5
