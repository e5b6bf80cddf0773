"""Checks of the kernel sources and of the build that need no GPU."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "baylorlqcd_b200" / "csrc"


def reads_after_stores(text):
    """Spinor fields that a block of code loads after storing them: (field, offset)."""
    text = re.sub(r"//[^\n]*", lambda m: " " * len(m.group()), text)
    found = []
    for st in re.finditer(r"IO(?:<\w+>)?::store\w*\(\s*([\w.\[\]]+)\.data\s*,", text):
        depth, end = 0, st.end()
        while end < len(text) and depth >= 0:  # to the end of the block that stores
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        if re.search(r"IO(?:<\w+>)?::load\(\s*%s\.data\s*," % re.escape(st.group(1)), text[st.end():end]):
            found.append((st.group(1), st.start()))
    return found


def test_no_kernel_loads_a_spinor_it_has_stored():
    """SpinorIO::load is __ldg, which is undefined for memory that the kernel writes: the
    load may return what was there before the store.  Sums over stored 16-bit values take
    them from store_rounded instead."""
    bad = "IO::store(A.r.data, A.r.norm, n, s, c);\n if (q) IO::load(A.r.data, A.r.norm, n, s, c);"
    assert reads_after_stores("{" + bad + "}") and not reads_after_stores("{ IO::store(A.r.data, c); } IO::load(A.r.data, c);")
    found = {f.name: reads_after_stores(f.read_text()) for f in CSRC.iterdir() if f.suffix in (".cu", ".cuh")}
    assert not {k: v for k, v in found.items() if v}
