"""Checks of the kernel sources and of the build that need no GPU."""
import re
import subprocess
from pathlib import Path

import numpy as np

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


DRIVER = r"""
#include <cstdio>
#include "qq_dense.h"
using namespace qq::dense;
int main() {
  const double scale[3] = {1.0, 1e170, 1e-170};
  for (double f : scale) {
    Mat H(4, 3);
    std::vector<cd> c(4, cd(0, 0)), y, srv;
    c[0] = cd(1, 2);
    for (int j = 0; j < 3; ++j)
      for (int i = 0; i <= j + 1; ++i) H(i, j) = f * cd(1.0 + i + 2 * j, 0.5 * i - j);
    hess_lsq(H, c, 3, y, srv);
    for (const cd& v : y) std::printf("%.17g %.17g\n", f * v.real(), f * v.imag());
  }
}
"""


def host_flags(monkeypatch):
    """The host-compiler options that the build gives each source."""
    from baylorlqcd_b200 import build

    cmds = []

    def record(cmd, **kw):
        cmds.append(cmd)
        return subprocess.CompletedProcess(cmd, 0, "", "")

    monkeypatch.setattr(build.subprocess, "run", record)
    for src in sorted(CSRC.glob("*.cu")):
        build._compile(src, float("inf"))
    monkeypatch.undo()
    return {tuple(b for a, b in zip(c, c[1:]) if a == "-Xcompiler") for c in cmds}


def test_host_code_keeps_its_range_and_its_cpus(monkeypatch, tmp_path):
    """All sources are compiled alike on the host: the shared headers' inline functions
    have one definition, no instruction set beyond the baseline is assumed, and complex
    divisions stay exact to the ends of the exponent range: the least-squares solution of
    f H y = c times f is the same for f = 1, 1e170 and 1e-170 but for rounding (1e-14: some
    hundred operations of 2^-53 on a matrix of condition below 100)."""
    flags = host_flags(monkeypatch)
    src, exe = tmp_path / "driver.cpp", tmp_path / "driver"
    src.write_text(DRIVER)
    for opts in flags:
        subprocess.run(["g++", "-std=c++17", "-I", str(CSRC), *opts, str(src), "-o", str(exe)], check=True)
        y = np.array(subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split(), float)
        y = y.reshape(3, -1)
        assert np.isfinite(y).all() and np.abs(y - y[0]).max() <= 1e-14 * np.abs(y[0]).max()
    assert len(flags) == 1 and not any(o.startswith("-m") for o in next(iter(flags)))
