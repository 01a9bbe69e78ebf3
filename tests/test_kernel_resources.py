"""Registers and spills of the built kernels, from the compiler's report that
build.py keeps beside each object."""
import os
import re

import pytest

from conftest import PKG_DIR


def kernels(source):
    """[(mangled name, registers, bytes of spill stores)] of one source."""
    path = os.path.join(PKG_DIR, "_build", source + ".ptxas")
    if not os.path.exists(path):
        pytest.skip("no compiler report: the objects were built elsewhere")
    return re.findall(r"Function properties for (\S+)\n.*?(\d+) bytes spill stores.*?\n.*?Used (\d+) registers",
                      open(path).read())


def test_monte_carlo_kernels_of_512_threads_hardly_spill():
    """One 512-thread CTA runs on an SM, so a Monte Carlo kernel may use 128
    registers; bounded to 64 they spilled 576-1,120 bytes a thread.  (The
    1,024-thread ones and those that share an SM have 64 and trade their spills for
    warps.)"""
    found = {(k, n): int(s) for n, s, _ in kernels("mc.cu")
             for k in re.findall(r"(mc_kernel(?=I[fd]Li512ELi\d+ELi1E)|mc_spec_kernel(?=I[fd]Li512E))", n)}
    assert {k for k, _ in found} == {"mc_kernel", "mc_spec_kernel"} and len(found) == 20
    assert max(found.values()) <= 128, found
