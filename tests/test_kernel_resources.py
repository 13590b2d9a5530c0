"""What the compiler reports of kernels whose speed hangs on it."""
import os
import re
import subprocess

from conftest import PKG


def shared_bytes(source, kernel):
    """Static shared memory of a kernel, from ptxas -v."""
    out = subprocess.run(
        ["nvcc", "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a",
         "-I../include", "-Icsrc", "--expt-relaxed-constexpr", "-Xptxas", "-v", "-cubin",
         "-o", os.devnull, os.path.join("csrc", source)],
        cwd=PKG, check=True, capture_output=True, text=True).stderr
    entry = re.search(r"Compiling entry function '[^']*" + kernel + r"[^']*'.*?Used ([^\n]*)", out,
                      re.S).group(1)
    smem = re.search(r"(\d+) bytes smem", entry)
    return int(smem.group(1)) if smem else 0


def test_long_partner_lists_keep_the_l1():
    """The fill pass sorts long partner lists through L1: its blocks hold the
    unit keys' histogram (three digits) in shared memory and nothing like a
    list per thread."""
    assert shared_bytes("collide.cu", "k_partners_fill") <= 3 * 256 * 4 + 16
