"""Resident blocks of the persistent kernels (csrc/launch_table.h), host-only:
the header is compiled into a small program and run without a GPU."""
import importlib
import os
import subprocess

import pytest

build = importlib.import_module("sol-rs_gb300.build")


def _run(tmp_path, body):
    src = tmp_path / "t.cpp"
    src.write_text('#include "launch_table.h"\n#include <cstdio>\nusing namespace solrt;\nint main() {\n%s\n}\n' % body)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", build.CSRC, str(src), "-o", exe], check=True)
    return subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()


@pytest.mark.parametrize("block", [64, 128, 256])
def test_no_more_threads_than_the_deep_stack_has(tmp_path, block):
    out = _run(tmp_path, 'for (int f : {0, 1, 5, 6, 7, 12, 13, 24, 25, 32}) std::printf("%%d ", resident_blocks(f, %du));' % block)
    assert [int(x) for x in out] == [min(max(f, 1), 1536 // block) for f in (0, 1, 5, 6, 7, 12, 13, 24, 25, 32)]


def test_cooperative_kernel_with_more_threads_is_refused(tmp_path):
    """A build that asks for more resident threads per SM than the contexts'
    traversal stacks are for does not compile."""
    r = subprocess.run([build.nvcc()] + build.ARCH + ["-std=c++17", "--expt-relaxed-constexpr", "-DSOLRT_COOP_MINB=13",
                       "-x", "cu", "-c", os.path.join(build.CSRC, "coop.cu"), "-o", str(tmp_path / "coop.o")],
                       capture_output=True, text=True)
    assert r.returncode != 0 and "traversal stacks" in r.stderr
