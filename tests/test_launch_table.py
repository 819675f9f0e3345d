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


def test_every_device_is_asked_for_once(tmp_path):
    """Occupancy and kernel attributes are per device: a second device of the
    process is looked up (and its attribute set) like the first, once per
    shape; a failed lookup is tried again."""
    out = _run(tmp_path, """
    static LaunchTable t;
    int asked = 0, b = 0;
    const auto query = [&](int n, int status) { return [&asked, n, status](int* fits) { ++asked; *fits = n; return status; }; };
    const auto get = [&](int dev, int shape, int n, int status) {
        const int s = t.blocks(dev, shape, 128u, query(n, status), &b);
        std::printf("%d,%d,%d ", s, s ? -1 : b, asked);
    };
    get(0, 2, 5, 0); get(0, 2, 9, 0);                    // one lookup
    get(1, 2, 7, 0); get(1, 2, 9, 0); get(0, 2, 9, 0);   // the second device has its own
    get(0, 3, 6, 0); get(1, 3, 8, 0);                    // and its own per shape
    get(2, 0, 4, 3); get(2, 0, 4, 0); get(2, 0, 9, 0);   // an error is not kept
    get(63, 5, 30, 0); get(64, 5, 4, 0); get(64, 5, 3, 0);  // clamped; past the table: asked each time
    """)
    assert out == ["0,5,1", "0,5,1", "0,7,2", "0,7,2", "0,5,2", "0,6,3", "0,8,4", "3,-1,5", "0,4,6", "0,4,6",
                   "0,12,7", "0,4,8", "0,3,9"]
