"""The bounds of look-ahead accesses (csrc/index_bounds.h) at the largest sizes a handle may have: no matrix of that size is
made, the arithmetic the kernels use is compiled for the host and compared with 64-bit sums."""
import os
import re
import subprocess

import pytest

from alsparse_b200 import build

MAIN = r"""
#include <limits.h>
#include <stdio.h>
#include "index_bounds.h"
int main() {
    using namespace asb;
    long long wrong = 0, seen = 0;
    const int most[] = {INT_MAX, INT_MAX - 1, INT_MAX - 32, INT_MAX - 33, INT_MAX - 64, INT_MAX - 65, 1 << 20, 100, 1, 0};
    for (int end : most)
        for (int left = 0; left <= 200 && left <= end; left++)
            for (int ahead = 0; ahead <= 224; ahead++, seen++) {
                const int at = end - left;
                const long long sum = (long long)at + ahead;
                wrong += ahead_inside(at, ahead, end) != (sum < end);
                wrong += ahead_complete(at, ahead, end) != (sum <= end);
                wrong += ahead_or_end(at, ahead, end) != (sum < end ? sum : end);
            }
    printf("%lld of %lld\n", wrong, seen);
    return wrong != 0;
}
"""


def test_bounds_at_the_largest_sizes(tmp_path):
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = tmp_path / "main"
    subprocess.check_call(["/usr/bin/g++", "-std=c++17", "-O1", "-ftrapv", "-Wall", "-Werror", "-I", build.CSRC,
                           str(tmp_path / "main.cpp"), "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


@pytest.mark.parametrize("kernel", ["spmm_stream_kernel"])
def test_kernels_request_ahead_through_the_bounds(kernel):
    """In a kernel that reads ahead no index is compared after a look-ahead was added to it."""
    source = "".join(open(os.path.join(build.CSRC, f)).read() for f in build.CUDA_SOURCES)
    at = re.search(r"\b%s\(" % kernel, source).start()
    body = source[at:source.index("\n}\n", at)]
    assert "ahead_inside(" in body
    for name in ("from", "k0", "kg", "r"):
        sums = re.findall(r"\b%s \+ [^;?]*(?:<=?) *(?:k_end|r_end|min\()" % name, body)
        assert not sums, sums
