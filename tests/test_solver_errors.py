"""What a failed solve leaves in its context. The library's own objects run
without a device here, so that the CUDA calls of the solver's set-up fail: what
failed must not count as done, or the next solve would launch on a layout that
was never made.
"""
import os
import subprocess

import pytest

from idp_gb300 import build

PROGRAM = r"""
#include "engine.hpp"
using namespace idp;
int main() {
    Arena A;
    Work W;
    A.nI = 1;
    A.V = 500;
    A.v_off = {0, 500};
    if (sell_plan(A, W, nullptr) == IDP_OK) return 1;
    if (W.sell.ready) return 2;  // the next solve makes the layout
    return 0;
}
"""


@pytest.fixture(scope="module")
def without_device(tmp_path_factory):
    """Compiles a program against the library's objects and returns its exit code
    in a process that sees no device."""
    build.build()
    d = tmp_path_factory.mktemp("errors")

    def run(name, program):
        src, exe = d / (name + ".cu"), d / name
        src.write_text(program)
        objs = [os.path.join(build.OUT_DIR, u + ".o") for u in build.UNITS]
        r = subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-I", build.SRC, "-I",
                            build.INCLUDE, str(src), *objs, "-lpthread", "-o", str(exe)], capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
        return subprocess.run([str(exe)], capture_output=True, env={**os.environ, "CUDA_VISIBLE_DEVICES": ""}).returncode

    return run


def test_a_failed_layout_is_made_again(without_device):
    assert without_device("layout", PROGRAM) == 0
