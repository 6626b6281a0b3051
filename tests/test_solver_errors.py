"""What a failed solve leaves in its context. The library's own objects run
without a device here, so that the CUDA calls of the solver's set-up fail: what
failed must not count as done, or the next solve would launch on a layout that
was never made.
"""
import os
import re
import subprocess

import pytest

from idp_gb300 import build

LAYOUT = r"""
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

SOLVE = r"""
#include "engine.hpp"
using namespace idp;
int main() {
    Arena A;
    Work W;
    ContactSet cs;
    A.nI = 1;
    A.V = 500;
    A.v_off = {0, 500};
    W.sell.xch_bytes = 4096;
    std::vector<int> its;
    std::vector<double> rel;
    if (pcg_solve(A, W, cs, false, nullptr, nullptr, 1e-6, 10, {1}, its, rel, nullptr) == IDP_OK) return 1;
    return W.sell.xch_bytes == 0 ? 0 : 2;
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
    assert without_device("layout", LAYOUT) == 0


def test_a_failed_solve_clears_the_exchange(without_device):
    """Its tags may have been used: the words are cleared before the next solve."""
    assert without_device("solve", SOLVE) == 0


def test_the_mask_of_a_failed_solve_is_unknown():
    """The refinement narrows the mask on the device and puts it back only when it
    ends well; set_mask skips an upload that it takes for held already. So every
    solve of the engine goes through the one function that forgets the mask on an
    error (the state is the library's own: read from the source)."""
    text = open(os.path.join(build.SRC, "engine.cpp")).read()
    assert len(re.findall(r"\bpcg_solve\(", text)) == 1
    body = text[text.index("int solve_directions("):]
    body = body[:body.index("\n}\n")]
    assert "pcg_solve(" in body and "if (rc) c->mask_dev.clear();" in body
