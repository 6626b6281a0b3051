"""Kernel launch attributes (dynamic shared memory, cluster sizes) belong to a
device, and a process may open contexts on several (idp_params.device): every
context sets what its launches need, once, on its own device. One GPU cannot
show a second device's launch being refused, so this runs on the CPU: the
context's helper against a runtime that counts the calls, and the sources, in
which nothing else may set an attribute.
"""
import os
import re
import shutil
import subprocess

import pytest

from idp_gb300 import build

PROGRAM = r"""
#include "attributes.hpp"
static int calls = 0, fail = 0;
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) {
    ++calls;
    return fail-- > 0 ? cudaErrorInvalidValue : cudaSuccess;
}
int main() {
    const int a = 0, b = 0;  // two kernels
    const cudaFuncAttribute what = cudaFuncAttributeMaxDynamicSharedMemorySize;
    idp::KernelAttributes first, second;  // of contexts on two devices
    for (int k = 0; k < 3; ++k)
        if (first.set(&a, what, 1) || first.set(&b, what, 1)) return 1;
    if (calls != 2) return 2;
    fail = 1;  // not remembered as set
    if (!second.set(&a, what, 1)) return 3;
    for (int k = 0; k < 3; ++k)
        if (second.set(&a, what, 1)) return 4;
    return calls == 4 ? 0 : 5;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_every_context_sets_its_attributes(tmp_path):
    src, exe = tmp_path / "attr.cpp", tmp_path / "attr"
    src.write_text(PROGRAM)
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
    r = subprocess.run(["g++", "-std=c++17", "-I", build.SRC, "-I", cuda, str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stderr)


def test_no_attribute_is_set_once_per_process():
    for unit in sorted(os.listdir(build.SRC)):
        text = open(os.path.join(build.SRC, unit)).read()
        want = 1 if unit == "attributes.hpp" else 0
        assert len(re.findall(r"\bcudaFuncSetAttribute\(", text)) == want, unit
