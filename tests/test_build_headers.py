"""Every header that a translation unit includes, directly or through another
header, counts as a dependency of the build: an edit to any of them recompiles."""
import os
import re

from idp_gb300 import build


def test_every_included_header_is_a_dependency():
    deps = {os.path.normpath(d) for d in build.dependencies()}
    for name in sorted(os.listdir(build.SRC)):
        with open(os.path.join(build.SRC, name)) as f:
            for inc in re.findall(r'^\s*#include\s+"([^"]+)"', f.read(), re.M):
                paths = [os.path.normpath(os.path.join(d, inc)) for d in (build.SRC, build.INCLUDE)]
                assert any(p in deps for p in paths), (name, inc)
