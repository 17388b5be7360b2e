"""An incremental build recompiles what a changed header reaches."""
import glob
import os
import re

from daxtoolkit_gb300 import build


def test_every_included_header_is_a_dependency():
    deps = {os.path.realpath(p) for p in build.headers()}
    found = 0
    for src in glob.glob(os.path.join(build.CSRC, "*.cu")) + glob.glob(os.path.join(build.CSRC, "*.cuh")):
        for inc in re.findall(r'^\s*#include "([^"]+)"', open(src).read(), re.M):
            path = os.path.join(os.path.dirname(src), inc)
            if not os.path.exists(path):
                path = os.path.join(build.HERE, "..", "include", inc)
            assert os.path.realpath(path) in deps, (src, inc)
            found += 1
    assert found > 20
