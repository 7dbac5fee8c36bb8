"""The library's build knows every header that its sources include, so that an edit of one rebuilds them."""
import importlib.util
import os
import re

from conftest import ROOT


def test_every_included_header_is_a_dependency():
    spec = importlib.util.spec_from_file_location(
        "pvb200_build_file", os.path.join(ROOT, "pointvortex_b200", "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    included = set()
    for name in os.listdir(build.CSRC):
        with open(os.path.join(build.CSRC, name)) as f:
            included |= set(re.findall(r'^\s*#include\s+"([^"]+)"', f.read(), re.M))
    assert included - {"pvb200.h"} == set(build.HEADERS)
