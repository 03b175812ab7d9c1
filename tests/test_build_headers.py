"""Every header that a translation unit includes is a dependency of the build, so an
edit of one rebuilds the objects that contain it."""
import os
import re

from codyfortran_gb300 import build


def test_included_headers_are_dependencies():
    names = set()
    for f in os.listdir(build.CSRC):
        with open(os.path.join(build.CSRC, f)) as h:
            names |= set(re.findall(r'#include "([^"/]+\.cuh)"', h.read()))
    assert names == set(build.HEADERS)
