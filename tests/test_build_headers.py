"""Every header that a source of the library includes is among those whose change rebuilds it."""
import os
import re

from emdee_gb300 import build


def test_included_headers_are_dependencies():
    known = {os.path.normpath(os.path.join(build.CSRC, h)) for h in build.HEADERS}
    for name in os.listdir(build.CSRC):
        for inc in re.findall(r'#include "([^"]+)"', open(os.path.join(build.CSRC, name)).read()):
            path = os.path.normpath(os.path.join(build.CSRC, inc))
            assert path in known or not os.path.exists(path), (name, inc)
            assert os.path.exists(path) or os.path.normpath(os.path.join(build.HERE, "..", "include", inc)) in known, (name, inc)
