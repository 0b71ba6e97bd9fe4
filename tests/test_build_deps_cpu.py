"""An object is out of date when any file of the library that its source includes,
directly or not, is newer: the build's list of dependencies covers them."""
import os
import re

import pytest

from lywell_gb300 import build


def _includes(path, seen):
    for name in re.findall(r'#include "([^"]+)"', open(path).read()):
        p = os.path.normpath(os.path.join(os.path.dirname(path), name))
        if os.path.exists(p) and p not in seen:
            seen.add(p)
            _includes(p, seen)
    return seen


@pytest.mark.parametrize("src", build.SOURCES)
def test_included_files_are_dependencies(src, tmp_path, monkeypatch):
    path = os.path.join(build.CSRC, src)
    obj = tmp_path / (os.path.splitext(src)[0] + ".o")
    obj.write_text("")
    monkeypatch.setattr(build, "OBJ_DIR", str(tmp_path))
    compiled = []
    monkeypatch.setattr(build.subprocess, "run", lambda cmd, **k: compiled.append(cmd) or type("R", (), {"returncode": 0}))
    now = os.stat(obj).st_mtime
    real = os.path.getmtime
    for dep in sorted(_includes(path, set())):
        # every file older than the object, but this one
        monkeypatch.setattr(os.path, "getmtime",
                            lambda p: now + 1 if os.path.normpath(p) == dep else now if str(p) == str(obj) else now - 1)
        compiled.clear()
        build._compile(src)
        assert compiled, (src, dep)
    monkeypatch.setattr(os.path, "getmtime", real)
