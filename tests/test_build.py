"""The library counts as stale when any file that it is compiled from is newer."""
import os
import re

import pytest

from ultrasound_solver_b200 import build


def _included():
    """Names of the package's own files that the sources include, directly or not."""
    seen, todo = set(), list(build.SOURCES)
    while todo:
        text = (build.CSRC / todo.pop()).read_text()
        for name in re.findall(r'^\s*#\s*include\s+"([^"]+)"', text, re.M):
            if name not in seen and (build.CSRC / name).exists():
                seen.add(name)
                todo.append(name)
    return sorted(seen)


FILES = [*_included(), *build.SOURCES]


@pytest.mark.parametrize("name", FILES)
def test_newer_file_makes_the_library_stale(tmp_path, monkeypatch, name):
    monkeypatch.setattr(build, "CSRC", tmp_path)
    monkeypatch.setattr(build, "INCLUDE", tmp_path)
    target = tmp_path / "lib.so"
    for f in [*FILES, "usv.h"]:
        (tmp_path / f).touch()
        os.utime(tmp_path / f, (1000, 1000))
    target.touch()
    os.utime(target, (2000, 2000))
    assert not build._stale(target)
    os.utime(tmp_path / name, (3000, 3000))
    assert build._stale(target)
