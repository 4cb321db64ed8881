"""The side-by-side build waits for every compiler before it reports that one
failed: none keeps writing objects behind a caller's back."""
import os
import stat
import subprocess

import pytest


def test_no_compiler_outlives_a_failed_build(tmp_path, monkeypatch):
    from meamzilla_b200 import build
    fake = tmp_path / "nvcc"
    fake.write_text("""#!/bin/sh
for a in "$@"; do case "$a" in *.cpp) exit 3;; *.cu) src=$a;; esac; done
sleep 1
touch "%s/$(basename "$src").done"
""" % tmp_path)
    fake.chmod(fake.stat().st_mode | stat.S_IXUSR)
    monkeypatch.setattr(build, "nvcc", lambda: str(fake))
    monkeypatch.setattr(build, "HERE", str(tmp_path))
    monkeypatch.setattr(build, "LIB", str(tmp_path / "lib.so"))
    with pytest.raises(subprocess.CalledProcessError) as e:
        build.build(force=True)
    assert e.value.returncode == 3
    for src in build.SOURCES:
        if src.endswith(".cu"):
            assert os.path.exists(tmp_path / (src + ".done")), src
    assert not os.path.exists(tmp_path / "lib.so")
