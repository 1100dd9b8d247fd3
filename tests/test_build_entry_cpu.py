"""The build entry point where the reference checkout is missing or its directory
is empty: the reference's kernels are left as they are and the build succeeds."""
import os
import subprocess
import sys

import pytest

from conftest import ORACLE, ROOT


@pytest.mark.parametrize("made", [False, True])
def test_build_without_a_reference_checkout(tmp_path, monkeypatch, made):
    sys.path.insert(0, ROOT)
    import __graft_entry__ as entry

    where = tmp_path / "reference"
    if made:
        where.mkdir()
    calls = []
    monkeypatch.setattr(entry, "REFERENCE", str(where))
    monkeypatch.setattr(entry.subprocess, "check_call", lambda cmd, **kw: calls.append(cmd))
    entry.build()
    assert len(calls) == 2 and all(c[0] == "make" for c in calls)
    monkeypatch.undo()
    res = subprocess.run([sys.executable, os.path.join(ORACLE, "build_ref.py"), "--reference", str(where)],
                         capture_output=True, text=True)
    assert res.returncode == 0 and "not present" in res.stderr
