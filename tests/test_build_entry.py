"""build() compiles the checker only where there is a reference checkout."""
import subprocess

import pytest


@pytest.mark.parametrize("checkout", [False, True])
def test_checker_is_built_only_from_a_checkout(tmp_path, monkeypatch, checkout):
    import __graft_entry__ as entry
    from gradientdomaintextureprocessing_b200 import build
    if checkout:
        (tmp_path / "include" / "Src").mkdir(parents=True)
    calls = []
    monkeypatch.setenv("GDTP_REFERENCE", str(tmp_path))
    monkeypatch.setattr(build, "build", lambda **_: None)
    monkeypatch.setattr(subprocess, "run", lambda *a, **_: calls.append(a))
    entry.build()
    assert len(calls) == (1 if checkout else 0)
