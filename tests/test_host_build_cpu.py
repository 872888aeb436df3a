"""When the operators' host library is built again."""
import importlib
import types
from pathlib import Path

import pytest

from rannc_b200 import build
from rannc_b200.ops import _lib


def test_a_library_that_does_not_load_is_rebuilt(monkeypatch):
    """One built against another PyTorch is newer than its sources and yet has to go."""
    real, calls = importlib.import_module, []
    fake = types.SimpleNamespace(init=lambda fns, err: calls.append(sorted(fns) == sorted(_lib._HOST_ENTRIES)))

    def load(name, *a):
        if name != "rannc_b200._host":
            return real(name, *a)
        if not calls:
            raise ImportError("undefined symbol")
        return fake

    monkeypatch.setattr(_lib, "_host", None)
    monkeypatch.setattr(importlib, "import_module", load)
    monkeypatch.setattr(build, "build_host", lambda verbose=False, force=False: calls.append(("force", force)))
    assert _lib.host() is fake
    assert calls == [("force", True), True]


@pytest.mark.parametrize("force", [False, True])
def test_force_builds_a_library_newer_than_its_sources(monkeypatch, tmp_path, force):
    ran = []

    def run(cmd):
        out = Path(cmd[cmd.index("-o") + 1])
        ran.append(out)
        out.write_bytes(b"new")
        return ""

    monkeypatch.setattr(build, "HERE", tmp_path)
    monkeypatch.setattr(build, "_run", run)
    path = build.build_host(force=True)
    ran.clear()
    path.write_bytes(b"old")
    assert build.build_host(force=force) == path
    assert path.read_bytes() == (b"new" if force else b"old") and len(ran) == int(force)
    assert [p.name for p in tmp_path.iterdir()] == [path.name]      # written beside and moved into place
