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


@pytest.mark.parametrize("rows,cols,inputs,pairs,room", [
    (85, 65536, 16384, 74, 0), (42, 131072, 16384, 74, 0), (87, 131072, 16384, 74, 0), (88, 65536, 16384, 74, 64),
    (29, 256000, 12288, 74, 0), (56, 131072, 12288, 74, 0), (88, 131072, 12288, 74, 64),
    (8192, 30528, 1024, 74, 6144), (6144, 30528, 1024, 74, 4608), (4096, 30528, 768, 74, 3072), (4099, 28680, 776, 74, 3072),
    (2048, 30528, 1024, 74, 0), (8192, 30529, 1024, 74, 0), (8192, 4095 * 8, 8192, 74, 0), (1 << 20, 1 << 20, 1024, 74, 1024),
    # the line for the tiles follows the SMs: an input gradient of 48 tiles on 74 pairs and on 76, a weight of 76
    (4096, 30528, 768, 76, 0), (1 << 16, 76 * 256, 256, 76, 49152), (1 << 16, 76 * 256, 256, 77, 0), (8192, 30528, 1024, 0, 0)])
def test_room_for_gathered_rows(rows, cols, inputs, pairs, room):
    """A wide layer's backward looks at its rows only where it has room for 64 of them or more: output layers of many inputs
    and few rows, for which nothing is left of three quarters in steps of 64, go over all rows."""
    import torch  # noqa: F401

    from rannc_b200 import _host

    assert _host.gather_room(rows, cols, inputs, pairs, 2) == room
    # one of the two products alone has to be as long as both; none is not worth a look
    alone = rows * cols * inputs >= 1.8e11
    assert _host.gather_room(rows, cols, inputs, pairs, 1) == (room if alone else 0)
    assert _host.gather_room(rows, cols, inputs, pairs, 0) == 0
